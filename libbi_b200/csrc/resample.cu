// Resamplers of the bootstrap particle filter, B200-native.
//
// Reference path (LibBi): Resampler<R>::resample
// (share/src/bi/resampler/Resampler.hpp:167-182) runs R::precompute
// (ScanResampler::precompute, share/src/bi/resampler/ScanResampler.hpp:35-40:
// a Thrust max pass and a Thrust transform_inclusive_scan of nanexp(lw - max))
// and R::ancestorsPermute, then gathers the state.  The reference's CUDA
// variants use Thrust for the scan and search and atomics for the
// permutation (share/src/bi/cuda/resampler/ResamplerKernel.cuh:78-165).
//
// Here every pass is a hand-written kernel over tiles of kTile = 512
// log-weights (256 threads x 2):
//   weight tile sums   exact 128-bit fixed-point sums of the weights; the
//                      last block to finish scans the tile sums (no waiting)
//   offspring          per tile: exact prefix -> FP64 cumulative weight ->
//                      cumulative offspring, childless counts
//   permute            survivors in place; copies fill childless slots by a
//                      search over the cumulative extra-copy counts
// Permuted systematic resampling runs all of these as phases of one
// cooperative launch: k_systematic_coop1 with one tile per block in one of
// six autotuned tile shapes, its phases handing over through tagged words
// that every block polls, or k_systematic_coop with several tiles per block
// and bounded grid barriers.  The passes above are the
// path for multinomial and Metropolis offspring.  The FP64 cumulative weight
// of element i is the exact sum rounded once, so ancestors are independent
// of tile order, tile shape, thread count and timing.
#include "internal.cuh"

#include <algorithm>
#include <mutex>
#include <vector>
#include "resample_common.cuh"
#include "handover.cuh"
#include "reduce.cuh"
#include "../../include/bpf_math.h"


namespace bpf {

// ---------------------------------------------------------------------------
// helpers
// ---------------------------------------------------------------------------

// Signal "this block is done" and return true in every thread of the last
// block of the grid to finish.  The caller's global writes must precede it.
__device__ __forceinline__ bool last_block_arrive(unsigned* counter) {
  __shared__ bool am_last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned ticket = atomicAdd(counter, 1u);
    am_last = (ticket == gridDim.x - 1);
  }
  __syncthreads();
  if (am_last) __threadfence();
  return am_last;
}

__device__ __forceinline__ u128 ldcg_u128(const u128* p) {
  u128 r;
  r.lo = __ldcg(&p->lo);
  r.hi = __ldcg(&p->hi);
  return r;
}

// Exclusive scan of in[0..T) into out[0..T] (out[T] = total), run by one block.
__device__ void block_scan_tiles_u128(const u128* in, u128* out, int T) {
  u128 carry = u128_zero();
  for (int base = 0; base < T; base += kTile) {
    u128 v[kItems];
    u128 loc = u128_zero();
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
      int i = base + threadIdx.x * kItems + k;
      v[k] = i < T ? ldcg_u128(&in[i]) : u128_zero();
      loc = u128_add(loc, v[k]);
    }
    u128 tot;
    u128 ex = u128_add(carry, block_exclusive_scan_u128(loc, &tot));
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
      int i = base + threadIdx.x * kItems + k;
      if (i < T) out[i] = ex;
      ex = u128_add(ex, v[k]);
    }
    carry = u128_add(carry, tot);
  }
  if (threadIdx.x == 0) out[T] = carry;
}

__device__ void block_scan_tiles_int(const int* in, int* out, int T) {
  int carry = 0;
  for (int base = 0; base < T; base += kTile) {
    int v[kItems];
    int loc = 0;
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
      int i = base + threadIdx.x * kItems + k;
      v[k] = i < T ? __ldcg(&in[i]) : 0;
      loc += v[k];
    }
    int tot;
    int ex = carry + block_exclusive_scan_int(loc, &tot);
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
      int i = base + threadIdx.x * kItems + k;
      if (i < T) out[i] = ex;
      ex += v[k];
    }
    carry += tot;
  }
  if (threadIdx.x == 0) out[T] = carry;
}

// Load the 8 consecutive log-weights of this thread (blocked layout).
__device__ __forceinline__ void load_blocked(const double* __restrict__ lw, int i0, int n, double v[kItems]) {
  if (i0 + kItems <= n && ((reinterpret_cast<uintptr_t>(lw + i0) & 15) == 0)) {
    const double2* p = reinterpret_cast<const double2*>(lw + i0);
#pragma unroll
    for (int k = 0; k < kItems / 2; ++k) {
      double2 t = __ldg(p + k);
      v[2 * k] = t.x;
      v[2 * k + 1] = t.y;
    }
  } else {
#pragma unroll
    for (int k = 0; k < kItems; ++k) v[k] = (i0 + k < n) ? __ldg(lw + i0 + k) : NAN;
  }
}

__device__ __forceinline__ int block_max_int(int v) {
  __shared__ int wm[kBlock / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, d));
  if (lane == 0) wm[warp] = v;
  __syncthreads();
  int r = lane < kBlock / 32 ? wm[lane] : 0;
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) r = max(r, __shfl_xor_sync(0xffffffffu, r, d));
  __syncthreads();
  return r;
}

// The first index whose entry of the nondecreasing A[0..n) exceeds x (n if
// none does), by a whole warp: 32 probes at a time, so that 2^20 entries take
// four round trips instead of twenty.
template <class T>
__device__ __forceinline__ int warp_upper_bound(const T* __restrict__ A, int n, T x) {
  const int lane = threadIdx.x & 31;
  int lo = 0, hi = n;
  while (lo < hi) {
    const int step = (hi - lo + 31) >> 5;
    const int i = lo + lane * step;
    const unsigned above = __ballot_sync(0xffffffffu, i < hi && __ldg(A + i) > x);
    // probes inside [lo, hi) that are not above x form a prefix of the lanes
    const int probes = (hi - lo + step - 1) / step;
    const int first = above ? __ffs(above) - 1 : probes;
    if (first < probes) hi = lo + first * step;
    if (first > 0) lo = lo + (first - 1) * step + 1;
  }
  return lo;
}

// The same for one x per thread, nondecreasing over the block's threads from
// x_first to x_last: two warps bracket the block's answers, then each thread
// searches between them (a few steps in lines its neighbours read too,
// instead of log2 n dependent loads).
template <class T>
__device__ __forceinline__ void block_bounds(const T* __restrict__ A, int n, T x_first, T x_last, int (&bound)[2]) {
  __shared__ int s_bound[2];
  const int warp = threadIdx.x >> 5;
  __syncthreads();  // an earlier call's bounds have been read
  if (warp < 2) {
    const int r = warp_upper_bound(A, n, warp == 0 ? x_first : x_last);
    if ((threadIdx.x & 31) == 0) s_bound[warp] = r;
  }
  __syncthreads();
  bound[0] = s_bound[0];
  bound[1] = s_bound[1];
}

template <class T>
__device__ __forceinline__ int upper_bound_in(const T* __restrict__ A, int lo, int hi, T x) {
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (__ldg(A + mid) > x) hi = mid; else lo = mid + 1;
  }
  return lo;
}

// K searches per thread side by side, so that their loads are in flight
// together: answers in [first, first + len], the same range for all.
template <int K, class T>
__device__ __forceinline__ void upper_bounds_between(const T* __restrict__ A, int first, int len, const T (&x)[K],
                                                     int (&b)[K]) {
#pragma unroll
  for (int k = 0; k < K; ++k) b[k] = first;
  while (len > 1) {
    const int half = len >> 1;
    T v[K];
#pragma unroll
    for (int k = 0; k < K; ++k) v[k] = A[b[k] + half - 1];
#pragma unroll
    for (int k = 0; k < K; ++k) b[k] = v[k] > x[k] ? b[k] : b[k] + half;
    len -= half;
  }
  if (len == 1) {
#pragma unroll
    for (int k = 0; k < K; ++k) b[k] += A[b[k]] > x[k] ? 0 : 1;
  }
}

template <int K, class T>
__device__ __forceinline__ void block_upper_bounds(const T* __restrict__ A, int n, const T (&x)[K], T x_first, T x_last,
                                                   int (&b)[K]) {
  int bound[2];
  block_bounds(A, n, x_first, x_last, bound);
  upper_bounds_between(A, bound[0], bound[1] - bound[0], x, b);
}

__device__ __forceinline__ bool gate_closed(const int* gate, const StepStats* st) {
  if (gate != nullptr && *gate == 0) return true;
  return st->status != BPF_OK;
}

// ---------------------------------------------------------------------------
// The first pass of a stand-alone call: the largest log-weight (NaN ignored),
// which is all the resamplers need of the statistics, and a clean start for
// the rest of the call (status, grid-barrier words, the one-launch kernel's
// epoch).  8 bytes per log-weight and two operations, against the full
// reduction's exp (k_lw_reduce: 17 us at 4 M log-weights in L2).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kBlock)
k_lw_max(const double* __restrict__ lw, int n, LwPartial* partials, StepStats* st, unsigned* counters) {
  constexpr int K = 8;
  double m = -INFINITY;
  const long long stride = (long long)gridDim.x * kBlock * K;
  long long i = (long long)(blockIdx.x * kBlock + threadIdx.x) * 2;
  if ((reinterpret_cast<uintptr_t>(lw) & 15) == 0) {
    // consecutive threads on consecutive pairs, K / 2 pairs in flight
    const long long row = (long long)gridDim.x * kBlock * 2;
    for (; i + (K / 2 - 1) * row + 1 < n; i += stride) {
      double2 v[K / 2];
#pragma unroll
      for (int k = 0; k < K / 2; ++k) v[k] = __ldg(reinterpret_cast<const double2*>(lw + i + k * row));
#pragma unroll
      for (int k = 0; k < K / 2; ++k) m = fmax(m, fmax(v[k].x, v[k].y));
    }
    for (; i < n; i += row) {
      m = fmax(m, __ldg(lw + i));
      if (i + 1 < n) m = fmax(m, __ldg(lw + i + 1));
    }
  } else {
    for (i = blockIdx.x * kBlock + threadIdx.x; i < n; i += gridDim.x * kBlock) m = fmax(m, __ldg(lw + i));
  }
  __shared__ double s_m[kBlock / 32];
  __shared__ bool am_last;
#pragma unroll 1
  for (int pass = 0;; ++pass) {
    m = warp_max(m);
    if ((threadIdx.x & 31) == 0) s_m[threadIdx.x >> 5] = m;
    __syncthreads();
    m = warp_max((threadIdx.x & 31) < kBlock / 32 ? s_m[threadIdx.x & 31] : -INFINITY);
    if (pass == 1 || gridDim.x == 1) break;  // one block's maximum is the result
    if (threadIdx.x == 0) {
      partials[blockIdx.x].mx = m;
      __threadfence();
      am_last = atomicAdd(counters + 3, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!am_last) return;
    __threadfence();
    m = -INFINITY;
    for (int b = threadIdx.x; b < (int)gridDim.x; b += kBlock) m = fmax(m, __ldcg(&partials[b].mx));
  }
  if (threadIdx.x == 0) {
    st->mx = m;
    st->status = BPF_OK;
    counters[3] = 0u;
    counters[8] = 0u;
    counters[9] = 0u;
    counters[kEpochWord] += 1u;
  }
}

// ---------------------------------------------------------------------------
// weight tile sums (+ spacing tile sums for multinomial)
// ---------------------------------------------------------------------------
// Block-wide sums of one u128 per thread of each of NV values (blockDim.x ==
// kBlock), in thread 0: exact, so any order gives the same.
template <int NV>
__device__ __forceinline__ void block_sum_u128(u128 (&v)[NV]) {
  __shared__ u128 ws[NV][kBlock / 32];
#pragma unroll
  for (int j = 0; j < NV; ++j) {
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
      u128 o;
      o.lo = __shfl_xor_sync(0xffffffffu, v[j].lo, d);
      o.hi = __shfl_xor_sync(0xffffffffu, v[j].hi, d);
      v[j] = u128_add(v[j], o);
    }
    if ((threadIdx.x & 31) == 0) ws[j][threadIdx.x >> 5] = v[j];
  }
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int j = 0; j < NV; ++j)
      for (int w = 1; w < kBlock / 32; ++w) v[j] = u128_add(v[j], ws[j][w]);
  }
}

// A tile is kBlock * ITEMS particles, consecutive threads on consecutive
// ones: only the tile's sums are needed, and loads and stores of a warp are
// then whole lines.  Bound by instruction issue (about 450 a particle with
// spacings) and the last block's scans of the tiles; at 10^6 particles 21.7
// us against 28 with tiles of 512 particles, each summed by two block scans,
// four chunks of which the last block then scanned one after another.
template <int ITEMS, bool MULT>
__global__ void __launch_bounds__(kBlock)
k_weight_tile_sums(const double* __restrict__ lw, int n, StepStats* st,
                   u128* tile_sum, u128* tile_prefix,
                   const double* u, uint64_t seed, int step,
                   u128* vtile_sum, u128* vtile_prefix, unsigned long long* qbuf, double* spbuf,
                   unsigned* counter, const int* gate) {
  if (gate_closed(gate, st)) return;
  const double mx = st->mx;
  const int t = blockIdx.x;
  const long long i0 = (long long)t * (kBlock * ITEMS) + threadIdx.x;
  u128 acc[MULT ? 2 : 1];
#pragma unroll
  for (int j = 0; j < (MULT ? 2 : 1); ++j) acc[j] = u128_zero();
  double nx[2];
#pragma unroll
  for (int j = 0; j < 2; ++j) nx[j] = i0 + j * kBlock < n ? __ldg(lw + i0 + j * kBlock) : 0.0;
  // two particles at a time, the next two's log-weights in flight: unrolled
  // further, the code (an exp, a draw, a logarithm and a division each) no
  // longer fits the instruction cache
#pragma unroll 1
  for (int k = 0; k < ITEMS; k += 2) {
    double v[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      v[j] = nx[j];
      const long long in = i0 + (k + 2 + j) * kBlock;
      if (k + 2 < ITEMS) nx[j] = in < n ? __ldg(lw + in) : 0.0;
    }
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const long long i = i0 + (k + j) * kBlock;
      if (i < n) {
        const double w = nanexp(__dsub_rn(v[j], mx));
        u128 q; q.lo = weight_to_fixed(w); q.hi = 0;
        acc[0] = u128_add(acc[0], q);
        if (MULT) {
          // kept for k_multinomial_prepare: 16 bytes against an exp, a draw,
          // a logarithm and a division
          const double sp = multinomial_spacing(u, (int)i, n, seed, step);
          acc[MULT ? 1 : 0] = u128_add(acc[MULT ? 1 : 0], spacing_to_fixed(sp));
          qbuf[i] = q.lo;
          spbuf[i] = sp;
        }
      }
    }
  }
  block_sum_u128(acc);
  if (threadIdx.x == 0) {
    tile_sum[t] = acc[0];
    if (MULT) vtile_sum[t] = acc[MULT ? 1 : 0];
  }
  if (last_block_arrive(counter)) {
    block_scan_tiles_u128(tile_sum, tile_prefix, gridDim.x);
    if (MULT) block_scan_tiles_u128(vtile_sum, vtile_prefix, gridDim.x);
    __syncthreads();
    if (threadIdx.x == 0) {
      *counter = 0;
      // SystematicResampler::cumulativeOffspring throws
      // ParticleFilterDegeneratedException unless W > 0
      // (share/src/bi/resampler/SystematicResampler.hpp:118-129)
      double W = u128_to_weight(tile_prefix[gridDim.x]);
      if (!(W > 0.0)) st->status = BPF_E_DEGENERATE;
    }
  }
}

// ---------------------------------------------------------------------------
// systematic: cumulative offspring and childless counts per tile
__global__ void __launch_bounds__(kBlock)
k_systematic_offspring(const double* __restrict__ lw, int n, StepStats* st,
                       const u128* tile_prefix, const double* a_in, uint64_t seed, int step,
                       int* Os, int* zcount, int* zprefix, unsigned* counter, const int* gate) {
  if (gate_closed(gate, st)) return;
  __shared__ int s_last[kBlock];
  const double mx = st->mx;
  const int t = blockIdx.x;
  const int T = gridDim.x;
  const int i0 = t * kTile + threadIdx.x * kItems;
  double a;
  if (a_in) {
    a = *a_in;
  } else {
    bpf_u32x4 r = bpf_draw(seed, 0u, (uint32_t)step, 0u, BPF_RNG_SYSTEMATIC);
    a = bpf_u01d(r.v[0], r.v[1]);
  }
  const double W = u128_to_weight(tile_prefix[T]);
  const double yW = __ddiv_rn(1.0, W);
  const double nd = (double)n;

  double v[kItems];
  load_blocked(lw, i0, n, v);
  unsigned long long q[kItems];
  u128 loc = u128_zero();
#pragma unroll
  for (int k = 0; k < kItems; ++k) {
    q[k] = (i0 + k < n) ? weight_to_fixed(nanexp(__dsub_rn(v[k], mx))) : 0ull;
    u128 qq; qq.lo = q[k]; qq.hi = 0;
    loc = u128_add(loc, qq);
  }
  u128 tot;
  u128 Q = u128_add(tile_prefix[t], block_exclusive_scan_u128(loc, &tot));
  int os[kItems];
#pragma unroll
  for (int k = 0; k < kItems; ++k) {
    u128 qq; qq.lo = q[k]; qq.hi = 0;
    Q = u128_add(Q, qq);
    os[k] = systematic_Os(u128_to_weight(Q), W, yW, nd, a, n);
  }
  s_last[threadIdx.x] = os[kItems - 1];
  __syncthreads();
  int prev;
  if (threadIdx.x > 0) {
    prev = s_last[threadIdx.x - 1];
  } else {
    prev = t == 0 ? 0 : systematic_Os(u128_to_weight(tile_prefix[t]), W, yW, nd, a, n);
  }
  int zeros = 0;
#pragma unroll
  for (int k = 0; k < kItems; ++k) {
    if (i0 + k < n) {
      Os[i0 + k] = os[k];
      zeros += (os[k] == prev);
    }
    prev = os[k];
  }
  int ztot;
  block_exclusive_scan_int(zeros, &ztot);
  if (threadIdx.x == 0) zcount[t] = ztot;
  if (last_block_arrive(counter)) {
    block_scan_tiles_int(zcount, zprefix, T);
    if (threadIdx.x == 0) *counter = 0;
  }
}

// ---------------------------------------------------------------------------
// systematic resampling in one cooperative launch
//
// The four passes above (weight sums, offspring, survivors, fill) run as
// phases of one kernel separated by grid-wide barriers.  The grid is at most
// as large as the GPU can hold at once and is launched cooperatively, so every
// block is resident and every barrier is reached; each wait is still bounded
// by a clock limit after which the kernel records BPF_E_TIMEOUT and returns.
// Block b owns the contiguous tiles [b T / G, (b+1) T / G); prefix sums over
// blocks are formed from the G block totals published at each barrier.
// Data written during the kernel is read with ld.global.cg (never through the
// read-only cache).
// ---------------------------------------------------------------------------
constexpr long long kBarrierTimeoutCycles = 4000000000ll;  // ~2 s at 2 GHz

// The limit the waits use, per device (set_barrier_limit).  A negative limit
// makes a block that finds the barrier still closed give up at once, which
// lets a test take the BPF_E_TIMEOUT path without a kernel that never
// arrives.
__device__ long long g_barrier_limit = kBarrierTimeoutCycles;

__device__ __forceinline__ unsigned long long atom_add_acq_rel_gpu_u64(unsigned long long* p, unsigned long long v) {
  unsigned long long old;
  asm volatile("atom.acq_rel.gpu.global.add.u64 %0, [%1], %2;" : "=l"(old) : "l"(p), "l"(v) : "memory");
  return old;
}

__device__ __forceinline__ void red_add_release_gpu_u64(unsigned long long* p, unsigned long long v) {
  asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

__device__ __forceinline__ unsigned long long ld_acquire_gpu_u64(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

// Bounded grid barrier on one 64-bit word (the two counter words from
// `word`, 8-byte aligned): its high half counts completed barriers (the
// generation), its low half the blocks arrived at the open one.  Thread 0
// of each block arrives with one acquire-release add (the block's writes,
// ordered before it by the block barrier, are released with it; the adds
// form one release sequence); the block whose add returned the count
// G - 1 has acquired every arrival and closes the barrier with a release
// add that moves the word to the next generation with count zero; the
// others poll the word with acquire loads until its generation changes.
// One L2 round trip to arrive and one to see the release, with no read of
// the generation before the arrival.  Returns false (in every thread) on
// timeout.  A block that gives up has already arrived, so after a timeout
// the count can stay above zero: the host clears the word together with
// the status before the next launch on the same scratch (the status reset
// of the stand-alone resampler, bpf_init and bpf_restore of a filter), and
// until then the sticky status keeps every later launch on that scratch
// from starting.
__device__ __forceinline__ bool grid_barrier(unsigned* word, unsigned* /* second half of the word */,
                                             StepStats* st) {
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long* w = reinterpret_cast<unsigned long long*>(word);
    const unsigned long long old = atom_add_acq_rel_gpu_u64(w, 1ull);
    const unsigned gen = (unsigned)(old >> 32);
    int ok = 1;
    if ((unsigned)old + 1u == gridDim.x) {
      red_add_release_gpu_u64(w, (1ull << 32) - (unsigned long long)gridDim.x);
    } else {
      const long long lim = g_barrier_limit;
      const long long t0 = clock64();
      while ((unsigned)(ld_acquire_gpu_u64(w) >> 32) == gen) {
        if (lim < 0 || clock64() - t0 > lim) {
          ok = 0;
          st->status = BPF_E_TIMEOUT;
          break;
        }
      }
    }
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

template <int IT>
__device__ __forceinline__ void load_blocked_n(const double* __restrict__ lw, int i0, int n, double (&v)[IT]) {
  if (i0 + IT <= n && ((reinterpret_cast<uintptr_t>(lw + i0) & 15) == 0)) {
    const double2* p = reinterpret_cast<const double2*>(lw + i0);
#pragma unroll
    for (int k = 0; k < IT / 2; ++k) {
      double2 t = __ldg(p + k);
      v[2 * k] = t.x;
      v[2 * k + 1] = t.y;
    }
  } else {
#pragma unroll
    for (int k = 0; k < IT; ++k) v[k] = (i0 + k < n) ? __ldg(lw + i0 + k) : NAN;
  }
}

__device__ __forceinline__ u128 block_sum_u128_from_global(const u128* a, int count) {
  // sum of a[0..count) by the whole block (exact, any order)
  u128 acc = u128_zero();
  for (int i = threadIdx.x; i < count; i += blockDim.x) acc = u128_add(acc, ldcg_u128(&a[i]));
  u128 tot;
  block_exclusive_scan_u128(acc, &tot);
  return tot;
}

__device__ __forceinline__ int block_sum_int_from_global(const int* a, int count) {
  int acc = 0;
  for (int i = threadIdx.x; i < count; i += blockDim.x) acc += __ldcg(&a[i]);
  int tot;
  block_exclusive_scan_int(acc, &tot);
  return tot;
}

// Warp-wide inclusive scans (32 lanes).
__device__ __forceinline__ u128 warp_inclusive_u128(u128 v) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const u128 o = shfl_up_u128(v, d);
    if (lane >= d) v = u128_add(v, o);
  }
  return v;
}

__device__ __forceinline__ int warp_inclusive_int(int v) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int o = __shfl_up_sync(0xffffffffu, v, d);
    if (lane >= d) v += o;
  }
  return v;
}

__device__ __forceinline__ int warp_inclusive_max_int(int v) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int o = __shfl_up_sync(0xffffffffu, v, d);
    if (lane >= d) v = max(v, o);
  }
  return v;
}

// The segments [s0, s1) of warp `warp` when segments [b0, b1) are shared by
// the block's warps in contiguous runs.
__device__ __forceinline__ void warp_segments(int b0, int b1, int warp, int nwarps, int* s0, int* s1) {
  const long long c = b1 - b0;
  *s0 = b0 + (int)(c * warp / nwarps);
  *s1 = b0 + (int)(c * (warp + 1) / nwarps);
}

// Several segments per block (n beyond one tile per resident block).  The
// particles are cut into segments of 32 x IT; block b owns a contiguous run
// of segments and each of its warps a contiguous run of those, so every
// scan inside a phase is a warp scan carried from segment to segment, and
// the block synchronises only at the phase boundaries.  Block prefixes come
// from the G block totals published at each grid barrier, warp prefixes
// from the block's per-warp totals in shared memory.
template <int IT>
__global__ void __launch_bounds__(kBlock)
k_systematic_coop(const double* __restrict__ lw, int n, StepStats* st, const double* a_in, uint64_t seed, int step,
                  int* Os, int* as, int* marks, int* slot, unsigned long long* qbuf, u128* block_w, int* block_z, int* block_m,
                  unsigned* bar_counter, unsigned* bar_gen, const int* gate) {
  pdl_trigger();  // as in k_systematic_coop1
  if (gate_closed(gate, st)) return;
  constexpr int NW = kBlock / 32;
  constexpr int S = 32 * IT;  // particles per segment
  __shared__ u128 s_wsum[NW];
  __shared__ int s_wint[NW];
  const int G = gridDim.x, b = blockIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int NS = (n + S - 1) / S;
  const int sb0 = (int)(((long long)b * NS) / G), sb1 = (int)(((long long)(b + 1) * NS) / G);
  int ws0, ws1;
  warp_segments(sb0, sb1, warp, NW, &ws0, &ws1);
  const double mx = st->mx;
  double a;
  if (a_in) {
    a = *a_in;
  } else {
    bpf_u32x4 r = bpf_draw(seed, 0u, (uint32_t)step, 0u, BPF_RNG_SYSTEMATIC);
    a = bpf_u01d(r.v[0], r.v[1]);
  }

  // phase 1: exact fixed-point weights (kept for phase 2) and their totals
  // per warp and per block
  {
    u128 wsum = u128_zero();
    // every segment loop issues the next segment's loads before the current
    // segment's arithmetic and scans, so the memory latency overlaps them
    double nv[IT];
    if (ws0 < ws1) load_blocked_n<IT>(lw, ws0 * S + lane * IT, n, nv);
    for (int sg = ws0; sg < ws1; ++sg) {
      const int i0 = sg * S + lane * IT;
      double v[IT];
#pragma unroll
      for (int k = 0; k < IT; ++k) v[k] = nv[k];
      if (sg + 1 < ws1) load_blocked_n<IT>(lw, i0 + S, n, nv);
#pragma unroll
      for (int k = 0; k < IT; ++k) {
        if (i0 + k < n) {
          u128 q; q.lo = weight_to_fixed(nanexp(__dsub_rn(v[k], mx))); q.hi = 0;
          qbuf[i0 + k] = q.lo;
          wsum = u128_add(wsum, q);
        }
      }
    }
    wsum = warp_inclusive_u128(wsum);  // lane 31: the warp's total
    if (lane == 31) s_wsum[warp] = wsum;
    __syncthreads();
    if (threadIdx.x == 0) {
      u128 t = u128_zero();
      for (int w = 0; w < NW; ++w) t = u128_add(t, s_wsum[w]);
      block_w[b] = t;
    }
  }
  if (!grid_barrier(bar_counter, bar_gen, st)) return;

  // phase 2: cumulative offspring and childless counts
  const u128 prefix_b = block_sum_u128_from_global(block_w, b);
  const u128 total = block_sum_u128_from_global(block_w, G);
  const double W = u128_to_weight(total);
  // SystematicResampler::cumulativeOffspring throws unless W > 0
  // (share/src/bi/resampler/SystematicResampler.hpp:118-129); every block
  // computes the same W and leaves together
  if (!(W > 0.0)) {
    if (b == 0 && threadIdx.x == 0) st->status = BPF_E_DEGENERATE;
    return;
  }
  const double nd = (double)n;
  const double yW = __ddiv_rn(1.0, W);
  {
    u128 carry = prefix_b;
    for (int w = 0; w < warp; ++w) carry = u128_add(carry, s_wsum[w]);
    // Os of the particle before the warp's first (0 before particle 0)
    int prev_os = ws0 == 0 ? 0 : systematic_Os(u128_to_weight(carry), W, yW, nd, a, n);
    int zeros = 0;
    unsigned long long nq[IT];
    if (ws0 < ws1) {
      const int j0 = ws0 * S + lane * IT;
#pragma unroll
      for (int k = 0; k < IT; ++k) nq[k] = (j0 + k < n) ? __ldcg(qbuf + j0 + k) : 0ull;
    }
    for (int sg = ws0; sg < ws1; ++sg) {
      const int i0 = sg * S + lane * IT;
      unsigned long long q[IT];
      u128 loc = u128_zero();
#pragma unroll
      for (int k = 0; k < IT; ++k) {
        q[k] = nq[k];
        u128 qq; qq.lo = q[k]; qq.hi = 0;
        loc = u128_add(loc, qq);
      }
      if (sg + 1 < ws1) {
#pragma unroll
        for (int k = 0; k < IT; ++k) nq[k] = (i0 + S + k < n) ? __ldcg(qbuf + i0 + S + k) : 0ull;
      }
      const u128 inc = warp_inclusive_u128(loc);
      u128 Q = u128_add(carry, u128_sub(inc, loc));
      int os[IT];
#pragma unroll
      for (int k = 0; k < IT; ++k) {
        u128 qq; qq.lo = q[k]; qq.hi = 0;
        Q = u128_add(Q, qq);
        os[k] = systematic_Os(u128_to_weight(Q), W, yW, nd, a, n);
      }
      const int up = __shfl_up_sync(0xffffffffu, os[IT - 1], 1);
      int prev = lane > 0 ? up : prev_os;
#pragma unroll
      for (int k = 0; k < IT; ++k) {
        if (i0 + k < n) {
          Os[i0 + k] = os[k];
          marks[i0 + k] = 0;
          zeros += (os[k] == prev);
        }
        prev = os[k];
      }
      carry = u128_add(carry, shfl_u128(inc, 31));
      prev_os = __shfl_sync(0xffffffffu, os[IT - 1], 31);
    }
    zeros = warp_inclusive_int(zeros);
    __syncthreads();  // every warp has read s_wsum
    if (lane == 31) s_wint[warp] = zeros;
    __syncthreads();
    if (threadIdx.x == 0) {
      int t = 0;
      for (int w = 0; w < NW; ++w) t += s_wint[w];
      block_z[b] = t;
    }
  }
  if (!grid_barrier(bar_counter, bar_gen, st)) return;

  // phase 3: ranks of childless slots, extra-copy marks, survivors in place
  const int zcarry_b = block_sum_int_from_global(block_z, b);
  const int R = block_sum_int_from_global(block_z, G);
  {
    int zc = zcarry_b;
    for (int w = 0; w < warp; ++w) zc += s_wint[w];
    const int first = ws0 * S;
    int prev_os = (ws0 < ws1 && first > 0) ? __ldcg(Os + first - 1) : 0;
    int nos[IT];
    if (ws0 < ws1) {
#pragma unroll
      for (int k = 0; k < IT; ++k) nos[k] = (first + lane * IT + k < n) ? __ldcg(Os + first + lane * IT + k) : 0;
    }
    for (int sg = ws0; sg < ws1; ++sg) {
      const int i0 = sg * S + lane * IT;
      int os[IT], z[IT];
#pragma unroll
      for (int k = 0; k < IT; ++k) os[k] = nos[k];
      if (sg + 1 < ws1) {
#pragma unroll
        for (int k = 0; k < IT; ++k) nos[k] = (i0 + S + k < n) ? __ldcg(Os + i0 + S + k) : 0;
      }
      const int up = __shfl_up_sync(0xffffffffu, os[IT - 1], 1);
      const int before0 = lane > 0 ? up : prev_os;
      int loc = 0;
      {
        int before = before0;
#pragma unroll
        for (int k = 0; k < IT; ++k) {
          z[k] = (i0 + k < n) && (os[k] == before);
          loc += z[k];
          before = os[k];
        }
      }
      const int inc = warp_inclusive_int(loc);
      int Z = zc + inc - loc;
      int before = before0;
#pragma unroll
      for (int k = 0; k < IT; ++k) {
        const int i = i0 + k;
        if (i < n) {
          // the first further copy of i (if any) has rank E_i = Os_{i-1} - i + Z_i
          if (os[k] - before >= 2) marks[before - i + Z] = i + 1;
          if (z[k]) slot[Z] = i;
          else as[i] = i;
        }
        Z += z[k];
        before = os[k];
      }
      zc += __shfl_sync(0xffffffffu, inc, 31);
      prev_os = __shfl_sync(0xffffffffu, os[IT - 1], 31);
    }
  }
  if (!grid_barrier(bar_counter, bar_gen, st)) return;

  // phase 4: the ancestor of rank r is the last a whose first further copy
  // has rank <= r, i.e. the running maximum of the marks up to r
  const int NR = (R + S - 1) / S;
  const int rb0 = (int)(((long long)b * NR) / G), rb1 = (int)(((long long)(b + 1) * NR) / G);
  int rs0, rs1;
  warp_segments(rb0, rb1, warp, NW, &rs0, &rs1);
  {
    int mloc = 0;
    for (int sg = rs0; sg < rs1; sg += 4) {  // four segments' loads in flight
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int r0 = (sg + u) * S + lane * IT;
#pragma unroll
        for (int k = 0; k < IT; ++k)
          if (sg + u < rs1 && r0 + k < R) mloc = max(mloc, __ldcg(marks + r0 + k));
      }
    }
    mloc = warp_inclusive_max_int(mloc);
    __syncthreads();  // every warp has read s_wint
    if (lane == 31) s_wint[warp] = mloc;
    __syncthreads();
    if (threadIdx.x == 0) {
      int t = 0;
      for (int w = 0; w < NW; ++w) t = max(t, s_wint[w]);
      block_m[b] = t;
    }
  }
  if (!grid_barrier(bar_counter, bar_gen, st)) return;
  {
    int mc = 0;
    for (int j = threadIdx.x; j < b; j += blockDim.x) mc = max(mc, __ldcg(block_m + j));
    mc = block_max_int(mc);
    for (int w = 0; w < warp; ++w) mc = max(mc, s_wint[w]);
    int nm[IT], nsl[IT];
    if (rs0 < rs1) {
      const int q0 = rs0 * S + lane * IT;
#pragma unroll
      for (int k = 0; k < IT; ++k) {
        nm[k] = (q0 + k < R) ? __ldcg(marks + q0 + k) : 0;
        nsl[k] = (q0 + k < R) ? __ldcg(slot + q0 + k) : 0;
      }
    }
    for (int sg = rs0; sg < rs1; ++sg) {
      const int r0 = sg * S + lane * IT;
      int m[IT], sl[IT];
      int run = 0;
#pragma unroll
      for (int k = 0; k < IT; ++k) {
        m[k] = nm[k];
        sl[k] = nsl[k];
        run = max(run, m[k]);
      }
      if (sg + 1 < rs1) {
#pragma unroll
        for (int k = 0; k < IT; ++k) {
          nm[k] = (r0 + S + k < R) ? __ldcg(marks + r0 + S + k) : 0;
          nsl[k] = (r0 + S + k < R) ? __ldcg(slot + r0 + S + k) : 0;
        }
      }
      const int inc = warp_inclusive_max_int(run);
      const int up = __shfl_up_sync(0xffffffffu, inc, 1);
      int ex = max(mc, lane > 0 ? up : 0);
#pragma unroll
      for (int k = 0; k < IT; ++k) {
        ex = max(ex, m[k]);
        if (r0 + k < R) as[sl[k]] = ex - 1;
      }
      mc = max(mc, __shfl_sync(0xffffffffu, inc, 31));
    }
  }
}

// One tile per block (n <= G * NT * IT): each thread keeps its fixed-point
// weights and cumulative offspring in registers across the phases, so after
// the log-weights are read the only global traffic is the G blocks'
// published words, the extra-copy index for the fill, and the ancestors.
// The phases hand over through tagged words (warp_poll_tagged) instead of
// grid barriers: a block publishes its weight total, then its childless
// count, then "E written", and each block's warp 0 polls every block's word
// of the phase, which carries the data it waits for.  NT threads of IT
// particles each: the tile shapes in kCoopShapes, all computing the same
// integers (the shape is chosen by the autotuner below).
// IT log-weights of one thread (16-byte loads when IT is even and aligned)
template <int IT>
__device__ __forceinline__ void load_items(const double* lw, int i0, int n, double (&v)[IT]) {
  if constexpr (IT % 2 == 0) {
    if (i0 + IT <= n && ((reinterpret_cast<uintptr_t>(lw + i0) & 15) == 0)) {
      const double2* p = reinterpret_cast<const double2*>(lw + i0);
#pragma unroll
      for (int k = 0; k < IT / 2; ++k) {
        const double2 t = p[k];
        v[2 * k] = t.x;
        v[2 * k + 1] = t.y;
      }
      return;
    }
  }
#pragma unroll
  for (int k = 0; k < IT; ++k) v[k] = (i0 + k < n) ? lw[i0 + k] : NAN;
}

template <int NT, int IT>
__global__ void __launch_bounds__(NT)
k_systematic_coop1(const double* lw, int n, StepStats* st, const double* a_in, uint64_t seed,
                   int step, int* Os_out, int* as, int* E, int* ecoarse, int coarse_shift, int* slot,
                   unsigned long long* pub, int pub_stride, unsigned* epoch_word, const int* gate) {
  // the next kernel (the transition, a programmatic dependent) may be
  // scheduled now; it waits for this kernel's completion before it reads.
  // This kernel is itself a programmatic dependent of the kernel before it
  // (the transition that wrote the log-weights and the statistics): its
  // blocks may be resident before that kernel has finished, and wait here.
  pdl_trigger();
  pdl_wait();
  if (gate_closed(gate, st)) return;
  // the epoch of this launch, read before this block publishes anything
  const unsigned epoch = ld_relaxed_u32(epoch_word);
  extern __shared__ int s_coarse[];
  __shared__ int s_last[NT];
  __shared__ u128 s_u128[2];
  __shared__ int s_int[2];
  __shared__ int s_ok;
  const int G = gridDim.x, b = blockIdx.x;
  const int i0 = b * (NT * IT) + threadIdx.x * IT;
  const double mx = st->mx;
  double a;
  if (a_in) {
    a = *a_in;
  } else {
    bpf_u32x4 r = bpf_draw(seed, 0u, (uint32_t)step, 0u, BPF_RNG_SYSTEMATIC);
    a = bpf_u01d(r.v[0], r.v[1]);
  }

  // phase 1: fixed-point weights (registers) and the block total
  double v[IT];
  load_items<IT>(lw, i0, n, v);
  unsigned long long q[IT];
  u128 loc = u128_zero();
#pragma unroll
  for (int k = 0; k < IT; ++k) {
    q[k] = (i0 + k < n) ? weight_to_fixed(nanexp(__dsub_rn(v[k], mx))) : 0ull;
    u128 qq; qq.lo = q[k]; qq.hi = 0;
    loc = u128_add(loc, qq);
  }
  u128 btot;
  const u128 texcl = block_exclusive_scan_u128_nt<NT>(loc, &btot);
  if (threadIdx.x == 0) {
    // the total (< 2^80) as three 32-bit payloads
    unsigned long long* mine = pub + (size_t)b * pub_stride;
    st_relaxed_u64(mine + 0, tagged(epoch, (unsigned)btot.lo));
    st_relaxed_u64(mine + 1, tagged(epoch, (unsigned)(btot.lo >> 32)));
    st_relaxed_u64(mine + 2, tagged(epoch, (unsigned)btot.hi));
  }

  // phase 2: block prefix and total W from every block's published total;
  // cumulative offspring (registers)
  if (threadIdx.x < 32) {
    u128 lo = u128_zero(), tot = u128_zero();
    const bool ok = warp_poll_tagged<3>(pub, pub_stride, G, epoch, g_barrier_limit, [&](int i, const unsigned* pl) {
      u128 v;
      v.lo = (unsigned long long)pl[0] | ((unsigned long long)pl[1] << 32);
      v.hi = pl[2];
      tot = u128_add(tot, v);
      if (i < b) lo = u128_add(lo, v);
    });
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
      u128 o1, o2;
      o1.lo = __shfl_xor_sync(0xffffffffu, lo.lo, d);
      o1.hi = __shfl_xor_sync(0xffffffffu, lo.hi, d);
      o2.lo = __shfl_xor_sync(0xffffffffu, tot.lo, d);
      o2.hi = __shfl_xor_sync(0xffffffffu, tot.hi, d);
      lo = u128_add(lo, o1);
      tot = u128_add(tot, o2);
    }
    if (threadIdx.x == 0) {
      s_u128[0] = lo;
      s_u128[1] = tot;
      s_ok = ok;
      // every block has published under this epoch, so every block has
      // read it: the next launch may use the next one
      if (ok && b == 0) *epoch_word = epoch + 1u;
      if (!ok) st->status = BPF_E_TIMEOUT;
    }
  }
  __syncthreads();
  if (!s_ok) return;
  const u128 prefix = s_u128[0], total = s_u128[1];
  const double W = u128_to_weight(total);
  if (!(W > 0.0)) {  // every block sees the same W and leaves here
    if (b == 0 && threadIdx.x == 0) st->status = BPF_E_DEGENERATE;
    return;
  }
  const double nd = (double)n;
  const double yW = __ddiv_rn(1.0, W);
  int os[IT];
  {
    u128 Q = u128_add(prefix, texcl);
#pragma unroll
    for (int k = 0; k < IT; ++k) {
      u128 qq; qq.lo = q[k]; qq.hi = 0;
      Q = u128_add(Q, qq);
      os[k] = systematic_Os(u128_to_weight(Q), W, yW, nd, a, n);
    }
  }
  s_last[threadIdx.x] = os[IT - 1];
  __syncthreads();
  const int before0 = threadIdx.x > 0 ? s_last[threadIdx.x - 1]
                                      : (b == 0 ? 0 : systematic_Os(u128_to_weight(prefix), W, yW, nd, a, n));
  int zl = 0;
  {
    int prev = before0;
#pragma unroll
    for (int k = 0; k < IT; ++k) {
      if (i0 + k < n) {
        zl += (os[k] == prev);
        if (Os_out) Os_out[i0 + k] = os[k];
      }
      prev = os[k];
    }
  }
  int ztot;
  const int zexcl = block_exclusive_scan_int_nt<NT>(zl, &ztot);
  if (threadIdx.x == 0) st_relaxed_u64(pub + (size_t)b * pub_stride + 3, tagged(epoch, (unsigned)ztot));

  // phase 3: ranks of childless slots, E, survivors in place
  if (threadIdx.x < 32) {
    int lo = 0, tot = 0;
    const bool ok = warp_poll_tagged<1>(pub + 3, pub_stride, G, epoch, g_barrier_limit, [&](int i, const unsigned* pl) {
      tot += (int)pl[0];
      if (i < b) lo += (int)pl[0];
    });
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
      lo += __shfl_xor_sync(0xffffffffu, lo, d);
      tot += __shfl_xor_sync(0xffffffffu, tot, d);
    }
    if (threadIdx.x == 0) {
      s_int[0] = lo;
      s_int[1] = tot;
      s_ok = ok;
      if (!ok) st->status = BPF_E_TIMEOUT;
    }
  }
  __syncthreads();
  if (!s_ok) return;
  const int zprefix = s_int[0], R = s_int[1];
  {
    int Z = zprefix + zexcl;
    int prev = before0;
#pragma unroll
    for (int k = 0; k < IT; ++k) {
      const int i = i0 + k;
      if (i < n) {
        const bool zero = os[k] == prev;
        const int e = prev - i + Z;
        E[i] = e;
        if ((i & ((1 << coarse_shift) - 1)) == 0) ecoarse[i >> coarse_shift] = e;
        if (zero) slot[Z] = i;
        else as[i] = i;
        Z += zero;
      }
      prev = os[k];
    }
  }
  // this block's E, coarse entries, slots and survivors are written: publish
  // that (a release, ordered after every thread's writes by the block
  // barrier), then wait for every block's
  __syncthreads();
  if (threadIdx.x == 0) st_release_u64(pub + (size_t)b * pub_stride + 4, tagged(epoch, 1u));
  if (threadIdx.x < 32) {
    const bool ok = warp_poll_tagged<1>(pub + 4, pub_stride, G, epoch, g_barrier_limit, [](int, const unsigned*) {});
    if (threadIdx.x == 0) {
      s_ok = ok;
      if (!ok) st->status = BPF_E_TIMEOUT;
    }
  }
  __syncthreads();
  if (!s_ok) return;

  // phase 4: childless slot of rank r <- ancestor a with E_a <= r < E_{a+1}.
  // The coarse index (every 2^coarse_shift-th E) comes into shared memory
  // with 16-byte loads, all in flight at once; a 16-wide window of E is
  // read as four 16-byte loads and counted in registers instead of four
  // dependent probes
  const int nc = ((n - 1) >> coarse_shift) + 1;
  {
    const int nc4 = nc >> 2;
    const int4* src = reinterpret_cast<const int4*>(ecoarse);
    int4* dst = reinterpret_cast<int4*>(s_coarse);
#pragma unroll 4
    for (int i = threadIdx.x; i < nc4; i += blockDim.x) dst[i] = __ldcg(src + i);
    for (int i = 4 * nc4 + threadIdx.x; i < nc; i += blockDim.x) s_coarse[i] = __ldcg(ecoarse + i);
  }
  __syncthreads();
  for (int r = b * blockDim.x + threadIdx.x; r < R; r += G * blockDim.x) {
    const int sl = __ldcg(slot + r);
    int clo = 0, chi = nc;
    while (clo < chi) {
      int mid = (clo + chi) >> 1;
      if (s_coarse[mid] <= r) clo = mid + 1; else chi = mid;
    }
    int lo = (clo - 1) << coarse_shift;
    int hi = min(n, lo + (1 << coarse_shift));
    if (coarse_shift == 4 && hi - lo == 16) {
      // lo is a multiple of 16: the window is 64-byte aligned
      const int4* w = reinterpret_cast<const int4*>(E + lo);
      int cnt = 0;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int4 e = __ldcg(w + j);
        cnt += (e.x <= r) + (e.y <= r) + (e.z <= r) + (e.w <= r);
      }
      lo += cnt;  // E is nondecreasing: the first index with E > r
    } else {
      while (lo < hi) {
        int mid = (lo + hi) >> 1;
        if (__ldcg(E + mid) <= r) lo = mid + 1; else hi = mid;
      }
    }
    as[sl] = lo - 1;
  }
}

// ---------------------------------------------------------------------------
// cumulative offspring from offspring counts o[] (Metropolis) or from sorted
// ancestors (multinomial), with childless counts per tile
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kBlock)
k_count_tile_sums(const int* __restrict__ o, int n, const StepStats* st, int* icount, int* iprefix,
                  unsigned* counter, const int* gate) {
  if (gate_closed(gate, st)) return;
  const int t = blockIdx.x;
  const int i0 = t * kTile + threadIdx.x * kItems;
  int loc = 0;
#pragma unroll
  for (int k = 0; k < kItems; ++k) loc += (i0 + k < n) ? o[i0 + k] : 0;
  int tot;
  block_exclusive_scan_int(loc, &tot);
  if (threadIdx.x == 0) icount[t] = tot;
  if (last_block_arrive(counter)) {
    block_scan_tiles_int(icount, iprefix, gridDim.x);
    if (threadIdx.x == 0) *counter = 0;
  }
}

// mode 0: o[] are offspring counts, Os = iprefix + inclusive scan
// mode 1: sorted[] are non-decreasing ancestors, Os_i = upper_bound(sorted, i)
__global__ void __launch_bounds__(kBlock)
k_offspring_from(const int* __restrict__ src, int n, int mode, const StepStats* st,
                 const int* iprefix, int* Os, int* zcount, int* zprefix,
                 unsigned* counter, const int* gate) {
  if (gate_closed(gate, st)) return;
  __shared__ int s_last[kBlock];
  const int t = blockIdx.x;
  const int T = gridDim.x;
  const int i0 = t * kTile + threadIdx.x * kItems;
  int os[kItems];
  int first_bound = 0;  // mode 1: the cumulative offspring before the tile
  if (mode == 0) {
    int v[kItems];
    int loc = 0;
#pragma unroll
    for (int k = 0; k < kItems; ++k) { v[k] = (i0 + k < n) ? src[i0 + k] : 0; loc += v[k]; }
    int tot;
    int run = iprefix[t] + block_exclusive_scan_int(loc, &tot);
#pragma unroll
    for (int k = 0; k < kItems; ++k) { run += v[k]; os[k] = run; }
  } else {
    int bound[2];
    block_bounds(src, n, t * kTile - 1, (t + 1) * kTile - 1, bound);
    first_bound = bound[0];
#pragma unroll
    for (int k = 0; k < kItems; ++k) os[k] = upper_bound_in(src, bound[0], bound[1], i0 + k);
  }
  s_last[threadIdx.x] = os[kItems - 1];
  __syncthreads();
  int prev;
  if (threadIdx.x > 0) {
    prev = s_last[threadIdx.x - 1];
  } else if (t == 0) {
    prev = 0;
  } else if (mode == 0) {
    prev = iprefix[t];
  } else {
    prev = first_bound;
  }
  int zeros = 0;
#pragma unroll
  for (int k = 0; k < kItems; ++k) {
    if (i0 + k < n) {
      Os[i0 + k] = os[k];
      zeros += (os[k] == prev);
    }
    prev = os[k];
  }
  int ztot;
  block_exclusive_scan_int(zeros, &ztot);
  if (threadIdx.x == 0) zcount[t] = ztot;
  if (last_block_arrive(counter)) {
    block_scan_tiles_int(zcount, zprefix, T);
    if (threadIdx.x == 0) *counter = 0;
  }
}

// ---------------------------------------------------------------------------
// permutation: the rule of ResamplerHost::cumulativeOffspringToAncestorsPermute
// (share/src/bi/host/resampler/ResamplerHost.hpp:134-168) in closed form.
//   o_i  = Os_i - Os_{i-1};  Z_i = #{m < i : o_m = 0}  (rank of a childless slot)
//   E_i  = #{extra copies of ancestors < i} = Os_{i-1} - i + Z_i
// Particle i with o_i > 0 keeps slot i; the childless slot of rank r receives
// the ancestor a with E_a <= r < E_{a+1}.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kBlock)
k_permute_survivors(const int* __restrict__ Os, int n, const int* zprefix, int* as, int* E, int* slot,
                    const StepStats* st, const int* gate) {
  if (gate_closed(gate, st)) return;
  const int t = blockIdx.x;
  const int i0 = t * kTile + threadIdx.x * kItems;
  int prev = i0 > 0 && i0 - 1 < n ? Os[i0 - 1] : 0;
  int os[kItems];
  int z[kItems];
  int loc = 0;
#pragma unroll
  for (int k = 0; k < kItems; ++k) {
    os[k] = (i0 + k < n) ? Os[i0 + k] : prev;
    z[k] = (i0 + k < n) && (os[k] == (k == 0 ? prev : os[k - 1]));
    loc += z[k];
  }
  int tot;
  int Z = zprefix[t] + block_exclusive_scan_int(loc, &tot);
#pragma unroll
  for (int k = 0; k < kItems; ++k) {
    int i = i0 + k;
    int before = (k == 0 ? prev : os[k - 1]);
    if (i < n) {
      const int e = before - i + Z;
      E[i] = e;
      if (z[k]) slot[Z] = i;
      else as[i] = i;
    }
    Z += z[k];
  }
}

// Childless slot of rank r receives the ancestor a with E_a <= r < E_{a+1}.
// One thread per rank, so the work is balanced however the copies are
// distributed.  Bound by the latency of the search's dependent loads: the
// part of E that brackets a block's ranks is fetched into shared memory when
// it fits (256 or 1024 ranks lie among some 700 or 2600 particles).
constexpr int kStage = 4096;
template <int K>
__global__ void __launch_bounds__(kBlock)
k_permute_fill(int* as, const int* __restrict__ E, const int* __restrict__ slot, const int* zprefix, int n, int T,
               const StepStats* st, const int* gate) {
  if (gate_closed(gate, st)) return;
  __shared__ int s_E[kStage];
  const int R = zprefix[T];
  constexpr int kSpan = kBlock * K;
  for (long long b0 = (long long)blockIdx.x * kSpan; b0 < R; b0 += (long long)gridDim.x * kSpan) {
    int r[K], b[K], to[K], bound[2];
#pragma unroll
    for (int k = 0; k < K; ++k) {
      r[k] = (int)min(b0 + k * kBlock + threadIdx.x, (long long)R - 1);
      to[k] = __ldg(slot + r[k]);
    }
    block_bounds(E, n, (int)b0, (int)min(b0 + kSpan, (long long)R) - 1, bound);
    const int len = bound[1] - bound[0];
    if (len <= kStage) {
      for (int i = threadIdx.x; i < len; i += kBlock) s_E[i] = __ldg(E + bound[0] + i);
      __syncthreads();
      upper_bounds_between(s_E, 0, len, r, b);
#pragma unroll
      for (int k = 0; k < K; ++k) b[k] += bound[0];
    } else {
      upper_bounds_between(E, bound[0], len, r, b);
    }
#pragma unroll
    for (int k = 0; k < K; ++k) as[to[k]] = b[k] - 1;
  }
}

// Unpermuted: as_j = i for Os_{i-1} <= j < Os_i, i.e. upper_bound(Os, j)
// (ResamplerHost::cumulativeOffspringToAncestors, ResamplerHost.hpp:110-131).
template <int K>
__global__ void __launch_bounds__(kBlock)
k_ancestors_from_Os(const int* __restrict__ Os, int n, int* as, const StepStats* st, const int* gate) {
  if (gate_closed(gate, st)) return;
  constexpr int kSpan = kBlock * K;
  for (long long b0 = (long long)blockIdx.x * kSpan; b0 < n; b0 += (long long)gridDim.x * kSpan) {
    int j[K], b[K];
#pragma unroll
    for (int k = 0; k < K; ++k) j[k] = (int)min(b0 + k * kBlock + threadIdx.x, (long long)n - 1);
    block_upper_bounds(Os, n, j, (int)b0, (int)min(b0 + kSpan, (long long)n) - 1, b);
#pragma unroll
    for (int k = 0; k < K; ++k) as[j[k]] = b[k] < n ? b[k] : n - 1;  // Os[n-1] == n for valid offsets; bounds any other
  }
}

// ---------------------------------------------------------------------------
// multinomial (sorted draws, Bentley & Saxe 1979), following
// MultinomialResamplerHost::ancestors (MultinomialResamplerHost.hpp:29-65)
// with one host thread: slot s gets the number of m with log(Ws_m) <= lu_s,
// lu_s = log(W) + lMax_s, lMax_s = sum_{i > s} log(u)/i.
// ---------------------------------------------------------------------------
// Ws: the fixed-point weights in, the logarithms of the cumulative weights
// out; lu: the spacings in, the log uniforms out (each thread's own entries,
// which the buffers' alignment allows in 16-byte pairs).
template <int ITEMS>
__global__ void __launch_bounds__(kBlock)
k_multinomial_prepare(int n, const StepStats* st, const u128* tile_prefix, const u128* vtile_prefix, double* Ws,
                      double* lu, const int* gate) {
  static_assert(ITEMS % 2 == 0, "entries in pairs");
  if (gate_closed(gate, st)) return;
  const int t = blockIdx.x;
  const int T = gridDim.x;
  const long long i0 = (long long)t * (kBlock * ITEMS) + threadIdx.x * ITEMS;
  const double lW = log(u128_to_weight(tile_prefix[T]));
  const u128 Vtot = vtile_prefix[T];
  unsigned long long q[ITEMS];
  double sp[ITEMS];
  u128 loc = u128_zero(), vloc = u128_zero();
  if (i0 + ITEMS <= n) {
#pragma unroll
    for (int k = 0; k < ITEMS; k += 2) {
      const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(Ws + i0 + k);
      const double2 b = *reinterpret_cast<const double2*>(lu + i0 + k);
      q[k] = a.x; q[k + 1] = a.y;
      sp[k] = b.x; sp[k + 1] = b.y;
    }
  } else {
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
      q[k] = i0 + k < n ? reinterpret_cast<const unsigned long long*>(Ws)[i0 + k] : 0ull;
      sp[k] = i0 + k < n ? lu[i0 + k] : 0.0;
    }
  }
#pragma unroll
  for (int k = 0; k < ITEMS; ++k) {
    u128 qq; qq.lo = q[k]; qq.hi = 0;
    loc = u128_add(loc, qq);
    vloc = u128_add(vloc, spacing_to_fixed(sp[k]));
  }
  u128 tot, vtot;
  u128 Q = u128_add(tile_prefix[t], block_exclusive_scan_u128(loc, &tot));
  u128 V = u128_add(vtile_prefix[t], block_exclusive_scan_u128(vloc, &vtot));
#pragma unroll
  for (int k = 0; k < ITEMS; k += 2) {
    double2 w, l;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      u128 qq; qq.lo = q[k + j]; qq.hi = 0;
      Q = u128_add(Q, qq);
      const double lq = log(u128_to_weight(Q));
      // suffix sum over slots >= s of the spacings, then lu = lW + lMax
      const double ls = __dadd_rn(lW, -fixed_to_spacing(u128_sub(Vtot, V)));
      V = u128_add(V, spacing_to_fixed(sp[k + j]));
      (j ? w.y : w.x) = lq;
      (j ? l.y : l.x) = ls;
    }
    if (i0 + k + 2 <= n) {
      *reinterpret_cast<double2*>(Ws + i0 + k) = w;
      *reinterpret_cast<double2*>(lu + i0 + k) = l;
    } else if (i0 + k < n) {
      Ws[i0 + k] = w.x;
      lu[i0 + k] = l.x;
    }
  }
}

// Bound by the latency of the searches' loads from L2: one bracketing and one
// round of ten dependent loads per 1024 slots, all blocks of 10^6 particles
// resident at once: 13.2 us against 21.9 with one slot per thread.
template <int K>
__global__ void __launch_bounds__(kBlock)
k_multinomial_search(const double* __restrict__ lWs, const double* __restrict__ lu, int n, int* as,
                     const StepStats* st, const int* gate) {
  if (gate_closed(gate, st)) return;
  constexpr int kSpan = kBlock * K;
  for (long long b0 = (long long)blockIdx.x * kSpan; b0 < n; b0 += (long long)gridDim.x * kSpan) {
    const int base = (int)b0;
    int s[K], b[K];
    double x[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
      s[k] = (int)min(b0 + k * kBlock + threadIdx.x, (long long)n - 1);
      x[k] = __ldg(lu + s[k]);
    }
    block_upper_bounds(lWs, n, x, __ldg(lu + base), __ldg(lu + (int)min(b0 + kSpan, (long long)n) - 1), b);
    // the reference's loop can leave j = n when lu rounds up to log(W); clamp
#pragma unroll
    for (int k = 0; k < K; ++k) as[s[k]] = b[k] < n ? b[k] : n - 1;
  }
}

// ---------------------------------------------------------------------------
// Metropolis, following MetropolisResamplerHost::ancestors
// (share/src/bi/host/resampler/MetropolisResamplerHost.hpp:290-321): B steps
// per particle; draw k uses (u_int, u_acc) = uniforms[2(p*B+k)], [2(p*B+k)+1].
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kBlock)
k_metropolis(const double* __restrict__ lw, int n, int B, const double* u, uint64_t seed, int step,
             int* as, int* o, const StepStats* st, const int* gate) {
  if (gate_closed(gate, st)) return;
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
    const int p1 = metropolis_ancestor(lw, n, B, u, seed, step, p);
    as[p] = p1;
    if (o) atomicAdd(o + p1, 1);
  }
}

// ---------------------------------------------------------------------------
// gather_rows, out of place: Y[j*ld + i] = X[j*ld + as[i]]
// ---------------------------------------------------------------------------
template <class T>
__global__ void __launch_bounds__(kBlock)
k_gather(const int* __restrict__ as, const T* __restrict__ X, T* __restrict__ Y, int n, int d, int ld,
         const int* gate) {
  if (gate != nullptr && *gate == 0) return;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int a = as[i];
  if (a < 0 || a >= n) return;  // an ancestor out of range leaves the row untouched
  for (int j = 0; j < d; ++j) Y[(size_t)j * ld + i] = __ldg(X + (size_t)j * ld + a);
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
// the last-block tickets and grid-barrier words back to zero, and the
// one-launch kernel's epoch one further: the published words of a launch
// that timed out (or of any earlier launch) then carry an epoch no later
// launch uses, whatever state that launch left them in
__global__ void k_reset_scratch_words(unsigned* counters) {
  const int i = threadIdx.x;
  if (i < kEpochWord) counters[i] = 0u;
  if (i == kEpochWord) counters[i] += 1u;
}

int reset_scratch_words(ResampleScratch& s, cudaStream_t st) {
  k_reset_scratch_words<<<1, 32, 0, st>>>(s.counters);
  BPF_TRY(cudaGetLastError());
  return BPF_OK;
}

int scratch_alloc(ResampleScratch& s, int max_n) {
  s.max_n = max_n;
  s.max_tiles = ntiles(max_n);
  const size_t T1 = (size_t)s.max_tiles + 1;
  const size_t N = (size_t)max_n;
  // one partial per block of the widest per-step grid (64-thread transition blocks)
  s.max_partials = (max_n + 63) / 64 + 1;
#define ALLOC(ptr, bytes) \
  if (cudaMalloc((void**)&(ptr), (bytes)) != cudaSuccess) { scratch_free(s); return BPF_E_NOMEM; }
  ALLOC(s.tile_sum, T1 * sizeof(u128));
  ALLOC(s.tile_prefix, T1 * sizeof(u128));
  ALLOC(s.vtile_sum, T1 * sizeof(u128));
  ALLOC(s.vtile_prefix, T1 * sizeof(u128));
  ALLOC(s.zcount, T1 * sizeof(int));
  ALLOC(s.zprefix, T1 * sizeof(int));
  ALLOC(s.icount, T1 * sizeof(int));
  ALLOC(s.iprefix, T1 * sizeof(int));
  ALLOC(s.Os, N * sizeof(int));
  ALLOC(s.E, N * sizeof(int));
  ALLOC(s.slot, N * sizeof(int));
  ALLOC(s.etile, (N / 16 + 2) * sizeof(int));
  ALLOC(s.o, N * sizeof(int));
  ALLOC(s.Ws, N * sizeof(double));
  ALLOC(s.lu, N * sizeof(double));
  ALLOC(s.counters, 16 * sizeof(unsigned));
  ALLOC(s.stats, sizeof(StepStats));
  ALLOC(s.partials, (size_t)s.max_partials * sizeof(LwPartial));
  s.pub_entries = pub_entries_for(max_n);
  ALLOC(s.pub, (size_t)s.pub_entries * kPubWords * sizeof(unsigned long long));
#undef ALLOC
  if (cudaMemset(s.counters, 0, 16 * sizeof(unsigned)) != cudaSuccess) { scratch_free(s); return BPF_E_CUDA; }
  // tags no epoch carries (the epoch starts at zero)
  if (cudaMemset(s.pub, 0xFF, (size_t)s.pub_entries * kPubWords * sizeof(unsigned long long)) != cudaSuccess) {
    scratch_free(s);
    return BPF_E_CUDA;
  }
  StepStats z{};
  z.status = BPF_OK;
  if (cudaMemcpy(s.stats, &z, sizeof(z), cudaMemcpyHostToDevice) != cudaSuccess) { scratch_free(s); return BPF_E_CUDA; }
  return BPF_OK;
}

void scratch_free(ResampleScratch& s) {
  void* ptrs[] = {s.tile_sum, s.tile_prefix, s.vtile_sum, s.vtile_prefix, s.zcount, s.zprefix,
                  s.icount, s.iprefix, s.Os, s.E, s.slot, s.etile, s.o, s.Ws, s.lu, s.counters, s.stats, s.partials,
                  s.pub};
  for (void* p : ptrs) if (p) cudaFree(p);
  s = ResampleScratch();
}

// coarse index stride: the smallest power of two >= 16 that keeps the index
// within max_entries entries
static inline int coarse_shift(int n, int max_entries) {
  int sh = 4;
  while ((((long long)n + (1ll << sh) - 1) >> sh) > max_entries) ++sh;
  return sh;
}

static inline size_t fill_smem(int n, int max_entries) {
  return (size_t)(((n - 1) >> coarse_shift(n, max_entries)) + 1) * sizeof(int);
}

// the cooperative kernel keeps its coarse index within 32 KB, leaving room
// for its static shared memory under the default 48 KB limit
constexpr int kMaxCoarseCoop = 8192;
// items per thread of the multi-tile cooperative kernel (tiles of 512)
constexpr int kCoopItems = 2;

static int launch_systematic_coop(const ResampleArgs& a, ResampleScratch& s, int* Os, cudaStream_t st);

static inline int grid_stride_blocks(int n) {
  int b = (n + kBlock - 1) / kBlock;
  return b < 148 * 8 ? (b > 0 ? b : 1) : 148 * 8;
}

// The kernels that search for each slot, with K searches per thread: one
// while all blocks are resident at once (148 SMs x 8), kWide beyond, so that
// a block's bracketing serves more slots and its searches overlap.
constexpr int kWide = 4;
template <class... KArgs, class... Args>
static void launch_searched(void (*one)(KArgs...), void (*wide)(KArgs...), int n, cudaStream_t st, Args... args) {
  const int blocks = (n + kBlock - 1) / kBlock, resident = 148 * 8;
  if (blocks <= resident)
    one<<<blocks, kBlock, 0, st>>>(args...);
  else
    wide<<<std::min((blocks + kWide - 1) / kWide, resident), kBlock, 0, st>>>(args...);
}

// The multinomial resampler's cumulative weights and log uniforms, in tiles
// of kBlock * ITEMS particles.  More particles per thread make fewer block
// sums and scans and fewer tiles for the last block to scan alone, fewer make
// more blocks.  A whole sorted resampling on B200 with 2 / 4 / 8 per thread:
// 56 / 57 / 64 us at 2^17 particles, 67 / 62 / 68 at 2^18, 72 / 70 / 67 at
// 2^19, 94 / 93 / 93 at 10^6, 245 / 217 / 207 at 2^22.
constexpr int kMultinomial4From = 1 << 18, kMultinomial8From = 1 << 19;
template <int ITEMS>
static void launch_multinomial_draws(const ResampleArgs& a, ResampleScratch& s, cudaStream_t st) {
  const int tiles = (a.n + kBlock * ITEMS - 1) / (kBlock * ITEMS);
  k_weight_tile_sums<ITEMS, true><<<tiles, kBlock, 0, st>>>(a.lw, a.n, s.stats, s.tile_sum, s.tile_prefix, a.uniforms,
                                                            a.seed, a.step, s.vtile_sum, s.vtile_prefix,
                                                            reinterpret_cast<unsigned long long*>(s.Ws), s.lu,
                                                            s.counters, a.gate);
  k_multinomial_prepare<ITEMS><<<tiles, kBlock, 0, st>>>(a.n, s.stats, s.tile_prefix, s.vtile_prefix, s.Ws, s.lu,
                                                         a.gate);
}

int launch_resample(const ResampleArgs& a, ResampleScratch& s, cudaStream_t st) {
  if (a.n <= 0 || a.n > s.max_n || a.as == nullptr) return BPF_E_INVALID;
  const int n = a.n;
  const int T = ntiles(n);
  int* Os = a.Os_out ? a.Os_out : s.Os;
  unsigned* c = s.counters;
  if (!a.max_known && a.kind != BPF_RESAMPLER_METROPOLIS) {
    // up to four blocks per SM, at least 2048 log-weights each
    int blocks = (n + 2047) / 2048;
    if (blocks > 148 * 4) blocks = 148 * 4;
    if (blocks > s.max_partials) blocks = s.max_partials;
    k_lw_max<<<blocks, kBlock, 0, st>>>(a.lw, n, s.partials, s.stats, s.counters);
    BPF_TRY(cudaGetLastError());
  }
  switch (a.kind) {
    case BPF_RESAMPLER_SYSTEMATIC: {
      if (a.permute) {
        int rc = launch_systematic_coop(a, s, a.Os_out, st);
        if (rc != BPF_E_INVALID) return rc;  // BPF_E_INVALID: cooperative launch unavailable, use the passes
      }
      k_weight_tile_sums<kItems, false><<<T, kBlock, 0, st>>>(a.lw, n, s.stats, s.tile_sum, s.tile_prefix, nullptr,
                                                              a.seed, a.step, nullptr, nullptr, nullptr, nullptr, c + 0,
                                                              a.gate);
      k_systematic_offspring<<<T, kBlock, 0, st>>>(a.lw, n, s.stats, s.tile_prefix, a.uniforms, a.seed,
                                                   a.step, Os, s.zcount, s.zprefix, c + 1, a.gate);
      if (a.permute) {
        k_permute_survivors<<<T, kBlock, 0, st>>>(Os, n, s.zprefix, a.as, s.E, s.slot, s.stats, a.gate);
        launch_searched(k_permute_fill<1>, k_permute_fill<kWide>, n, st, a.as, s.E, s.slot, s.zprefix, n, T,
                        s.stats, a.gate);
      } else {
        launch_searched(k_ancestors_from_Os<1>, k_ancestors_from_Os<kWide>, n, st, (const int*)Os, n, a.as, s.stats, a.gate);
      }
      break;
    }
    case BPF_RESAMPLER_MULTINOMIAL: {
      if (n >= kMultinomial8From) launch_multinomial_draws<8>(a, s, st);
      else if (n >= kMultinomial4From) launch_multinomial_draws<4>(a, s, st);
      else launch_multinomial_draws<2>(a, s, st);
      launch_searched(k_multinomial_search<1>, k_multinomial_search<kWide>, n, st, (const double*)s.Ws, (const double*)s.lu, n, a.as,
                      s.stats, a.gate);
      if (a.permute || a.Os_out) {
        k_offspring_from<<<T, kBlock, 0, st>>>(a.as, n, 1, s.stats, nullptr, Os, s.zcount, s.zprefix, c + 1,
                                               a.gate);
      }
      if (a.permute) {
        k_permute_survivors<<<T, kBlock, 0, st>>>(Os, n, s.zprefix, a.as, s.E, s.slot, s.stats, a.gate);
        launch_searched(k_permute_fill<1>, k_permute_fill<kWide>, n, st, a.as, s.E, s.slot, s.zprefix, n, T,
                        s.stats, a.gate);
      }
      break;
    }
    case BPF_RESAMPLER_METROPOLIS: {
      const bool need_counts = a.permute || a.Os_out;
      if (need_counts) BPF_TRY(cudaMemsetAsync(s.o, 0, (size_t)n * sizeof(int), st));
      k_metropolis<<<grid_stride_blocks(n), kBlock, 0, st>>>(a.lw, n, a.B, a.uniforms, a.seed, a.step, a.as,
                                                            need_counts ? s.o : nullptr, s.stats, a.gate);
      if (need_counts) {
        k_count_tile_sums<<<T, kBlock, 0, st>>>(s.o, n, s.stats, s.icount, s.iprefix, c + 2, a.gate);
        k_offspring_from<<<T, kBlock, 0, st>>>(s.o, n, 0, s.stats, s.iprefix, Os, s.zcount, s.zprefix, c + 1,
                                               a.gate);
      }
      if (a.permute) {
        k_permute_survivors<<<T, kBlock, 0, st>>>(Os, n, s.zprefix, a.as, s.E, s.slot, s.stats, a.gate);
        launch_searched(k_permute_fill<1>, k_permute_fill<kWide>, n, st, a.as, s.E, s.slot, s.zprefix, n, T,
                        s.stats, a.gate);
      }
      break;
    }
    default:
      return BPF_E_INVALID;
  }
  BPF_TRY(cudaGetLastError());
  return BPF_OK;
}

// Cooperative launch of k_systematic_coop over at most as many blocks as the
// GPU holds at once (and at most one per tile).  Returns BPF_E_INVALID when a
// cooperative launch is not possible, so the caller can run the passes.
// ---------------------------------------------------------------------------
// tile shapes of the one-launch resampler and their autotuner
// ---------------------------------------------------------------------------
struct CoopShape {
  int nt, it;        // threads per block, particles per thread
  const void* fn;    // the kernel instantiation
};
// every tile holds at least kTile particles, so the block totals fit the
// scratch sized for kTile tiles
static const CoopShape kCoopShapes[BPF_RESAMPLE_SHAPES] = {
    {256, 2, (const void*)k_systematic_coop1<256, 2>}, {128, 4, (const void*)k_systematic_coop1<128, 4>},
    {512, 1, (const void*)k_systematic_coop1<512, 1>}, {512, 2, (const void*)k_systematic_coop1<512, 2>},
    {256, 4, (const void*)k_systematic_coop1<256, 4>}, {1024, 1, (const void*)k_systematic_coop1<1024, 1>},
};

// process-wide autotuned shape per device and size class (ceil log2 n);
// -1: not tuned, -2: no shape fits in one wave (the default shape 0, or
// the multi-tile kernel, is used for both)
static std::mutex g_tune_mu;
static int g_tuned[16][32];
static bool g_tuned_init = false;

static int size_class(int n) {
  int c = 0;
  while (c < 31 && (1 << c) < n) ++c;
  return c;
}

static int tuned_shape(int dev, int n) {
  std::lock_guard<std::mutex> lk(g_tune_mu);
  if (!g_tuned_init) {
    for (auto& row : g_tuned)
      for (int& v : row) v = -1;
    g_tuned_init = true;
  }
  return dev >= 0 && dev < 16 ? g_tuned[dev][size_class(n)] : -1;
}

static void set_tuned_shape(int dev, int n, int shape) {
  tuned_shape(dev, n);  // initialises the table
  std::lock_guard<std::mutex> lk(g_tune_mu);
  if (dev >= 0 && dev < 16) g_tuned[dev][size_class(n)] = shape;
}

// Device attributes and occupancies of the cooperative launches, kept per
// device: a process may drive several GPUs (one handle per host thread), so
// nothing here may come from whichever device happened to be current first.
// The launch is on every filter step, hence the cache.
constexpr int kMaxCoopDevices = 64;
struct CoopDevice {
  bool init = false;
  int coop = 0, sms = 0;
  int per_sm_multi = 0;                      // k_systematic_coop blocks per SM
  size_t smem[BPF_RESAMPLE_SHAPES] = {};     // shared memory the cached occupancy is for
  int per[BPF_RESAMPLE_SHAPES] = {};         // resident blocks per SM of each shape
  bool have[BPF_RESAMPLE_SHAPES] = {};
};
static std::mutex g_coop_mu;
static CoopDevice g_coop[kMaxCoopDevices];

// the current device's entry, filled on first use
static int coop_device(int* dev_out, CoopDevice** out) {
  int dev = 0;
  BPF_TRY(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxCoopDevices) return BPF_E_INVALID;
  std::lock_guard<std::mutex> lk(g_coop_mu);
  CoopDevice& d = g_coop[dev];
  if (!d.init) {
    BPF_TRY(cudaDeviceGetAttribute(&d.coop, cudaDevAttrCooperativeLaunch, dev));
    BPF_TRY(cudaDeviceGetAttribute(&d.sms, cudaDevAttrMultiProcessorCount, dev));
    BPF_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&d.per_sm_multi, k_systematic_coop<kCoopItems>, kBlock, 0));
    d.init = true;
  }
  *dev_out = dev;
  *out = &d;
  return BPF_OK;
}

// resident blocks per SM of shape k at a dynamic shared-memory size on the
// device of entry d
static int shape_per_sm(CoopDevice& d, int k, size_t smem) {
  std::lock_guard<std::mutex> lk(g_coop_mu);
  if (!d.have[k] || d.smem[k] != smem) {
    int v = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, kCoopShapes[k].fn, kCoopShapes[k].nt, smem) != cudaSuccess) {
      cudaGetLastError();
      v = 0;
    }
    d.per[k] = v;
    d.smem[k] = smem;
    d.have[k] = true;
  }
  return d.per[k];
}

// launch shape k of the one-launch kernel if its tiles fit the GPU in one
// wave; BPF_E_INVALID when they do not
static int launch_coop1_shape(int k, const ResampleArgs& a, ResampleScratch& s, int* Os_out, CoopDevice& d,
                              cudaStream_t st) {
  const int n = a.n;
  const int tile = kCoopShapes[k].nt * kCoopShapes[k].it;
  const int G = (n + tile - 1) / tile;
  const size_t smem = fill_smem(n, kMaxCoarseCoop);
  if (G < 1 || G > d.sms * shape_per_sm(d, k, smem)) return BPF_E_INVALID;
  int sh = coarse_shift(n, kMaxCoarseCoop);
  const double* lw = a.lw;
  StepStats* stats = s.stats;
  const double* a_in = a.uniforms;
  uint64_t seed = a.seed;
  int step = a.step;
  int* as = a.as;
  int* E = s.E;
  int* ec = s.etile;
  int* slot = s.slot;
  unsigned long long* pub = s.pub;  // G blocks' published words
  int pstride = kPubWords;
  unsigned* ew = s.counters + kEpochWord;
  const int* gate = a.gate;
  int nn = n;
  int* Oo = Os_out;
  if (!pub || G > s.pub_entries) return BPF_E_INVALID;
  void* args[] = {(void*)&lw, (void*)&nn, (void*)&stats, (void*)&a_in, (void*)&seed, (void*)&step, (void*)&Oo,
                  (void*)&as, (void*)&E, (void*)&ec, (void*)&sh, (void*)&slot, (void*)&pub, (void*)&pstride,
                  (void*)&ew, (void*)&gate};
  // cooperative (every block resident: the blocks poll each other's
  // words) and a programmatic dependent of the kernel before it
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.gridDim = dim3((unsigned)G);
  cfg.blockDim = dim3((unsigned)kCoopShapes[k].nt);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = at;
  cfg.numAttrs = 2;
  BPF_TRY(cudaLaunchKernelExC(&cfg, kCoopShapes[k].fn, args));
  return BPF_OK;
}

// Systematic resampling in one cooperative launch when the GPU can hold the
// grid; BPF_E_INVALID when a cooperative launch is not possible, so the
// caller can run the passes.
static int launch_systematic_coop(const ResampleArgs& a, ResampleScratch& s, int* Os_out, cudaStream_t st) {
  int dev = 0;
  CoopDevice* d = nullptr;
  int rc = coop_device(&dev, &d);
  if (rc) return rc;
  if (!d->coop) return BPF_E_INVALID;
  const int n = a.n;
  // one tile per block: the pinned shape, else the autotuned one, else the
  // default; then any other shape that fits
  int first = a.shape >= 0 && a.shape < BPF_RESAMPLE_SHAPES ? a.shape : tuned_shape(dev, n);
  if (first < 0) first = 0;  // untuned, or nothing fits (the loop below then falls through)
  rc = launch_coop1_shape(first, a, s, Os_out, *d, st);
  for (int k = 0; rc == BPF_E_INVALID && k < BPF_RESAMPLE_SHAPES; ++k)
    if (k != first) rc = launch_coop1_shape(k, a, s, Os_out, *d, st);
  if (rc != BPF_E_INVALID) return rc;
  // several tiles per block
  const int sms = d->sms, per_sm = d->per_sm_multi;
  const int T8 = (n + kBlock * kCoopItems - 1) / (kBlock * kCoopItems);  // tiles of the multi-tile variant
  int G = sms * per_sm;
  if (G > T8) G = T8;
  if (G < 1) return BPF_E_INVALID;
  // the multi-tile variant also needs marks, stored weights and block maxima
  if (s.o == nullptr || s.Ws == nullptr || s.icount == nullptr) return BPF_E_INVALID;
  const double* lw = a.lw;
  StepStats* stats = s.stats;
  const double* a_in = a.uniforms;
  uint64_t seed = a.seed;
  int step = a.step;
  int* as = a.as;
  int* slot = s.slot;
  u128* bw = s.tile_sum;
  int* bz = s.zcount;
  unsigned* bc = s.counters + 8;
  unsigned* bg = s.counters + 9;
  const int* gate = a.gate;
  int nn = n;
  int* Os = Os_out ? Os_out : s.Os;  // the multi-tile variant keeps Os in global memory
  int* marks = s.o;     // n ints
  int* bm = s.icount;   // G <= T block maxima
  unsigned long long* qb = reinterpret_cast<unsigned long long*>(s.Ws);  // n fixed-point weights
  void* args[] = {(void*)&lw, (void*)&nn, (void*)&stats, (void*)&a_in, (void*)&seed, (void*)&step, (void*)&Os,
                  (void*)&as, (void*)&marks, (void*)&slot, (void*)&qb, (void*)&bw, (void*)&bz, (void*)&bm,
                  (void*)&bc, (void*)&bg, (void*)&gate};
  BPF_TRY(cudaLaunchCooperativeKernel((const void*)k_systematic_coop<kCoopItems>, dim3(G), dim3(kBlock), args, 0,
                                      st));
  return BPF_OK;
}

// seeded synthetic log-weights N(0, 2^2), the bench's distribution
__global__ void k_synthetic_lw(double* lw, int n) {
  const int i = 2 * (blockIdx.x * blockDim.x + threadIdx.x);
  if (i >= n) return;
  const bpf_u32x4 r = bpf_draw(0x5eedull, (uint32_t)i, 0u, 0u, BPF_RNG_DATA);
  double z0, z1;
  bpf_normal_pair_d(r.v[0], r.v[1], &z0, &z1);
  lw[i] = 2.0 * z0;
  if (i + 1 < n) lw[i + 1] = 2.0 * z1;
}

int autotune_systematic(int n, cudaStream_t st, int* best, double* us) {
  if (n <= 0 || !best) return BPF_E_INVALID;
  *best = -1;
  for (int k = 0; k < BPF_RESAMPLE_SHAPES; ++k)
    if (us) us[k] = 0.0;
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  BPF_TRY(cudaStreamIsCapturing(st, &cs));
  if (cs != cudaStreamCaptureStatusNone) return BPF_E_INVALID;  // no timing inside a capture
  int dev = 0;
  CoopDevice* d = nullptr;
  {
    const int drc = coop_device(&dev, &d);
    if (drc) return drc;
  }
  if (!d->coop) return BPF_E_INVALID;
  // nothing to time when no shape holds n particles in one wave
  bool any = false;
  for (int k = 0; k < BPF_RESAMPLE_SHAPES; ++k) {
    const int tile = kCoopShapes[k].nt * kCoopShapes[k].it;
    any |= (n + tile - 1) / tile <= d->sms * shape_per_sm(*d, k, fill_smem(n, kMaxCoarseCoop));
  }
  if (!any) {
    set_tuned_shape(dev, n, -2);
    return BPF_E_INVALID;
  }
  ResampleScratch s;
  double* lw = nullptr;
  int* as = nullptr;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  int rc = scratch_alloc(s, n);
  if (!rc && (cudaMalloc((void**)&lw, (size_t)n * sizeof(double)) != cudaSuccess ||
              cudaMalloc((void**)&as, (size_t)n * sizeof(int)) != cudaSuccess))
    rc = BPF_E_NOMEM;
  if (!rc && (cudaEventCreate(&e0) != cudaSuccess || cudaEventCreate(&e1) != cudaSuccess)) rc = BPF_E_CUDA;
  if (!rc) {
    k_synthetic_lw<<<(n / 2 + 256) / 256, 256, 0, st>>>(lw, n);
    if (cudaGetLastError() != cudaSuccess) rc = BPF_E_CUDA;
  }
  if (!rc) rc = launch_lw_reduce(lw, n, s, st);  // the maximum the kernels read
  ResampleArgs a{};
  a.kind = BPF_RESAMPLER_SYSTEMATIC;
  a.n = n;
  a.lw = lw;
  a.seed = 1;
  a.step = 1;
  a.permute = 1;
  a.as = as;
  a.max_known = true;
  a.shape = -1;
  // the shapes take turns, round after round, so that a drift of clocks or
  // caches during the tuning reaches every shape alike; each shape's median
  // decides
  constexpr int kReps = 15;
  float t[BPF_RESAMPLE_SHAPES][kReps];
  bool fits[BPF_RESAMPLE_SHAPES];
  for (int k = 0; k < BPF_RESAMPLE_SHAPES; ++k) fits[k] = true;
  for (int r = -2; !rc && r < kReps; ++r) {  // two untimed rounds first
    for (int k = 0; !rc && k < BPF_RESAMPLE_SHAPES; ++k) {
      if (!fits[k]) continue;
      if (r >= 0 && cudaEventRecord(e0, st) != cudaSuccess) { rc = BPF_E_CUDA; break; }
      const int krc = launch_coop1_shape(k, a, s, nullptr, *d, st);
      if (krc == BPF_E_INVALID) { fits[k] = false; continue; }  // this shape does not fit in one wave
      if (krc) { rc = krc; break; }
      if (r >= 0 && (cudaEventRecord(e1, st) != cudaSuccess || cudaEventSynchronize(e1) != cudaSuccess ||
                     cudaEventElapsedTime(&t[k][r], e0, e1) != cudaSuccess))
        rc = BPF_E_CUDA;
    }
  }
  double best_us = 0.0;
  for (int k = 0; !rc && k < BPF_RESAMPLE_SHAPES; ++k) {
    if (!fits[k]) continue;
    std::sort(t[k], t[k] + kReps);
    const double med = 1e3 * t[k][kReps / 2];
    if (us) us[k] = med;
    if (*best < 0 || med < best_us) { *best = k; best_us = med; }
  }
  if (!rc && cudaStreamSynchronize(st) != cudaSuccess) rc = BPF_E_CUDA;
  if (!rc) {
    // the kernels report problems in the status word
    StepStats hs{};
    if (cudaMemcpy(&hs, s.stats, sizeof(StepStats), cudaMemcpyDeviceToHost) != cudaSuccess) rc = BPF_E_CUDA;
    else if (hs.status != BPF_OK) rc = hs.status;
  }
  if (!rc && *best >= 0) set_tuned_shape(dev, n, *best);
  if (e0) cudaEventDestroy(e0);
  if (e1) cudaEventDestroy(e1);
  if (lw) cudaFree(lw);
  if (as) cudaFree(as);
  scratch_free(s);
  if (rc) cudaGetLastError();
  return rc ? rc : (*best >= 0 ? BPF_OK : BPF_E_INVALID);
}

// host copy of each device's limit, for kernels that take it as an argument
static long long g_host_limit[64];
static bool g_host_limit_init = false;
static std::mutex g_limit_mu;

int set_barrier_limit(long long cycles) {
  int dev = 0;
  BPF_TRY(cudaGetDevice(&dev));
  BPF_TRY(cudaMemcpyToSymbol(g_barrier_limit, &cycles, sizeof(cycles)));
  barrier_limit();  // initialises the table
  std::lock_guard<std::mutex> lk(g_limit_mu);
  if (dev >= 0 && dev < 64) g_host_limit[dev] = cycles;
  return BPF_OK;
}

long long barrier_limit() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) dev = 0;
  std::lock_guard<std::mutex> lk(g_limit_mu);
  if (!g_host_limit_init) {
    for (long long& v : g_host_limit) v = kBarrierTimeoutCycles;
    g_host_limit_init = true;
  }
  return dev >= 0 && dev < 64 ? g_host_limit[dev] : kBarrierTimeoutCycles;
}

int autotuned_shape(int n) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return -1;
  return tuned_shape(dev, n);
}

int launch_gather(const int* as, const void* X, void* Y, int n, int d, int ld, int esz, const int* gate,
                  cudaStream_t st) {
  if (n <= 0 || d <= 0 || ld < n) return BPF_E_INVALID;
  const int g = (n + kBlock - 1) / kBlock;
  if (esz == 4) {
    k_gather<float><<<g, kBlock, 0, st>>>(as, (const float*)X, (float*)Y, n, d, ld, gate);
  } else if (esz == 8) {
    k_gather<double><<<g, kBlock, 0, st>>>(as, (const double*)X, (double*)Y, n, d, ld, gate);
  } else {
    return BPF_E_INVALID;
  }
  BPF_TRY(cudaGetLastError());
  return BPF_OK;
}

}  // namespace bpf
