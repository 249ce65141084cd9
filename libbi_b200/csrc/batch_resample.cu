// The resampler of a batch of filters (and of every single filter small
// enough for it): permuted systematic, multinomial or Metropolis ancestors,
// computed on chip, for every filter of the batch in one launch.
//
// A filter is resampled by the CTAs of one thread-block cluster (1, 2, 4 or
// 8 of them), each holding a contiguous share of its particles: one SM's
// issue slots bound a filter resampled by one CTA (about 370 instructions a
// particle, 12 us at N = 4096, 250 us at 32768), while every further CTA
// costs its scans and cluster barriers.  The cluster size and the threads per
// CTA are timed when a batch is created (tune_batch_resample).  Block totals
// cross the cluster through distributed shared memory (each CTA
// writes its total into every other CTA's slot) and the hardware cluster
// barrier.  The fixed-point weights and cumulative offspring stay in shared
// memory from the first pass to the last, so a weight's exp is evaluated
// once, the log-weights are read once and the ancestors written once.
#include "internal.cuh"
#include "resample_common.cuh"
#include "batch.cuh"
#include "tune_pick.h"
#include "../../include/bpf_math.h"

#include <algorithm>

namespace bpf {

namespace {

constexpr int kGroup = 8;             // CTAs of a cluster at most (the portable maximum)
constexpr int kCtaParticles = 4096;   // particles of one CTA at most
static_assert(kGroup * kCtaParticles >= BPF_BATCH_MAX_PARTICLES, "the largest filter fits a cluster");
// extra copies of one particle above which the block writes them together
constexpr int kBlockCopies = 512;
constexpr int kBigMax = BPF_BATCH_MAX_PARTICLES / kBlockCopies + 1;
// the multinomial resampler's coarse index: every 16th log uniform, so that
// the rest of a search is one 128-byte line
constexpr int kCoarse = 16;

__device__ __forceinline__ uint32_t cluster_map(const void* p, uint32_t rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
  return r;
}
__device__ __forceinline__ void st_cluster(uint32_t a, unsigned long long v) {
  asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(a), "l"(v) : "memory");
}
__device__ __forceinline__ void st_cluster(uint32_t a, int v) {
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
// every thread of every CTA of the cluster; what they wrote before it (to
// shared memory of any of them, or to global memory) is visible after it
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
__device__ __forceinline__ void cluster_sync(int G) {
  if (G == 1) {
    __syncthreads();
    return;
  }
  cluster_arrive();
  cluster_wait();
}

// a block total into slot [rank] of every CTA of the cluster
__device__ __forceinline__ void publish(int G, int rank, u128 (&slot)[kGroup], u128 v) {
  if (threadIdx.x < G) {
    const uint32_t a = cluster_map(&slot[rank], threadIdx.x);
    st_cluster(a, v.lo);
    st_cluster(a + 8, v.hi);
  }
}
__device__ __forceinline__ void publish(int G, int rank, int (&slot)[kGroup], int v) {
  if (threadIdx.x < G) st_cluster(cluster_map(&slot[rank], threadIdx.x), v);
}
// after the cluster's synchronisation: the sum of the CTAs before this one,
// and of all of them
__device__ __forceinline__ u128 cluster_prefix(int G, int rank, const u128 (&slot)[kGroup], u128* total) {
  u128 before = u128_zero(), all = u128_zero();
#pragma unroll
  for (int r = 0; r < kGroup; ++r) {
    if (r == rank) before = all;
    if (r < G) all = u128_add(all, slot[r]);
  }
  *total = all;
  return before;
}
__device__ __forceinline__ int cluster_prefix(int G, int rank, const int (&slot)[kGroup], int* total) {
  int before = 0, all = 0;
#pragma unroll
  for (int r = 0; r < kGroup; ++r) {
    if (r == rank) before = all;
    if (r < G) all += slot[r];
  }
  *total = all;
  return before;
}

// exclusive running maximum over the block's threads (v >= 0; 0 before the
// first)
template <int NT>
__device__ __forceinline__ int block_exclusive_max_nt(int v) {
  __shared__ int wt[NT / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int inc = v;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int o = __shfl_up_sync(0xffffffffu, inc, d);
    if (lane >= d) inc = max(inc, o);
  }
  int r = __shfl_up_sync(0xffffffffu, inc, 1);
  if (lane == 0) r = 0;
  if (lane == 31) wt[warp] = inc;
  __syncthreads();
  int t = lane < warp ? wt[lane] : 0;
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) t = max(t, __shfl_xor_sync(0xffffffffu, t, d));
  return max(r, t);
}

// below this difference to the largest log-weight a weight is zero in the
// fixed-point format: exp(-44.5) 2^63 < 1/2
constexpr double kZeroBelow = -44.5;

__device__ __forceinline__ u128 u128_of(unsigned long long q) {
  u128 r; r.lo = q; r.hi = 0; return r;
}

// Number of entries of the nondecreasing lu[0..n) below x.  coarse holds
// every kCoarse-th entry (shared memory); the run's entries come from L2
// with 16-byte loads in one round trip.
__device__ __forceinline__ int count_below(const double* lu, const double* coarse, int nc, int n, double x) {
  int lo = 0, hi = nc;  // first coarse entry not below x
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (coarse[mid] < x) lo = mid + 1; else hi = mid;
  }
  if (lo == 0) return 0;
  const int base = kCoarse * (lo - 1);
  int c = 0;
  if (base + kCoarse <= n) {
    const double2* p = reinterpret_cast<const double2*>(lu + base);
    double2 v[kCoarse / 2];
#pragma unroll
    for (int j = 0; j < kCoarse / 2; ++j) v[j] = __ldcg(p + j);
#pragma unroll
    for (int j = 0; j < kCoarse / 2; ++j) c += (v[j].x < x) + (v[j].y < x);
  } else {
    for (int j = base; j < n; ++j) c += __ldcg(lu + j) < x;
  }
  return base + c;
}

// particles of one CTA of a filter of n resampled by G: a multiple of
// kCoarse, so that the coarse entries fall on the starts of runs
__host__ __device__ __forceinline__ int chunk_of(int n, int G) { return (n + kCoarse * G - 1) / (kCoarse * G) * kCoarse; }

// Shared memory of a CTA, for chunks of at most `chunk` particles: a slot of
// 8 bytes per particle (its fixed-point weight, then its cumulative
// offspring, then its outcome and the rank of its first extra copy), and for the multinomial resampler the
// spacings in as many slots and the coarse index.
// One slot of padding per 16 keeps the reads of each thread's run free of
// bank conflicts.
__host__ __device__ __forceinline__ int pad16(int l) { return l + (l >> 4); }
__host__ __device__ inline int smem_slots(int chunk) { return (pad16(chunk) + 2) / 2 * 16; }
inline int smem_bytes(int max_n, int G, bool mult) {
  return smem_slots(chunk_of(max_n, G)) * (mult ? 2 : 1) + (mult ? (max_n + kCoarse - 1) / kCoarse * 8 : 0);
}

// Permuted ancestors of the filters, the rule of
// ResamplerHost::cumulativeOffspringToAncestorsPermute
// (share/src/bi/host/resampler/ResamplerHost.hpp:134-168) in closed form:
// survivors in place, extra copies by ancestor into the childless slots in
// ascending order.  Cumulative offspring of
//   systematic   SystematicResampler::cumulativeOffspring (SystematicResampler.hpp:111-130)
//   multinomial  MultinomialResamplerHost::ancestors (MultinomialResamplerHost.hpp:29-65)
//   Metropolis   MetropolisResamplerHost::ancestors (MetropolisResamplerHost.hpp:32-62)
// computed exactly as the grid-wide kernels compute them (resample.cu).
//
// The loops over a thread's particles stay rolled and their arrays in shared
// memory: a launch fetches its instructions anew, and unrolled into registers
// the loops took longer (14.2 against 12.6 us at N = 4096 on one CTA).
template <int NT>
__global__ void __launch_bounds__(NT, 1024 / NT)
k_batch_resample(const double* lw, int* __restrict__ as, const BatchFilter* __restrict__ sorted,
                 const int* __restrict__ order, StepStats* stats, double* lu_buf, int* os_buf, int step,
                 int G, int slot_bytes) {
  extern __shared__ __align__(16) unsigned char s_raw[];
  __shared__ u128 s_w[kGroup], s_v[kGroup], s_before;
  __shared__ double s_W, s_yW;  // the weights' sum; its reciprocal, or its logarithm (multinomial)
  __shared__ int s_i[kGroup], s_z[kGroup], s_nbig, s_end;
  __shared__ int s_big[kBigMax][3];
  // the transition after this kernel, a programmatic dependent, may be
  // scheduled; this kernel is one of the transition before it
  pdl_trigger();
  pdl_wait();
  // the filter's entry and number, then its first log-weights and its gate:
  // two rounds of loads
  const BatchFilter fd = sorted[blockIdx.x / G];
  const int f = order[blockIdx.x / G], rank = blockIdx.x % G;
  StepStats* st = stats + f;
  const int n = fd.n, tid = threadIdx.x, lane = tid & 31;
  const double* lwf = lw + fd.off;
  const int chunk = chunk_of(n, G);
  const int begin = min(n, rank * chunk), cn = min(n, begin + chunk) - begin;
  double nx = tid < cn ? lwf[begin + tid] : 0.0;
  if (st->resample == 0 || st->status != BPF_OK) return;  // uniform over the cluster
  // the cluster's CTAs may write to each other's shared memory once all of
  // them run: arrive here, wait before the first such write
  if (G > 1) cluster_arrive();
  int* asf = as + fd.off;
  int* ancf = os_buf + fd.off;  // the extra copies' ancestors by rank
  unsigned long long* s_q = reinterpret_cast<unsigned long long*>(s_raw);
  auto slot = [&](int l) -> int& { return reinterpret_cast<int*>(s_raw)[2 * pad16(l)]; };
  auto first_rank = [&](int l) -> int& { return reinterpret_cast<int*>(s_raw)[2 * pad16(l) + 1]; };
  double* s_sp = reinterpret_cast<double*>(s_raw + slot_bytes);
  double* s_coarse = reinterpret_cast<double*>(s_raw + 2 * slot_bytes);
  // thread t owns the run [t ipt, (t + 1) ipt) of the CTA's particles
  const int ipt = (cn + NT - 1) / NT;
  const int l0 = min(cn, tid * ipt), l1 = min(cn, l0 + ipt);
  const double mx = st->mx;
  const double nd = (double)n;
  if (tid == 0) s_nbig = 0;

  // ---- cumulative offspring, into the particles' slots ----
  int before0 = 0;  // of the particle before the thread's first
  int zl = 0;       // childless particles of the thread
  if (fd.resampler == BPF_RESAMPLER_SYSTEMATIC || fd.resampler == BPF_RESAMPLER_MULTINOMIAL) {
    const bool mult = fd.resampler == BPF_RESAMPLER_MULTINOMIAL;
    double* luf = lu_buf + fd.off;  // the log uniforms
    {
      // the weights, consecutive threads on consecutive particles
#pragma unroll 1
      for (int l = tid; l < cn; l += NT) {
        const double x = nx;
        if (l + NT < cn) nx = lwf[begin + l + NT];
        const double d = __dsub_rn(x, mx);
        unsigned long long q = 0ull;
        if (!(d < kZeroBelow)) q = weight_to_fixed(nanexp(d));
        s_q[pad16(l)] = q;
        if (mult) s_sp[pad16(l)] = multinomial_spacing(nullptr, begin + l, n, fd.seed, step);
      }
    }
    double a = 0.0;  // the systematic offset
    if (!mult) {
      const bpf_u32x4 r = bpf_draw(fd.seed, 0u, (uint32_t)step, 0u, BPF_RNG_SYSTEMATIC);
      a = bpf_u01d(r.v[0], r.v[1]);
    }
    __syncthreads();
    u128 acc = u128_zero(), vacc = u128_zero();
#pragma unroll 1
    for (int l = l0; l < l1; ++l) {
      acc = u128_add(acc, u128_of(s_q[pad16(l)]));
      if (mult) vacc = u128_add(vacc, spacing_to_fixed(s_sp[pad16(l)]));
    }
    u128 btot, bv, vexcl = u128_zero(), Wtot;
    const u128 texcl = block_exclusive_scan_u128_nt<NT>(acc, &btot);
    if (mult) vexcl = block_exclusive_scan_u128_nt<NT>(vacc, &bv);
    if (G > 1) cluster_wait();
    publish(G, rank, s_w, btot);
    if (mult) publish(G, rank, s_v, bv);
    cluster_sync(G);
    // the cluster's totals once per CTA (in every thread their 100 or so
    // instructions took up to 1500 cycles)
    if (tid < 32) {
      const u128 before = cluster_prefix(G, rank, s_w, &Wtot);
      const double Wt = u128_to_weight(Wtot);
      if (lane == 0) {
        s_before = before;
        s_W = Wt;
        s_yW = mult ? log(Wt) : __ddiv_rn(1.0, Wt);
      }
    }
    __syncthreads();
    u128 Q = u128_add(s_before, texcl);
    const double W = s_W;
    // SystematicResampler::cumulativeOffspring throws
    // ParticleFilterDegeneratedException unless W > 0
    // (share/src/bi/resampler/SystematicResampler.hpp:118-129)
    if (!(W > 0.0)) {
      if (rank == 0 && tid == 0) st->status = BPF_E_DEGENERATE;
      return;
    }
    if (!mult) {
      const double yW = s_yW;
      // the first pass gives the offspring before the thread's run (none
      // before the filter's first particle)
      int prev = 0;
#pragma unroll 1
      for (int l = l0 - 1; l < l1; ++l) {
        const bool run = l >= l0;
        const unsigned long long q = run ? s_q[pad16(l)] : 1ull;
        int o = prev;
        if (q != 0ull) {  // a weight of zero has no offspring
          if (run) Q = u128_add(Q, u128_of(q));
          o = begin + l >= 0 ? systematic_Os(u128_to_weight(Q), W, yW, nd, a, n) : 0;
        }
        if (run) {
          slot(l) = o;
          zl += o == prev;
        } else {
          before0 = o;
        }
        prev = o;
      }
    } else {
      // lu_s = lW + lMax_s, lMax_s = -(sum of the spacings of slots >= s)
      u128 Vtot;
      u128 V = u128_add(cluster_prefix(G, rank, s_v, &Vtot), vexcl);
      const double lW = s_yW;
#pragma unroll 1
      for (int l = l0; l < l1; ++l) {
        const int s = begin + l;
        const double v = s_sp[pad16(l)];
        const double lu = __dadd_rn(lW, -fixed_to_spacing(u128_sub(Vtot, V)));
        V = u128_add(V, spacing_to_fixed(v));
        luf[s] = lu;
        if (s % kCoarse == 0) {
          for (int c = 0; c < G; ++c)
            st_cluster(cluster_map(s_coarse + s / kCoarse, c), (unsigned long long)__double_as_longlong(lu));
        }
      }
      cluster_sync(G);
      // slot s takes the number of m with log(Ws_m) <= lu_s (clamped to n-1),
      // so Os_m = #{s : lu_s < log(Ws_m)} for m < n-1 and Os_{n-1} = n
      // (a weight of zero has no offspring: Os_m = Os_{m-1} without a search)
      const int nc = (n + kCoarse - 1) / kCoarse;
      auto offspring = [&](int m) {
        return m >= n - 1 ? n : count_below(luf, s_coarse, nc, n, log(u128_to_weight(Q)));
      };
      // before a later CTA's first particle
      const int first = tid == 0 && begin > 0 ? offspring(begin - 1) : 0;
      int last = first;
#pragma unroll 1
      for (int l = l0; l < l1; ++l) {
        const unsigned long long q = s_q[pad16(l)];
        if (q != 0ull || begin + l == n - 1) {
          Q = u128_add(Q, u128_of(q));
          last = offspring(begin + l);
        }
        slot(l) = last;
      }
      // the runs before this one, whose counts are nondecreasing
      before0 = block_exclusive_max_nt<NT>(last);
      if (tid == 0) before0 = first;
      int prev = before0;
#pragma unroll 1
      for (int l = l0; l < l1; ++l) {
        const int o = max(slot(l), before0);
        slot(l) = o;
        zl += o == prev;
        prev = o;
      }
    }
  } else {
    // Metropolis: B steps per particle, then offspring counts and their
    // cumulative sums
    for (int l = tid; l < cn; l += NT) __stcg(ancf + begin + l, 0);
    if (G > 1) cluster_wait();
    cluster_sync(G);
    for (int l = tid; l < cn; l += NT)
      atomicAdd(ancf + metropolis_ancestor(lwf, n, fd.B, nullptr, fd.seed, step, begin + l), 1);
    cluster_sync(G);
    int loc = 0;
    for (int l = l0; l < l1; ++l) {
      const int c = __ldcg(ancf + begin + l);
      slot(l) = c;
      loc += c;
      zl += c == 0;
    }
    int btot, tot;
    int run = block_exclusive_scan_int_nt<NT>(loc, &btot);
    publish(G, rank, s_i, btot);
    cluster_sync(G);
    run += cluster_prefix(G, rank, s_i, &tot);
    before0 = run;
    for (int l = l0; l < l1; ++l) {
      run += slot(l);
      slot(l) = run;
    }
  }

  // ---- permutation: ranks of the childless slots ----
  int bz, R;
  const int zexcl = block_exclusive_scan_int_nt<NT>(zl, &bz);
  publish(G, rank, s_z, bz);
  cluster_sync(G);
  // ---- each particle's outcome (the rank of its childless slot, or -1 for a
  //      survivor) and the rank E_i = Os_{i-1} - i + Z_i of its first extra
  //      copy; then the ancestor of each extra copy, by its rank ----
  int Z = zexcl + cluster_prefix(G, rank, s_z, &R);
  {
    int prev = before0;
#pragma unroll 1
    for (int l = l0; l < l1; ++l) {
      const int o = slot(l);
      slot(l) = o == prev ? Z : -1;
      first_rank(l) = prev - (begin + l) + Z;
      if (l == cn - 1) s_end = o - (begin + cn) + Z + (o == prev);  // E of the particle after the chunk
      Z += o == prev;
      prev = o;
    }
  }
  __syncthreads();
  auto put = [&](int r, int i) {
    if (r >= 0 && r < R) __stcg(ancf + r, i);  // a consistent Os stays in range
  };
  // a warp takes 32 consecutive particles, whose extra copies have
  // consecutive ranks, and writes 32 ranks at a time: the ancestor of rank r
  // is the last particle whose first rank is not above r
#pragma unroll 1
  for (int base = tid & ~31; base < cn; base += NT) {
    const int l = base + lane;
    const int e = l < cn ? first_rank(l) : s_end;
    int e1 = __shfl_down_sync(0xffffffffu, e, 1);
    if (lane == 31) e1 = l + 1 < cn ? first_rank(l + 1) : s_end;
    const int lo = __shfl_sync(0xffffffffu, e, 0), hi = __shfl_sync(0xffffffffu, e1, 31);
    const bool big = e1 - e > kBlockCopies;
    if (__any_sync(0xffffffffu, big)) {
      // a particle with very many copies is left to the whole block
      if (big) {
        const int b = atomicAdd(&s_nbig, 1);
        if (b < kBigMax) {
          s_big[b][0] = e;
          s_big[b][1] = e1 - e;
          s_big[b][2] = begin + l;
        }
      } else {
        for (int r = e; r < e1; ++r) put(r, begin + l);
      }
      continue;
    }
#pragma unroll 1
    for (int r0 = lo; r0 < hi; r0 += 64) {  // two independent searches at a time
      const int ra = r0 + lane, rb = ra + 32;
      int sa = 0, sb = 0;
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) {
        const int ta = __shfl_sync(0xffffffffu, e, sa + d), tb = __shfl_sync(0xffffffffu, e, sb + d);
        if (ta <= ra) sa += d;
        if (tb <= rb) sb += d;
      }
      if (ra < hi) put(ra, begin + base + sa);
      if (rb < hi) put(rb, begin + base + sb);
    }
  }
  __syncthreads();
  const int nbig = min(s_nbig, kBigMax);
  for (int b = 0; b < nbig; ++b)
    for (int j = tid; j < s_big[b][1]; j += NT) put(s_big[b][0] + j, s_big[b][2]);
  cluster_sync(G);
  // ---- survivors keep their place, childless slots take their ancestor ----
#pragma unroll 4
  for (int l = tid; l < cn; l += NT) {
    const int i = begin + l, r = slot(l);
    const int a = r >= 0 && r < R ? __ldcg(ancf + r) : i;
    asf[i] = a >= 0 && a < n ? a : i;
  }
}

}  // namespace

template <int NT>
static int launch_nt(const double* lw, int* as, const ResamplePlan& p, StepStats* stats,
                     double* lu_buf, int* os_buf, int step, cudaStream_t st) {
  static unsigned configured = 0;
  BPF_TRY(set_dyn_smem_once(k_batch_resample<NT>, smem_bytes(BPF_BATCH_MAX_PARTICLES, kGroup, true), configured));
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[2];
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)p.group;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3((unsigned)(p.group * p.nf));
  cfg.blockDim = dim3(NT);
  cfg.dynamicSmemBytes = (size_t)smem_bytes(p.max_n, p.group, p.mult);
  cfg.stream = st;
  cfg.attrs = at;
  cfg.numAttrs = 2;
  BPF_TRY(cudaLaunchKernelEx(&cfg, k_batch_resample<NT>, lw, as, p.sorted, p.order, stats, lu_buf, os_buf, step, p.group,
                             smem_slots(chunk_of(p.max_n, p.group))));
  return BPF_OK;
}

bool batch_resample_holds(const ResamplePlan& p, int group) {
  return p.max_n > 0 && p.max_n <= BPF_BATCH_MAX_PARTICLES && group >= 1 && group <= kGroup &&
         (group & (group - 1)) == 0 && chunk_of(p.max_n, group) <= kCtaParticles;
}

// threads per CTA: 256, 512 or 1024 (the in-CTA arithmetic is exact, so the
// count changes the speed only)
int launch_batch_resample(const double* lw, int* as, const ResamplePlan& p, StepStats* stats,
                          double* lu_buf, int* os_buf, int step, cudaStream_t st) {
  if (p.nf <= 0 || !batch_resample_holds(p, p.group)) return BPF_E_INVALID;
  switch (p.threads) {
    case 256: return launch_nt<256>(lw, as, p, stats, lu_buf, os_buf, step, st);
    case 512: return launch_nt<512>(lw, as, p, stats, lu_buf, os_buf, step, st);
    case 1024: return launch_nt<1024>(lw, as, p, stats, lu_buf, os_buf, step, st);
    default: return BPF_E_INVALID;
  }
}

// the largest filter's size and whether any is multinomial; the smallest
// cluster that holds the largest filter, until the plan is tuned
void plan_batch_resample(const BatchFilter* filt, int nf, ResamplePlan* p) {
  p->nf = nf;
  p->max_n = 0;
  p->mult = false;
  for (int f = 0; f < nf; ++f) {
    p->max_n = std::max(p->max_n, filt[f].n);
    p->mult |= filt[f].resampler == BPF_RESAMPLER_MULTINOMIAL;
  }
  p->group = 1;
  while (chunk_of(p->max_n, p->group) > kCtaParticles) p->group *= 2;
  p->threads = 1024;
}

// synthetic log-weights 2 N(0, 1) over the whole buffer, for the autotuner
__global__ void k_batch_synthetic_lw(double* lw, int ld) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= ld) return;
  const bpf_u32x4 r = bpf_draw(0x7a11ull, (uint32_t)i, 0u, 0u, BPF_RNG_DATA);
  double z0, z1;
  bpf_normal_pair_d(r.v[0], r.v[1], &z0, &z1);
  lw[i] = 2.0 * z0;
}

// statistics that open every filter's resampling gate, with each filter's
// maximum log-weight
__global__ void k_batch_tune_stats(const double* lw, const BatchFilter* filt, StepStats* st, int nf) {
  const int f = blockIdx.x;
  if (f >= nf) return;
  const BatchFilter fd = filt[f];
  double m = -INFINITY;
  for (int i = threadIdx.x; i < fd.n; i += blockDim.x) m = fmax(m, lw[fd.off + i]);
  m = warp_max(m);
  __shared__ double s_m[32];
  if ((threadIdx.x & 31) == 0) s_m[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) m = fmax(m, s_m[w]);
    m = fmax(m, s_m[0]);
    StepStats z{};
    z.mx = m;
    z.resample = 1;
    z.status = BPF_OK;
    z.n = fd.n;
    st[f] = z;
  }
}

// Time the cluster sizes that hold the largest filter, each with the three
// thread counts, on synthetic log-weights laid out as the batch's
// filters (scratch buffers: the batch's own state is untouched), and put the
// fastest into the plan; its cluster size's medians go to us[3] (256, 512,
// 1024 threads; infinite for one that could not be launched).
int tune_batch_resample(const BatchFilter* filt, ResamplePlan* p, int ld, cudaStream_t st, double* us) {
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  BPF_TRY(cudaStreamIsCapturing(st, &cs));
  if (cs != cudaStreamCaptureStatusNone) return BPF_OK;  // no timing inside a capture: keep the default
  double* lw = nullptr;
  double* lu = nullptr;
  int *as = nullptr, *os = nullptr;
  StepStats* stats = nullptr;
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  int rc = BPF_OK;
  auto A = [&](void** q, size_t b) {
    if (!rc && cudaMalloc(q, b) != cudaSuccess) rc = BPF_E_NOMEM;
  };
  A((void**)&lw, (size_t)ld * sizeof(double));
  A((void**)&lu, (size_t)ld * sizeof(double));
  A((void**)&as, (size_t)ld * sizeof(int));
  A((void**)&os, (size_t)ld * sizeof(int));
  A((void**)&stats, (size_t)p->nf * sizeof(StepStats));
  if (!rc && (cudaEventCreate(&e0) != cudaSuccess || cudaEventCreate(&e1) != cudaSuccess)) rc = BPF_E_CUDA;
  if (!rc) {
    k_batch_synthetic_lw<<<(ld + 255) / 256, 256, 0, st>>>(lw, ld);
    k_batch_tune_stats<<<p->nf, 256, 0, st>>>(lw, filt, stats, p->nf);
    if (cudaGetLastError() != cudaSuccess) rc = BPF_E_CUDA;
  }
  // candidates: every cluster size from the smallest that holds the largest
  // filter, each with the three thread counts.  The first launch of each
  // count, which loads its code, is not timed.
  constexpr int kReps = 3, kMax = 12;
  constexpr float kNear = 1.25f;
  ResamplePlan c[kMax];
  float med[kMax];
  int nc = 0, best = -1;
  for (int g = p->group; g <= kGroup; g *= 2)
    for (int thr = 256; thr <= 1024; thr *= 2) {
      c[nc] = *p;
      c[nc].group = g;
      c[nc++].threads = thr;
    }
  auto timed = [&](int k, float* ms) -> int {
    if (cudaEventRecord(e0, st) != cudaSuccess) return BPF_E_CUDA;
    const int e = launch_batch_resample(lw, as, c[k], stats, lu, os, 1, st);
    if (e) {
      cudaGetLastError();  // this candidate's alone
      return e;
    }
    if (cudaEventRecord(e1, st) != cudaSuccess || cudaEventSynchronize(e1) != cudaSuccess ||
        cudaEventElapsedTime(ms, e0, e1) != cudaSuccess)
      return BPF_E_CUDA;
    return BPF_OK;
  };
  if (!rc) {
    for (int k = 0; k < 3; ++k)
      if (launch_batch_resample(lw, as, c[k], stats, lu, os, 1, st)) cudaGetLastError();
    rc = pick_fastest<kMax, kReps>(nc, kNear, timed, med, &best);
  }
  if (!rc) {
    *p = c[best];
    // the thread counts' times with the kept cluster size
    if (us)
      for (int k = 0; k < 3; ++k) us[k] = 1e3 * med[best / 3 * 3 + k];
  }
  if (e0) cudaEventDestroy(e0);
  if (e1) cudaEventDestroy(e1);
  void* ps[] = {lw, lu, as, os, stats};
  for (void* q : ps)
    if (q) cudaFree(q);
  if (rc) cudaGetLastError();
  return rc;
}

}  // namespace bpf
