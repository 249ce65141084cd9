// A training step of the Lorenz-96 proposal (80-128-128-80, proposal.cu) in
// two launches:
//   k_train_tile    one CTA per 128 minibatch rows (persistent when there are
//                   more tiles than SMs): gathers and standardises the rows,
//                   runs the three layers forward, the loss gradient, the two
//                   back-propagated errors and the three weight gradients,
//                   all on tcgen05 with the activations in shared memory and
//                   the accumulators in tensor memory; only the tile's share
//                   of the weight gradients (147 KB), its bias sums and its
//                   loss leave the SM;
//   k_reduce_adam   adds the shares in the order of the CTAs, applies Adam and
//                   refreshes the BF16 copy and the shared-memory images of
//                   the weights.
// Layer by layer (eight dense launches with transposed staging, three split-K
// reductions and nine small kernels, every activation through memory) a step
// of 8192 rows took 510 us, most of it in kernels of 64 CTAs that staged
// their operands element by element; the arithmetic is under 2 us of tensor
// time.  The tile kernel is bound by the latency of its six dependent MMA and
// epilogue phases.
//
// An activation tile is written once, in the canonical K-major layout of
// tc.cuh ((r/8) KC 16 + (c/8) 128 + (r%8) 16 + (c%8) 2 for row r, column c).
// The same bytes are an MN-major operand over the rows: its core matrix is
// eight columns (16 contiguous bytes) by eight rows (16 bytes apart), the
// next one along the columns 128 bytes away (SBO), along the rows KC 16
// (LBO).  So the weight gradients, which contract over the rows, and the
// back-propagated errors, which contract over a weight image's rows, need no
// transposed copies.
//
// Every sum has a fixed order, so training is reproducible bit for bit: a
// weight gradient 128 rows at a time in K steps of 16, up to 148 tiles in the
// order of the tiles; beyond, CTA c adds tiles c, c + 148, ... in tensor
// memory, and the CTAs' shares are added in order.  Bias gradients in chunks
// of 64 rows, in order.
#include "internal.cuh"
#include "tc.cuh"
#include "proposal.cuh"
#include "guided_tc.cuh"

namespace bpf {
namespace {

constexpr int kDin = 80, kH = kProposalHidden, kD = 40, kDout = 80, kRows = 128;
constexpr int kTrainThreads = 256;  // thread t: row t % 128, column half t / 128
// shared memory: the weight images, the activation tiles (H1 and H2 are
// overwritten in place by dZ1 and dZ2), vectors
constexpr uint32_t kW1B = kH * kDin * 2, kW2B = kH * kH * 2, kW3B = kDout * kH * 2;
constexpr uint32_t kUB = kRows * kDin * 2, kHB = kRows * kH * 2, kOB = kRows * kDout * 2;
constexpr uint32_t kVecB = (2 * kDin + 2 * kH + kDout) * 4;
constexpr int kTrainSmem = (int)(kW1B + kW2B + kW3B + kUB + 2 * kHB + kOB + kVecB) + 1024;
// tensor memory columns: the layers' accumulator, then the three weight
// gradients (dW3 and dW2 transposed: lane = input feature)
constexpr uint32_t kTAcc = 0, kTW3 = 128, kTW2 = 256, kTW1 = 384;
constexpr int kColChunkRows = 64;
constexpr int kColWidth = kDout + 2 * kH;  // bias sums per chunk: layer 3, 2, 1

struct TrainTileArgs {
  // the minibatch: drawn from the data set (xt != null) or given (U, r0)
  const float *xt, *mt, *xt1, *yt1;
  int n, step;
  uint64_t seed;
  const float *shift, *scale;
  const __nv_bfloat16* U;
  const float* r0;
  int B, tiles;
  const unsigned char* packed;
  int pk_w1, pk_w2, pk_w3;
  const float *b1, *b2, *b3;
  int o_w1, o_w2, o_w3, nparams;
  float* ws;          // gridDim.x x nparams: weight-gradient shares
  float* colpart;     // per 64-row chunk: bias sums
  double* loss_part;  // per tile
  int* err;
};

template <bool VEC>
__device__ __forceinline__ float4 load4(const float* p) {
  if (VEC) return __ldg(reinterpret_cast<const float4*>(p));
  return make_float4(__ldg(p), __ldg(p + 1), __ldg(p + 2), __ldg(p + 3));
}

// D (+)= A B^T over 16-element K steps.  AMN / BMN: the operand's image is
// read as MN-major (its rows are the K dimension).  KCA, KCB: columns of the
// images.
template <int K, int N, int KCA, int KCB, bool AMN, bool BMN>
__device__ __forceinline__ void chain(uint32_t tmem, const unsigned char* A, const unsigned char* B, bool accumulate) {
  constexpr uint32_t idesc = tc::idesc_bf16(128, N) | (AMN ? 1u << 15 : 0u) | (BMN ? 1u << 16 : 0u);
#pragma unroll
  for (int ks = 0; ks < K / 16; ++ks) {
    const uint64_t ad = AMN ? tc::smem_desc(tc::smem_u32(A) + ks * 2 * KCA * 16, KCA * 16, 128)
                            : tc::smem_desc(tc::smem_u32(A) + ks * 256, 128, KCA * 16);
    const uint64_t bd = BMN ? tc::smem_desc(tc::smem_u32(B) + ks * 2 * KCB * 16, KCB * 16, 128)
                            : tc::smem_desc(tc::smem_u32(B) + ks * 256, 128, KCB * 16);
    tc::mma_bf16(tmem, ad, bd, idesc, accumulate || ks > 0 ? 1u : 0u);
  }
}

// this thread's 64 columns of its accumulator row + bias, ReLU, BF16, into
// row r of the tile
__device__ __forceinline__ void hidden_half(uint32_t trow, const float* bias, unsigned char* sH, int r, int half) {
#pragma unroll 1
  for (int n0 = 64 * half; n0 < 64 * half + 64; n0 += 32) {
    float v[32];
    tc::tmem_ld32(trow + (uint32_t)n0, v);
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = fmaxf(v[j] + bias[n0 + j], 0.0f);
#pragma unroll
    for (int c = 0; c < 4; ++c)
      *reinterpret_cast<uint4*>(sH + tc::kmajor_off(r, n0 + 8 * c, kH)) = pack8(v + 8 * c);
  }
}

// dZ = dH where the layer's output is positive, in place of the output
__device__ __forceinline__ void relu_back_half(uint32_t trow, unsigned char* sH, int r, int half) {
#pragma unroll 1
  for (int n0 = 64 * half; n0 < 64 * half + 64; n0 += 32) {
    float v[32];
    tc::tmem_ld32(trow + (uint32_t)n0, v);
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      uint4* p = reinterpret_cast<uint4*>(sH + tc::kmajor_off(r, n0 + 8 * c, kH));
      const uint4 h = *p;
      const __nv_bfloat16* hb = reinterpret_cast<const __nv_bfloat16*>(&h);
#pragma unroll
      for (int j = 0; j < 8; ++j) v[8 * c + j] = __bfloat162float(hb[j]) > 0.0f ? v[8 * c + j] : 0.0f;
      *p = pack8(v + 8 * c);
    }
  }
}

// column sums of a tile in chunks of 64 rows, in row order
template <int N>
__device__ __forceinline__ void column_sums(const unsigned char* s, float* part) {
  const int t = threadIdx.x;
  if (t >= 2 * N) return;
  const int j = t % N, c = t / N;
  float a = 0.0f;
#pragma unroll 8
  for (int r = c * kColChunkRows; r < (c + 1) * kColChunkRows; ++r)
    a += __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(s + tc::kmajor_off(r, j, N)));
  part[(size_t)c * kColWidth + j] = a;
}

// N accumulator columns of this thread's lane (its half of them) to
// dst[col * ld + lane] for lane < lanes
template <int N>
__device__ __forceinline__ void store_share(uint32_t trow, float* dst, int ld, int lane, int lanes, int half) {
#pragma unroll 1
  for (int n0 = 16 * half; n0 < N; n0 += 32) {
    float v[16];
    tc::tmem_ld16(trow + (uint32_t)n0, v);
    if (lane < lanes) {
#pragma unroll
      for (int j = 0; j < 16; ++j) dst[(size_t)(n0 + j) * ld + lane] = v[j];
    }
  }
}

// VEC: the data set's arrays are 16-byte aligned (their rows are 160 bytes)
template <bool VEC>
__global__ void __launch_bounds__(kTrainThreads, 1) k_train_tile(TrainTileArgs a) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  unsigned char* sW1 = smem;
  unsigned char* sW2 = sW1 + kW1B;
  unsigned char* sW3 = sW2 + kW2B;
  // U first of the tiles: the MN-major read of its 80 columns as 128 runs
  // past its end into the next tile (lanes 80.. of dW1, never stored)
  unsigned char* sU = sW3 + kW3B;
  unsigned char* sO = sU + kUB;
  unsigned char* sH1 = sO + kOB;
  unsigned char* sH2 = sH1 + kHB;
  float* sShift = reinterpret_cast<float*>(sH2 + kHB);
  float* sScale = sShift + kDin;
  float* sB1 = sScale + kDin;
  float* sB2 = sB1 + kH;
  float* sB3 = sB2 + kH;
  __shared__ uint64_t mbar, wbar;
  __shared__ uint32_t s_taddr;
  __shared__ double s_loss[kTrainThreads / 32];
  const int tid = threadIdx.x, warp = tid >> 5, r = tid % kRows, half = tid / kRows;
  if (warp == 0) tc::tmem_alloc(&s_taddr, 512);
  if (tid == 0) {
    tc::mbar_init(&mbar, 1);
    tc::mbar_init(&wbar, 1);
  }
  pdl_wait();  // the weights of the step before
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t taddr = s_taddr;
  const uint32_t trow = taddr + ((uint32_t)((warp & 3) * 32) << 16);
  if (tid == 0) {
    tc::mbar_expect_tx(&wbar, kW1B + kW2B + kW3B);
    tc::bulk_g2s(sW1, a.packed + a.pk_w1, kW1B, &wbar);
    tc::bulk_g2s(sW2, a.packed + a.pk_w2, kW2B, &wbar);
    tc::bulk_g2s(sW3, a.packed + a.pk_w3, kW3B, &wbar);
  }
  if (tid < kDin) {
    sShift[tid] = a.xt ? a.shift[tid] : 0.0f;
    sScale[tid] = a.xt ? a.scale[tid] : 0.0f;
  }
  if (tid < kH) {
    sB1[tid] = a.b1[tid];
    sB2[tid] = a.b2[tid];
  }
  if (tid < kDout) sB3[tid] = a.b3[tid];
  __syncthreads();
  // components of the loss this thread forms: 0..23 or 24..39
  const int i0 = 24 * half, ni = half ? 16 : 24;
  bool ok = true;
  uint32_t phase = 0;
  bool first = true;
  const float invB = 1.0f / (float)a.B;
  for (int tile = blockIdx.x; tile < a.tiles; tile += gridDim.x) {
    const int b = tile * kRows + r;
    const bool live = b < a.B;
    float res[24];  // x_{t+1} - m
    {
      // the row's half of the standardised inputs [x_t, y - m]
      float u[kD];
      if (!live) {
#pragma unroll
        for (int j = 0; j < kD; ++j) u[j] = 0.0f;
#pragma unroll
        for (int j = 0; j < 24; ++j) res[j] = 0.0f;
      } else if (a.xt) {
        const bpf_u32x4 w = bpf_draw(a.seed, (uint32_t)b, (uint32_t)a.step, 0u, BPF_RNG_DATA);
        const size_t row = (size_t)(((uint64_t)w.v[0] << 32 | w.v[1]) % (uint64_t)a.n) * kD;
        const float *px = (half ? a.yt1 : a.xt) + row, *pm = a.mt + row, *p1 = a.xt1 + row;
#pragma unroll
        for (int q = 0; q < kD / 4; ++q) {
          const float4 v = load4<VEC>(px + 4 * q);
          u[4 * q] = v.x; u[4 * q + 1] = v.y; u[4 * q + 2] = v.z; u[4 * q + 3] = v.w;
        }
#pragma unroll
        for (int q = 0; q < 6; ++q)
          if (4 * q < ni) {
            const float4 v = load4<VEC>(p1 + i0 + 4 * q), m = load4<VEC>(pm + i0 + 4 * q);
            res[4 * q] = v.x - m.x; res[4 * q + 1] = v.y - m.y;
            res[4 * q + 2] = v.z - m.z; res[4 * q + 3] = v.w - m.w;
          }
        if (half) {
#pragma unroll
          for (int q = 0; q < kD / 4; ++q) {
            const float4 m = load4<VEC>(pm + 4 * q);
            u[4 * q] -= m.x; u[4 * q + 1] -= m.y; u[4 * q + 2] -= m.z; u[4 * q + 3] -= m.w;
          }
        }
#pragma unroll
        for (int j = 0; j < kD; ++j) u[j] = (u[j] - sShift[kD * half + j]) * sScale[kD * half + j];
      } else {
#pragma unroll
        for (int j = 0; j < kD; ++j) u[j] = __bfloat162float(a.U[(size_t)b * kDin + kD * half + j]);
#pragma unroll
        for (int j = 0; j < 24; ++j) res[j] = j < ni ? a.r0[(size_t)b * kD + i0 + j] : 0.0f;
      }
#pragma unroll
      for (int c = 0; c < kD / 8; ++c)
        *reinterpret_cast<uint4*>(sU + tc::kmajor_off(r, kD * half + 8 * c, kDin)) = pack8(u + 8 * c);
    }
    // forward
    ok = weights_ready(&wbar, 0u, ok);  // later tiles: the phase is complete
    if (ok && tid == 0) {
      tc::fence_after_sync();
      chain<kDin, kH, kDin, kDin, false, false>(taddr + kTAcc, sU, sW1, false);
      tc::mma_commit(&mbar);
    }
    ok = layer_done(&mbar, phase, ok);
    phase ^= 1u;
    if (ok) hidden_half(trow + kTAcc, sB1, sH1, r, half);
    ok = weights_ready(&wbar, 0u, ok);
    if (ok && tid == 0) {
      tc::fence_after_sync();
      chain<kH, kH, kH, kH, false, false>(taddr + kTAcc, sH1, sW2, false);
      tc::mma_commit(&mbar);
    }
    ok = layer_done(&mbar, phase, ok);
    phase ^= 1u;
    if (ok) hidden_half(trow + kTAcc, sB2, sH2, r, half);
    ok = weights_ready(&wbar, 0u, ok);
    if (ok && tid == 0) {
      tc::fence_after_sync();
      chain<kH, kDout, kH, kH, false, false>(taddr + kTAcc, sH2, sW3, false);
      tc::mma_commit(&mbar);
    }
    ok = layer_done(&mbar, phase, ok);
    phase ^= 1u;
    // the loss and its gradient, eight components at a time
    double l = 0.0;
    if (ok) {
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        if (8 * c < ni) {
          const int i = i0 + 8 * c;
          float d[8], s[8];
          tc::tmem_ld8(trow + kTAcc + (uint32_t)i, d);
          tc::tmem_ld8(trow + kTAcc + (uint32_t)(kD + i), s);
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float sr = s[j] + sB3[kD + i + j];
            const float sc = fminf(fmaxf(sr, kSMin), kSMax);
            const float e = expf(-2.0f * sc);
            const float q = res[8 * c + j] - (d[j] + sB3[i + j]);
            if (live) l += (double)(sc + 0.5f * q * q * e);
            const bool inside = sr > kSMin && sr < kSMax;
            d[j] = live ? -q * e * invB : 0.0f;
            s[j] = live && inside ? (1.0f - q * q * e) * invB : 0.0f;
          }
          *reinterpret_cast<uint4*>(sO + tc::kmajor_off(r, i, kDout)) = pack8(d);
          *reinterpret_cast<uint4*>(sO + tc::kmajor_off(r, kD + i, kDout)) = pack8(s);
        }
      }
    }
    l = warp_sum(l);
    if ((tid & 31) == 0) s_loss[warp] = l;
    // backward; each phase's weight gradient and back-propagated error run
    // while the bias sums are formed
    float* part = a.colpart + (size_t)(2 * tile) * kColWidth;
    const bool acc = !first;
    ok = weights_ready(&wbar, 0u, ok);
    if (ok && tid == 0) {
      tc::fence_after_sync();
      chain<kRows, kDout, kH, kDout, true, true>(taddr + kTW3, sH2, sO, acc);
      chain<kDout, kH, kDout, kH, false, true>(taddr + kTAcc, sO, sW3, false);
      tc::mma_commit(&mbar);
    }
    if (ok) column_sums<kDout>(sO, part);
    if (tid == 0) {
      double t = 0.0;
      for (int w = 0; w < kTrainThreads / 32; ++w) t += s_loss[w];
      a.loss_part[tile] = t;
    }
    ok = layer_done(&mbar, phase, ok);
    phase ^= 1u;
    if (ok) relu_back_half(trow + kTAcc, sH2, r, half);
    ok = weights_ready(&wbar, 0u, ok);
    if (ok && tid == 0) {
      tc::fence_after_sync();
      chain<kRows, kH, kH, kH, true, true>(taddr + kTW2, sH1, sH2, acc);
      chain<kH, kH, kH, kH, false, true>(taddr + kTAcc, sH2, sW2, false);
      tc::mma_commit(&mbar);
    }
    if (ok) column_sums<kH>(sH2, part + kDout);
    ok = layer_done(&mbar, phase, ok);
    phase ^= 1u;
    if (ok) relu_back_half(trow + kTAcc, sH1, r, half);
    ok = weights_ready(&wbar, 0u, ok);
    if (ok && tid == 0) {
      tc::fence_after_sync();
      chain<kRows, kH, kDin, kH, true, true>(taddr + kTW1, sU, sH1, acc);
      tc::mma_commit(&mbar);
    }
    if (ok) column_sums<kH>(sH1, part + kDout + kH);
    ok = layer_done(&mbar, phase, ok);
    phase ^= 1u;
    first = false;
    if (!ok) break;
  }
  pdl_trigger();
  if (ok && !first) {
    float* w = a.ws + (size_t)blockIdx.x * a.nparams;
    store_share<kDout>(trow + kTW3, w + a.o_w3, kH, r, kH, half);
    store_share<kH>(trow + kTW2, w + a.o_w2, kH, r, kH, half);
    store_share<kH>(trow + kTW1, w + a.o_w1, kDin, r, kDin, half);
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(taddr, 512);
  if (!ok && tid == 0) atomicExch(a.err, 1);
}

struct ReduceAdamArgs {
  const float* ws;
  int shares;
  const float* colpart;
  int chunks;
  const double* loss_part;
  int tiles, B;
  double* loss;
  float* grads;
  int nparams, o_b1, o_w2, o_b2, o_w3, o_b3;
  // Adam; P null: the gradient alone
  float *P, *M1, *M2;
  __nv_bfloat16* Ph;
  unsigned char* packed;
  int pk_w1, pk_w2, pk_w3;
  float lr, b1, b2, eps, c1, c2;
};

// One thread per parameter; the block after the last one forms the loss.
__global__ void __launch_bounds__(64) k_reduce_adam(ReduceAdamArgs a) {
  pdl_trigger();
  pdl_wait();  // the tiles' shares
  if (blockIdx.x == gridDim.x - 1) {
    if (threadIdx.x < 32) {
      double t = 0.0;
      for (int k = threadIdx.x; k < a.tiles; k += 32) t += a.loss_part[k];
      t = warp_sum(t);
      if (threadIdx.x == 0) *a.loss = t / (double)a.B;
    }
    return;
  }
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.nparams) return;
  // this parameter's place: a weight (row, col of its image) or a bias
  int bias = -1, row = 0, col = 0, pk = 0, kc = kH;
  if (i < a.o_b1) {
    row = i / kDin, col = i % kDin, pk = a.pk_w1, kc = kDin;
  } else if (i < a.o_w2) {
    bias = kDout + kH + i - a.o_b1;
  } else if (i < a.o_b2) {
    row = (i - a.o_w2) / kH, col = (i - a.o_w2) % kH, pk = a.pk_w2;
  } else if (i < a.o_w3) {
    bias = kDout + i - a.o_b2;
  } else if (i < a.o_b3) {
    row = (i - a.o_w3) / kH, col = (i - a.o_w3) % kH, pk = a.pk_w3;
  } else {
    bias = i - a.o_b3;
  }
  const float* src = bias >= 0 ? a.colpart + bias : a.ws + i;
  const size_t stride = bias >= 0 ? (size_t)kColWidth : (size_t)a.nparams;
  const int terms = bias >= 0 ? a.chunks : a.shares;
  // the terms in order, 32 loads in flight
  float g = 0.0f;
  int k = 0;
#pragma unroll 1
  for (; k + 32 <= terms; k += 32) {
    float v[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = src[(k + j) * stride];
#pragma unroll
    for (int j = 0; j < 32; ++j) g += v[j];
  }
#pragma unroll 4
  for (; k < terms; ++k) g += src[k * stride];
  a.grads[i] = g;
  if (!a.P) return;
  // the fused products are spelled out: the moments' bits are then the same
  // whatever the compiler makes of the sums
  const float m = __fmaf_rn(1.0f - a.b1, g, __fmul_rn(a.b1, a.M1[i]));
  const float v = __fmaf_rn(__fmul_rn(1.0f - a.b2, g), g, __fmul_rn(a.b2, a.M2[i]));
  a.M1[i] = m;
  a.M2[i] = v;
  const float p = a.P[i] - a.lr * (m / a.c1) / (sqrtf(v / a.c2) + a.eps);
  a.P[i] = p;
  const __nv_bfloat16 h = __float2bfloat16(p);
  a.Ph[i] = h;
  if (bias < 0) *reinterpret_cast<__nv_bfloat16*>(a.packed + pk + tc::kmajor_off(row, col, kc)) = h;
}

}  // namespace

int train_shares(int B) {
  const int tiles = (B + kRows - 1) / kRows;
  return tiles < kTrainMaxShares ? tiles : kTrainMaxShares;
}
long long train_colpart_floats(int cap) { return (long long)((cap + kRows - 1) / kRows) * 2 * kColWidth; }

int launch_train_tile(ProposalNet& p, const TrainBatch& t, cudaStream_t st) {
  if (!p.l96 || t.B < 1 || t.B > p.cap) return BPF_E_INVALID;
  static unsigned configured[2] = {0, 0};
  BPF_TRY(set_dyn_smem_once(k_train_tile<true>, kTrainSmem, configured[0]));
  BPF_TRY(set_dyn_smem_once(k_train_tile<false>, kTrainSmem, configured[1]));
  TrainTileArgs a{};
  a.xt = t.xt; a.mt = p.mt; a.xt1 = t.xt1; a.yt1 = t.yt1;
  a.n = t.n; a.step = t.step; a.seed = t.seed;
  a.shift = p.shift; a.scale = p.scale;
  a.U = p.U; a.r0 = p.r0;
  a.B = t.B;
  a.tiles = (t.B + kRows - 1) / kRows;
  a.packed = p.packed;
  a.pk_w1 = p.pk_w1; a.pk_w2 = p.pk_w2; a.pk_w3 = p.pk_w3;
  a.b1 = p.b1(); a.b2 = p.b2(); a.b3 = p.b3();
  a.o_w1 = p.o_w1; a.o_w2 = p.o_w2; a.o_w3 = p.o_w3; a.nparams = p.nparams;
  const bool vec = ((reinterpret_cast<uintptr_t>(t.xt) | reinterpret_cast<uintptr_t>(p.mt) | reinterpret_cast<uintptr_t>(t.xt1) |
            reinterpret_cast<uintptr_t>(t.yt1)) & 15) == 0;
  a.ws = p.ws;
  a.colpart = p.colpart;
  a.loss_part = p.loss_part;
  a.err = p.err;
  BPF_TRY(launch_pdl(vec ? k_train_tile<true> : k_train_tile<false>, dim3((unsigned)train_shares(t.B)), dim3(kTrainThreads), (size_t)kTrainSmem, st, a));
  return BPF_OK;
}

int launch_reduce_adam(ProposalNet& p, int B, double* loss, bool update, float lr, float b1, float b2, float eps,
                       float c1, float c2, cudaStream_t st) {
  ReduceAdamArgs a{};
  a.ws = p.ws;
  a.shares = train_shares(B);
  a.colpart = p.colpart;
  a.chunks = (B + kColChunkRows - 1) / kColChunkRows;
  a.loss_part = p.loss_part;
  a.tiles = (B + kRows - 1) / kRows;
  a.B = B;
  a.loss = loss;
  a.grads = p.grads;
  a.nparams = p.nparams;
  a.o_b1 = p.o_b1; a.o_w2 = p.o_w2; a.o_b2 = p.o_b2; a.o_w3 = p.o_w3; a.o_b3 = p.o_b3;
  if (update) {
    a.P = p.params; a.M1 = p.m1; a.M2 = p.m2; a.Ph = p.params_h; a.packed = p.packed;
  }
  a.pk_w1 = p.pk_w1; a.pk_w2 = p.pk_w2; a.pk_w3 = p.pk_w3;
  a.lr = lr; a.b1 = b1; a.b2 = b2; a.eps = eps; a.c1 = c1; a.c2 = c2;
  BPF_TRY(launch_pdl(k_reduce_adam, dim3((unsigned)((p.nparams + 63) / 64 + 1)), dim3(64), 0, st, a));
  return BPF_OK;
}

}  // namespace bpf
