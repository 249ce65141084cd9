// The packed Box-Muller pairs (libbi_b200/csrc/f32x2.cuh) against
// bpf_normal_pair_f, whose quotient and square root are CUDA's correctly
// rounded ones: every one of the 2^23 radius uniforms and of the 2^23 angle
// uniforms in both halves of a packed pair.  Prints the number of values whose
// bits differ.
#include "../../libbi_b200/csrc/f32x2.cuh"

#include <cstdio>

constexpr uint32_t kValues = 1u << 23;

__device__ bool same(float a, float b) { return __float_as_uint(a) == __float_as_uint(b); }

// fixed_angle: the angle 2^-24, whose cosine is 1, so that the radius itself
// is compared; else the angles run through all values in another order
__global__ void k_compare(int fixed_angle, unsigned long long* bad) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= kValues) return;
  const uint32_t low = i & 511u;  // bits that a uniform does not use
  const uint32_t aA = i << 9 | low, aB = (kValues - 1u - i) << 9 | low;
  // an odd factor permutes the values
  const uint32_t bA = fixed_angle ? low : (i * 2654435761u) << 9 | low;
  const uint32_t bB = fixed_angle ? low : (i * 2246822519u + 12345u) << 9 | low;
  bpf::pair::f2 z0, z1;
  bpf::pair::normal_pair(aA, bA, aB, bB, z0, z1);
  float p0, p1, q0, q1, w0, w1, v0, v1;
  bpf::pair::unpack(z0, p0, q0);
  bpf::pair::unpack(z1, p1, q1);
  bpf_normal_pair_f(aA, bA, &w0, &w1);
  bpf_normal_pair_f(aB, bB, &v0, &v1);
  const int d = !same(p0, w0) + !same(p1, w1) + !same(q0, v0) + !same(q1, v1);
  if (d) atomicAdd(bad, (unsigned long long)d);
}

int main() {
  unsigned long long *bad = nullptr, h = ~0ull;
  if (cudaMalloc(&bad, sizeof(*bad)) != cudaSuccess || cudaMemset(bad, 0, sizeof(*bad)) != cudaSuccess) return 1;
  for (int fixed = 0; fixed < 2; ++fixed) k_compare<<<kValues / 256, 256>>>(fixed, bad);
  if (cudaMemcpy(&h, bad, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
  std::printf("%llu\n", h);
  return 0;
}
