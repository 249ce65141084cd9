// A batch of independent filters in shared structure-of-arrays buffers
// (batch.cu): the per-filter layout the batch kernels index through, and
// the per-step history record.  The guided step of a batch (guided.cu) uses
// the same layout.
#pragma once
#include "internal.cuh"

namespace bpf {

struct BatchFilter {
  int n;          // particles
  int off;        // first column in the shared buffers
  int block0;     // first transition block (and partial)
  int nblocks;    // transition blocks
  int resampler;  // BPF_RESAMPLER_*
  int B;          // Metropolis steps
  uint64_t seed;
  int tile0;      // first 128-particle tile of the guided step
  int ntiles;     // 128-particle tiles of the guided step
};

// the finalising block of filter f appends (logIncrement, ESS, resampled)
__device__ __forceinline__ void batch_record(const StepStats* st, double* hist, int nf, int f, int k) {
  if (hist && threadIdx.x == 0) {
    double* h = hist + 3 * ((size_t)k * nf + f);
    h[0] = st->inc;
    h[1] = st->ess;
    h[2] = (double)st->resampled;
  }
}

// the batched resampler (batch_resample.cu): how a batch's filters are
// resampled
struct ResamplePlan {
  const int* order = nullptr;           // the filters, the largest first (device)
  const BatchFilter* sorted = nullptr;  // their entries in that order (device)
  int nf = 0;
  int max_n = 0;      // particles of the largest filter
  bool mult = false;  // any multinomial resampler
  int group = 1;      // CTAs per filter (one thread-block cluster)
  int threads = 1024; // per CTA
};
// whether clusters of `group` CTAs hold the plan's largest filter
bool batch_resample_holds(const ResamplePlan& p, int group);
// fills all of the plan but order and sorted
void plan_batch_resample(const BatchFilter* filt, int nf, ResamplePlan* p);
int launch_batch_resample(const double* lw, int* as, const ResamplePlan& p, StepStats* stats, double* lu_buf,
                          int* os_buf, int step, cudaStream_t st);
int tune_batch_resample(const BatchFilter* filt, ResamplePlan* p, int ld, cudaStream_t st, double* us);

}  // namespace bpf
