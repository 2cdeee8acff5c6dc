// k_batch.cu -- many independent views rendered in one launch sequence.
//
// A batch frame renders one frame for each of n sessions (different scenes,
// sizes, bounce counts, cameras).  The sessions' pixels are laid out back to
// back in one global index space; a warp of consecutive pixels finds its job
// with one load per 32 jobs over the jobs' first pixels, a path from a list by a
// binary search over them.  The wavefront path tracer runs
// over all jobs at once -- one persistent trace launch per wave serves rays
// of every scene -- followed by one temporal, three a-trous and one present
// launch over all jobs.  Per-pixel arithmetic is the single-session code
// (wavefront_core.cuh, image_core.cuh), so each job's image is bit-identical
// to rendering that session alone.
#include <cstddef>
#include "wavefront_core.cuh"
#include "atrous_tile.cuh"

namespace vrt {

static_assert(sizeof(JobDev) == sizeof(JobHost), "job table layouts differ");
static_assert(offsetof(JobDev, S) == offsetof(JobHost, vox), "job table layouts differ");
static_assert(offsetof(JobDev, S.mw) == offsetof(JobHost, mw), "job table layouts differ");
static_assert(offsetof(JobDev, out) == offsetof(JobHost, rad16), "job table layouts differ");
static_assert(offsetof(JobDev, W) == offsetof(JobHost, W), "job table layouts differ");
static_assert(offsetof(JobDev, acc_prev) == offsetof(JobHost, acc_prev), "job table layouts differ");
static_assert(offsetof(JobDev, acc_f32) == offsetof(JobHost, acc_f32), "job table layouts differ");
static_assert(offsetof(JobDev, cache) == offsetof(JobHost, cache), "job table layouts differ");

// temporal.wgsl:17-77 over all jobs.
__global__ void __launch_bounds__(256) k_b_temporal(MultiJob J, uint32_t P) {
  frame_begin();
  const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = J.job_of_warp(g);
  if (g >= P) return;
  const JobDev& jd = J.jobs[j];
  const int W = jd.W, H = jd.H;
  const uint32_t lp = g - jd.first;
  const int x = (int)(lp % (uint32_t)W), y = (int)(lp / (uint32_t)W);
  const float4 res = temporal_pixel(jd.u, W, H, x, y, jd.out.rad16, jd.out.gbuf, jd.acc_prev, jd.acc_f32 != 0,
                                    jd.gbuf_prev);
  store_px(jd.acc_cur, jd.acc_f32 != 0, lp, res);
}

// atrous.wgsl:26-83 iteration `it` (step 1 << it) of every job whose denoise
// flag is set; chain accum -> dA -> dB -> dA (main.js:503-507).  A CTA computes
// one tile of one job (atrous_tile.cuh).  tiles: m + 1 prefix counts of the jobs'
// tiles, in which CTA b finds its job.
template <int S>
__global__ void __launch_bounds__(kAtrousThreads, kAtrousBlocks) k_b_atrous(MultiJob J, const uint32_t* __restrict__ tiles) {
  frame_begin();
  extern __shared__ float4 sm[];
  const uint32_t b = blockIdx.x;
  const int lo = last_at_or_before(tiles, J.n, b);
  const JobDev& jd = J.jobs[lo];
  if ((jd.u.params0[2] & 2u) == 0u) return;
  const int tb = (int)(b - __ldg(tiles + lo)), tw = (jd.W + kAtrousW - 1) / kAtrousW;
  const void* src = S == 1 ? jd.acc_cur : (S == 2 ? (const void*)jd.den0 : (const void*)jd.den1);
  uint2* dst = S == 2 ? jd.den1 : jd.den0;
  const int x0 = (tb % tw) * kAtrousW, y0 = (tb / tw) * kAtrousH;
  // one copy of the filter for each type of history, as for a single view
  if (S == 1 && jd.acc_f32 != 0) atrous_tile<S>(sm, AtrousImage{jd.W, jd.H, src, true, jd.out.gbuf, dst}, x0, y0);
  else atrous_tile<S>(sm, AtrousImage{jd.W, jd.H, src, false, jd.out.gbuf, dst}, x0, y0);
}

template <int S>
static cudaError_t launch_b_atrous(const MultiJob& J, const AtrousTiles& at, cudaStream_t st) {
  using G = AtrousGeom<S>;
  const cudaError_t e =
      cudaFuncSetAttribute(k_b_atrous<S>, cudaFuncAttributeMaxDynamicSharedMemorySize, G::smem);
  if (e != cudaSuccess) return e;
  launch_after(k_b_atrous<S>, at.n, kAtrousThreads, G::smem, st, J, at.first);
  return cudaGetLastError();
}

// present.wgsl:40-55 over all jobs.
__global__ void __launch_bounds__(256) k_b_present(MultiJob J, uint32_t P, const float* __restrict__ lut) {
  frame_begin();
  const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = J.job_of_warp(g);
  if (g >= P) return;
  const JobDev& jd = J.jobs[j];
  const uint32_t lp = g - jd.first;
  const bool denoise = (jd.u.params0[2] & 2u) != 0u;
  const float4 il = denoise ? load_px(jd.den0, false, lp) : load_px(jd.acc_cur, jd.acc_f32 != 0, lp);
  jd.ldr[lp] = present_pixel(jd.u.params1[2], il, jd.out.alb8[lp], lut);
}

cudaError_t launch_batch_frame(const void* d_jobs, const uint32_t* d_firsts, int n, int max_bg, uint32_t P, int waves,
                               const WavefrontBufs& wb, const WavefrontTuning& tune, unsigned long long* stats,
                               cudaStream_t st, uint32_t* launches, const float* present_lut, const AtrousTiles& at,
                               const CacheLaunch* cls, int ncl) {
  MultiJob J;
  J.jobs = (const JobDev*)d_jobs;
  J.firsts = d_firsts;
  J.n = n;
  J.cache_jobs = ncl;
  J.max_bg = max_bg;
  const int tail = frame_tail(tune, P, waves, ncl > 0, ncl > 0 && ncl == n);
  cudaError_t e = wf_launch_frame(J, P, waves, wb, tune, stats, st, launches, nullptr, 0, nullptr, n, tail);
  if (e != cudaSuccess) return e;
  // the cache jobs' inference, resolve and training, all jobs per launch
  if (ncl > 0 && (e = launch_cache_post(J, wf_view(wb), cls, ncl, stats, st, launches)) != cudaSuccess) return e;
  const unsigned blocks = (P + 255) / 256;
  launch_after(k_b_temporal, blocks, 256, 0, st, J, P);
  if ((e = launch_b_atrous<1>(J, at, st)) != cudaSuccess || (e = launch_b_atrous<2>(J, at, st)) != cudaSuccess ||
      (e = launch_b_atrous<4>(J, at, st)) != cudaSuccess)
    return e;
  launch_after(k_b_present, blocks, 256, 0, st, J, P, present_lut);
  if (launches) *launches += 5;
  return cudaGetLastError();
}

}  // namespace vrt
