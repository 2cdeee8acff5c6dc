// k_wavefront.cu -- wavefront form of the plain path tracer (sm_100a), for
// one session.
//
// The megakernel (k_trace.cu) runs one path per thread; its warps idle on
// sky pixels, skipped shadow rays and on the longest DDA walk of each warp
// (ncu: ~11% of lanes active per instruction).  Here a frame is split into
// waves:
//
//   generate  : per pixel RNG init, sub-pixel jitter, camera ray
//   trace(0)  : primary rays (implicit queue = all pixels)
//   shade(0)  : G-buffer/albedo, vertex 0 (emission, sun NEE sample, bounce
//               sample) -> shadow + bounce rays appended to queue 1
//   trace(k)  : queue k;  shade(k): resolve vertex k-1's shadow ray, shade
//               vertex k, append queue k+1 ... until every path terminated.
//
// Queues and active-path lists are compacted with one atomic per block.  The
// trace kernel is persistent: each warp owns 32 lanes that step through bricks
// or voxels in one loop (dda_walk.cuh) and change between the levels together;
// lanes whose ray ended are refilled from the queue once enough of them are
// idle, so warps stay full until the queue drains.  The kernels are defined in
// wavefront_core.cuh and shared with the batched form (k_batch.cu).
//
// The per-path arithmetic (RNG draws, shading, order of radiance sums) is
// exactly the megakernel's, so results are bit-identical to it and to the
// CPU oracle.
#include "trace_kernel.cuh"
#include "wavefront_core.cuh"
#include <algorithm>
#include <cstring>

namespace vrt {

// Queue capacity: a plain path appends at most a shadow and a bounce ray per
// wave; with several slots a path (or the spatial pass's pixel) up to four.
static size_t queue_entries(size_t P, int slots) { return (slots > 1 ? 4 : 2) * P; }

size_t wavefront_bytes(int W, int H, int max_waves, int slots) {
  const size_t P = (size_t)W * H;
  return P * 16 * (4 + 3 * (size_t)slots) + queue_entries(P, slots) * 4 * 2 + P * 4 * 2 + (size_t)max_waves * 20;
}

void carve_wavefront(void* mem, size_t P, int max_waves, WavefrontBufs& wb, int slots) {
  char* m = (char*)mem;
  const size_t big = (size_t)slots * P;
  void** f4[7] = {&wb.R0, &wb.R1, &wb.R2, &wb.S0, &wb.S1, &wb.S2, &wb.hit};
  for (auto* f : f4) {
    const bool twice = f == &wb.R0 || f == &wb.R2 || f == &wb.hit;
    *f = m;
    m += (twice ? big : P) * 16;
  }
  for (int i = 0; i < 2; i++) { wb.q[i] = (uint32_t*)m; m += queue_entries(P, slots) * 4; }
  wb.qcap = queue_entries(P, slots);
  for (int i = 0; i < 2; i++) { wb.act[i] = (uint32_t*)m; m += P * 4; }
  wb.acap = P;
  wb.ctr = (int*)m;
  wb.max_waves = max_waves;
  wb.slots = slots;
}

static SingleJob make_job(const SceneDev& s, const VrtUniforms& uu, float fclamp, int W, int H, const PathOut& out) {
  SingleJob job;
  job.u = to_uni(uu);
  job.S = to_dscene(s);
  job.out.rad16 = (uint2*)out.rad16;
  job.out.rad32 = (float4*)out.rad32;
  job.out.alb8 = out.alb8;
  job.out.gbuf = (float4*)out.gbuf;
  job.fclamp = fclamp;
  job.W = W;
  job.H = H;
  return job;
}

cudaError_t launch_wavefront(const SceneDev& s, const VrtUniforms& uu, float fclamp, int W, int H,
                             const PathOut& out, const WavefrontBufs& wb, const WavefrontTuning& tune,
                             cudaStream_t st, uint32_t* launches, cudaEvent_t* trace_ev, int max_timed_waves,
                             int* timed_waves, const CacheLaunch* cache, cudaEvent_t* cache_ev) {
  SingleJob job = make_job(s, uu, fclamp, W, H, out);
  std::memset(&job.cc, 0, sizeof job.cc);
  if (cache) job.cc = cache->cd;
  // cache-assisted frames run as many waves as their training paths need
  const int waves = (job.cc.on ? (int)job.cc.train_bounces : (int)job.u.params0[1]) + 2;
  const bool cc = job.cc.on != 0;
  const int tail = frame_tail(tune, (uint32_t)(W * H), waves, cc, cc);
  cudaError_t e = wf_launch_frame(job, (uint32_t)(W * H), waves, wb, tune, out.stats, st, launches, trace_ev,
                                  max_timed_waves, timed_waves, 1, tail);
  if (e != cudaSuccess || !job.cc.on) return e;
  if (cache_ev && (e = cudaEventRecord(cache_ev[0], st)) != cudaSuccess) return e;
  e = launch_cache_post(job, wf_view(wb), cache, 1, out.stats, st, launches);
  if (e != cudaSuccess) return e;
  if (cache_ev) e = cudaEventRecord(cache_ev[1], st);
  return e;
}

}  // namespace vrt
