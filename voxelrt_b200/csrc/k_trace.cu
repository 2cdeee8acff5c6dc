// k_trace.cu -- path-trace pass and the ray-batch entry (sm_100a).
//
// k_pathtrace is the plain branch of pathtrace.wgsl (lines 248-330): one
// thread per pixel, 16x16-pixel blocks whose warps cover 8x4 pixel tiles so
// primary rays of a warp stay coherent.  The brick occupancy bitmap (one bit
// per 8^3 brick, 4 KB at 256^3, 32 KB at 512^3) is staged once per block in
// shared memory; brick masks and voxels are read through the read-only path
// (L1/L2 resident: 2 MB + 64 MB at 256^3 fit the 126 MB L2).
#include <algorithm>
#include "dda_walk.cuh"
#include "trace_kernel.cuh"

namespace vrt {

// One pixel of the plain path (pathtrace.wgsl:248-330).
VRT_DI void path_pixel(const DScene& S, const uint32_t* occ, const Uni& u, float fclamp, uint32_t gx, uint32_t gy,
                       uint32_t W, uint32_t H, float4& rad, uint32_t& alb, float4& gb, DCount& cnt) {
  uint32_t rng = init_rng(gx, gy, u.params0[0]);
  const float jx = rand_(rng) - 0.5f;
  const float jy = rand_(rng) - 0.5f;
  const float uvx = (((float)gx + 0.5f) + jx) / (float)W;
  const float uvy = (((float)gy + 0.5f) + jy) / (float)H;
  const F3 ro = f3(u.camPos[0], u.camPos[1], u.camPos[2]);
  F3 rd = camera_ray(u, uvx, uvy);

  const DHit h0 = trace<true>(S, occ, ro, rd, 1e4f, cnt);
  if (h0.t < 0.0f) {
    const F3 sky = sky_color(u, rd, true);
    rad = make_float4(sky.x, sky.y, sky.z, 1.0f);
    alb = 0xffffffffu;
    gb = make_float4(-rd.x, -rd.y, -rd.z, -1.0f);
    return;
  }
  const Mat mat1 = unpack_material(h0.mat);
  const F3 x1 = ro + rd * h0.t;
  const F3 n1 = h0.n;
  alb = sqrt_albedo8(h0.mat);
  gb = make_float4(n1.x, n1.y, n1.z, h0.t);

  F3 radiance = f3(0.0f, 0.0f, 0.0f);
  F3 tp = f3(1.0f, 1.0f, 1.0f);
  F3 pos = x1, n = n1;
  Mat mat = mat1;
  const uint32_t nB = u.params0[1];
  const F3 sunRad = f3(u.sunRadiance[0], u.sunRadiance[1], u.sunRadiance[2]);
  for (uint32_t bounce = 0; bounce <= nB; bounce++) {
    if (mat.emissive > 0.0f) radiance = radiance + (tp * mat.albedo) * (mat.emissive * kEmissiveScale);
    const F3 surf = pos + n * 1e-3f;
    const F3 l = sample_sun_dir(u, rng);
    const float ndl = dot3(n, l);
    if (ndl > 0.0f && l.y > 0.0f) {
      const DHit hs = trace<true>(S, occ, surf, l, 1e4f, cnt);
      if (!(hs.t >= 0.0f)) radiance = radiance + (((tp * mat.albedo) * kInvPi) * ndl) * sunRad;
    }
    if (bounce == nB) break;
    rd = cosine_hemisphere(n, rng);
    tp = tp * mat.albedo;
    if (bounce >= 2u) {
      const float p = clamp_(fmax_(tp.x, fmax_(tp.y, tp.z)), 0.05f, 0.95f);
      if (rand_(rng) > p) break;
      tp = f3(tp.x / p, tp.y / p, tp.z / p);
    }
    const DHit h = trace<true>(S, occ, surf, rd, 1e4f, cnt);
    if (h.t < 0.0f) {
      radiance = radiance + tp * sky_color(u, rd, false);
      break;
    }
    pos = surf + rd * h.t;
    n = h.n;
    mat = unpack_material(h.mat);
  }
  if (!(fclamp <= 0.0f)) radiance = min3(radiance, f3(fclamp, fclamp, fclamp));
  const F3 den = max3(mat1.albedo, f3(1e-3f, 1e-3f, 1e-3f));
  rad = make_float4(radiance.x / den.x, radiance.y / den.y, radiance.z / den.z, 1.0f);
}

template <bool kSmem>
__global__ void __launch_bounds__(256) k_pathtrace(DScene S, Uni u, float fclamp, int W, int H, PathOut out) {
  extern __shared__ uint32_t s_occ[];
  const uint32_t* occ = stage_occupancy<kSmem>(S, s_occ);
  int gx, gy;
  block_pixel_16x16(gx, gy);
  DCount cnt{0u, 0u, 0u, 0u};
  uint32_t pix = 0;
  if (gx < W && gy < H) {
    float4 rad, gb;
    uint32_t alb;
    path_pixel(S, occ, u, fclamp, (uint32_t)gx, (uint32_t)gy, (uint32_t)W, (uint32_t)H, rad, alb, gb, cnt);
    const size_t p = (size_t)gy * W + gx;
    reinterpret_cast<uint2*>(out.rad16)[p] = pack_h4(rad.x, rad.y, rad.z, rad.w);
    if (out.rad32) reinterpret_cast<float4*>(out.rad32)[p] = rad;
    out.alb8[p] = alb;
    reinterpret_cast<float4*>(out.gbuf)[p] = gb;
    pix = 1;
  }
  if (out.stats) block_flush_stats(out.stats, cnt, pix);
}

// A batch of rays on the resumable walk (dda_walk.cuh).  A warp owns a run of
// `run` consecutive rays and refills its idle lanes from it, so no counter in
// memory is needed; blocks are many and short, and the block scheduler evens
// the runs out.  Bound by instruction issue, like the queue tracer; against one
// thread per ray on the nested loops, 2 M incoherent rays at 256^3 took 470 ->
// 256 us (call with its wait), 1.2 M at 128^3 256 -> 166, 64 rays 27 -> 13, 1000
// 27 -> 19.
constexpr int kRayThreads = 128, kRayRefill = 12, kRayMaxRun = 256;

template <bool kWide>
__global__ void __launch_bounds__(kRayThreads, 9) k_trace_rays(DScene S, const float* __restrict__ o,
                                                               const float* __restrict__ d,
                                                               const float* __restrict__ tmax, int n, int run,
                                                               VrtHit* __restrict__ out) {
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const long long first = ((long long)blockIdx.x * (kRayThreads / 32) + (threadIdx.x >> 5)) * run;
  if (first >= n) return;                                   // warp-uniform
  uint32_t next = (uint32_t)first;
  const uint32_t end = (uint32_t)min((long long)n, first + run);
  DCount c{0u, 0u, 0u, 0u};
  Walk<kWide> w;
  F3 rd = f3(0.0f, 0.0f, 0.0f);
  uint32_t i = 0u;
  bool active = false, held = false;
  while (true) {
    const unsigned idle = __ballot_sync(full, !active);
    const int nidle = __popc(idle);
    if (nidle >= kRayRefill || next >= end) {
      if (held && !active) {
        VrtHit r;
        int vx = -1, vy = -1, vz = -1;
        const bool hit = w.finish(S, c, vx, vy, vz);
        const F3 nrm = hit ? hit_normal(w.hit_axis(S), rd) : f3(-rd.x, -rd.y, -rd.z);
        r.t = w.tHit; r.n[0] = nrm.x; r.n[1] = nrm.y; r.n[2] = nrm.z; r.mat = w.mat;
        r.voxel[0] = hit ? vx : -1; r.voxel[1] = hit ? vy : -1; r.voxel[2] = hit ? vz : -1;
        r.face = r.t >= 0.0f ? face_of(nrm) : -1;
        r.steps = c.outer + c.inner;
        r.bytes = 4u * (c.outer + c.inner + c.vreads);
        r.pad = 0u;
        out[i] = r;
        held = false;
      }
      if (next < end) {
        const uint32_t mine = next + __popc(idle & ((1u << lane) - 1u));
        next += (uint32_t)nidle;
        if (!active && mine < end) {
          i = mine;
          rd = f3(d[3 * (size_t)i], d[3 * (size_t)i + 1], d[3 * (size_t)i + 2]);
          w.init(S, f3(o[3 * (size_t)i], o[3 * (size_t)i + 1], o[3 * (size_t)i + 2]), rd, tmax[i]);
          c = DCount{0u, 0u, 0u, 0u};
          active = held = true;
        }
      } else if (nidle == 32) {
        return;
      }
    }
    if (active) {
#pragma unroll 1
      for (int k = 0; k < 3; k++) {
        w.template walk_run<5>(S);
        if (!w.walking() && !w.done()) w.transition(S, rd, c);
      }
      active = !w.done();
    }
  }
}

// The same batch with one thread per ray on the nested loops.  A ray's walk is
// latency there as here, but its lane never waits for the warp's transitions.
template <int kThreads>
__global__ void __launch_bounds__(kThreads) k_trace_rays_nested(DScene S, const float* __restrict__ o,
                                                           const float* __restrict__ d,
                                                           const float* __restrict__ tmax, int n,
                                                           VrtHit* __restrict__ out) {
  extern __shared__ uint32_t s_occ[];
  const uint32_t* occ = stage_occupancy<true>(S, s_occ);
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  DCount cnt{0u, 0u, 0u, 0u};
  const F3 ro = f3(o[3 * i], o[3 * i + 1], o[3 * i + 2]);
  const F3 rd = f3(d[3 * i], d[3 * i + 1], d[3 * i + 2]);
  const DHit h = trace<true>(S, occ, ro, rd, tmax[i], cnt);
  VrtHit r;
  r.t = h.t; r.n[0] = h.n.x; r.n[1] = h.n.y; r.n[2] = h.n.z; r.mat = h.mat;
  r.voxel[0] = h.vx; r.voxel[1] = h.vy; r.voxel[2] = h.vz;
  r.face = h.t >= 0.0f ? face_of(h.n) : -1;
  r.steps = cnt.outer + cnt.inner;
  r.bytes = 4u * (cnt.outer + cnt.inner + cnt.vreads);
  r.pad = 0u;
  out[i] = r;
}

cudaError_t launch_pathtrace(const SceneDev& s, const VrtUniforms& u, float fclamp, int W, int H,
                             const PathOut& out, cudaStream_t st) {
  const size_t smem = pad_words(s.BG) * sizeof(uint32_t);
  dim3 grid((W + 15) / 16, (H + 15) / 16);
  if (smem <= kMaxSmemOccBytes) {
    if (smem > 48 * 1024) {
      cudaError_t e = cudaFuncSetAttribute(k_pathtrace<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (e != cudaSuccess) return e;
    }
    k_pathtrace<true><<<grid, 256, smem, st>>>(to_dscene(s), to_uni(u), fclamp, W, H, out);
  } else {
    k_pathtrace<false><<<grid, 256, 0, st>>>(to_dscene(s), to_uni(u), fclamp, W, H, out);
  }
  return cudaGetLastError();
}

cudaError_t launch_trace_rays(const SceneDev& s, const float* o, const float* d, const float* tmax, int n,
                              VrtHit* out, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  // Where one thread per ray about fills the GPU and the longest walk decides, the nested loops are the safe
  // choice: from some 14 K rays to one wave of their blocks (1024 rays an SM).  us per call, nested / walk, means of
  // three worlds and two batches, in 80^3, 128^3 and 256^3 voxels: 12 K rays 24.9 / 21.3, 30.5 / 26.5, 37.3 / 31.4;
  // 24 K 25.2 / 25.4, 32.4 / 30.4, 39.0 / 36.9 (single batches up to 0.83 of the nested loops' rate); 64 K
  // 26.5 / 29.8, 33.6 / 34.9, 44.5 / 44.9; 130 K 33.3 / 36.2, 41.4 / 41.4, 54.8 / 55.1; 185 K 41.9 / 42.8, 51.5 / 47.0,
  // 67.4 / 61.0.  Small worlds end a walk so soon that its refills and transitions pay only where its long runs
  // begin: 32^3 at 5 K 14.2 / 12.9, 8 K 14.5 / 15.1, 800 K 75 / 91, 2 M 173 / 172; 64^3 at 800 K 107 / 110, 1.2 M
  // 153 / 133; 80^3 at 270 K 51.4 / 51.4, 330 K 58.5 / 57.8.
  const int sms = wf_sm_count(), wave = 1024 * sms;
  const size_t smem = pad_words(s.BG) * sizeof(uint32_t);
  const int nested_from = s.BG <= 4 ? 7000 : 14000;
  const int nested_to = s.BG <= 4 ? 1600000 : (s.BG <= 8 ? 1000000 : (s.BG <= 10 ? 320000 : wave));
  if (n >= nested_from && n <= nested_to && smem <= kMaxSmemOccBytes) {
    // past one wave smaller blocks even the end out (800 K rays at 64^3: 110 -> 105 us); within it they lie
    // unevenly on the SMs (145 K rays at 80^3: 34.5 -> 36.0)
    const int threads = n <= wave ? 256 : 128;
    auto* fn = threads == 256 ? k_trace_rays_nested<256> : k_trace_rays_nested<128>;
    if (smem > 48 * 1024) {
      cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (e != cudaSuccess) return e;
    }
    fn<<<(unsigned)((n + threads - 1) / threads), threads, smem, st>>>(to_dscene(s), o, d, tmax, n, out);
    return cudaGetLastError();
  }
  // Rays per warp.  Few rays are spread over all warps the GPU holds (9 blocks
  // on each SM), down to one per warp, since lanes on different paths
  // take turns; from 32 per warp on, one per lane until the rays fill the GPU
  // three times over, then longer runs with refills.
  const int warps = kRayThreads / 32, resident = sms * 9 * warps;
  const int run = n <= 32 * resident ? (n + resident - 1) / resident
                                     : std::min(kRayMaxRun, std::max(32, n / (3 * resident) / 32 * 32));
  const unsigned blocks = (unsigned)(((long long)n + (long long)run * warps - 1) / ((long long)run * warps));
  if (s.BG > kNarrowBG) k_trace_rays<true><<<blocks, kRayThreads, 0, st>>>(to_dscene(s), o, d, tmax, n, run, out);
  else k_trace_rays<false><<<blocks, kRayThreads, 0, st>>>(to_dscene(s), o, d, tmax, n, run, out);
  return cudaGetLastError();
}

}  // namespace vrt
