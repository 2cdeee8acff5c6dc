// trace_kernel.cuh -- per-block helpers shared by the one-thread-per-pixel
// kernels (plain path megakernel, ray batches, ReSTIR passes).
#pragma once
#include "vrt_device.cuh"
#include "vrt_internal.h"
#include <cstring>

namespace vrt {

// Largest occupancy bitmap staged in shared memory (640^3 grid; a 512^3 grid's takes 36 KB).
constexpr size_t kMaxSmemOccBytes = 68 * 1024;

// Stage the padded grid's occupancy bitmap in shared memory (kSmem) or use
// the global copy.  Every thread of the block must call it.
template <bool kSmem>
VRT_DI const uint32_t* stage_occupancy(const DScene& S, uint32_t* s_occ) {
  if (!kSmem) return S.cells;
  const int P = S.BG + 2, nwords = (P * P * P + 31) >> 5;
  for (int i = threadIdx.x; i < nwords; i += blockDim.x) s_occ[i] = __ldg(S.cells + i);
  __syncthreads();
  return s_occ;
}


inline DScene to_dscene(const SceneDev& s) {
  DScene d;
  d.vox = s.vox; d.cells = s.cells; d.N = s.N; d.BG = s.BG;
  d.rP = recip_pad(s.BG); d.rP2 = recip_pad2(s.BG);
  d.mw = (uint32_t)mask_word(s.BG); d.pad = 0u;
  return d;
}

inline Uni to_uni(const VrtUniforms& u) {
  Uni r;
  static_assert(offsetof(Uni, sunT) == sizeof(VrtUniforms), "uniform layouts differ");
  std::memcpy(&r, &u, sizeof(VrtUniforms));
  sun_frame(u.sunDir, r.sunT, r.sunB);
  return r;
}

// Pixel of thread `threadIdx.x` in a 16 x 16 block whose eight warps each
// cover an 8 x 4 tile (coherent primary rays within a warp).
VRT_DI void block_pixel_16x16(int& gx, int& gy) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  gx = blockIdx.x * 16 + (warp & 1) * 8 + (lane & 7);
  gy = blockIdx.y * 16 + (warp >> 1) * 4 + (lane >> 3);
}

}  // namespace vrt
