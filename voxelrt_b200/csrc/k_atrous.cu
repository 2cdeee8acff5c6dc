// k_atrous.cu -- the a-trous iteration (atrous.wgsl:26-83) of one image.
#include "atrous_tile.cuh"
#include "vrt_internal.h"

namespace vrt {

// Three iterations back to back, against the form before (one pixel per thread,
// tiles staged by TMA; odd widths unstaged): 1920x1080 260 -> 173 us, with
// normals off the axes 260 -> 239; 641x361 60 -> 42.  Tiles that hold a negative, infinite or NaN
// colour keep the sums of skipped taps by selects: with one such pixel in a
// thousand 1920x1080 takes 183 (negative) to 196 us (NaN, infinite), 260 and 269 before, and
// 177 with 30% of the colours -0.  (One thread per pixel
// on the unstaged image for those tiles took 529 and 605.)  24 resident warps per SM (80 registers);
// 32 (64 registers, spilling) measure the same.  Issue slots 64% busy, FMA pipe
// 51% (a packed instruction holds it twice as long).
//
// Tiles of 32 rows read less halo; 16 rows make twice the blocks.  Measured at
// 16 / 32 rows: 320x180 32 / 33 us, 800x450 52 / 56, 960x540 69 / 68, 1283x721
// 104 / 107, 1920x1080 201 / 197: the line is at two full waves of 32-row tiles
// (3 on each SM).  8 rows: no better at any size.
template <int S, int R, bool kSrcF32>
__global__ void __launch_bounds__(8 * R, 96 / R) k_atrous(int W, int H, const void* src, const float4* gbuf,
                                                          uint2* __restrict__ dst) {
  frame_begin();
  extern __shared__ float4 sm[];
  atrous_tile<S, R>(sm, AtrousImage{W, H, src, kSrcF32, gbuf, dst}, blockIdx.x * kAtrousTile, blockIdx.y * R);
}

template <int S, int R, bool kSrcF32>
static cudaError_t run_tiles(int W, int H, const void* src, const void* gbuf, void* dst, cudaStream_t st) {
  using G = AtrousGeom<S, R>;
  auto* fn = k_atrous<S, R, kSrcF32>;
  const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, G::smem);
  if (e != cudaSuccess) return e;
  const dim3 grid((W + kAtrousTile - 1) / kAtrousTile, (H + R - 1) / R);
  launch_after(fn, grid, G::threads, G::smem, st, W, H, src, (const float4*)gbuf, (uint2*)dst);
  return cudaGetLastError();
}

template <int S, bool kSrcF32>
static cudaError_t run(int W, int H, const void* src, const void* gbuf, void* dst, cudaStream_t st) {
  const long tiles = (long)((W + 31) / 32) * ((H + 31) / 32);
  return tiles < 6 * wf_sm_count() ? run_tiles<S, 16, kSrcF32>(W, H, src, gbuf, dst, st)
                     : run_tiles<S, 32, kSrcF32>(W, H, src, gbuf, dst, st);
}

cudaError_t launch_atrous(int W, int H, const void* src, bool src_f32, const void* gbuf, void* dst, int step,
                          cudaStream_t st) {
  switch (step) {
    case 1: return src_f32 ? run<1, true>(W, H, src, gbuf, dst, st) : run<1, false>(W, H, src, gbuf, dst, st);
    case 2: return src_f32 ? run<2, true>(W, H, src, gbuf, dst, st) : run<2, false>(W, H, src, gbuf, dst, st);
    case 4: return src_f32 ? run<4, true>(W, H, src, gbuf, dst, st) : run<4, false>(W, H, src, gbuf, dst, st);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace vrt
