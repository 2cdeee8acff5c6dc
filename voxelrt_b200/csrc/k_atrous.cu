// k_atrous.cu -- the a-trous iteration (atrous.wgsl:26-83) of one image.
#include "atrous_tile.cuh"
#include "vrt_internal.h"

namespace vrt {

// Three iterations back to back, against the form before (one pixel per thread,
// tiles staged by TMA; odd widths unstaged): 1920x1080 260 -> 172 us, with
// normals off the axes 260 -> 226; 960x540 82 -> 49; 641x361 60 -> 30; 320x180
// 31 -> 21; 128x72 25.7 -> 15.5.  Tiles that hold a negative, infinite or NaN
// colour keep the sums of skipped taps by selects: with one such pixel in a
// thousand 1920x1080 takes 178 (negative) to 188 us (NaN, infinite), 260 and 269
// before, and 176 with 30% of the colours -0.  (One thread per pixel on the
// unstaged image for those tiles took 529 and 605.)  Three blocks of 256 threads
// on an SM, 78 registers; four (64 registers, spilling) take 166 us at 1920x1080, but
// 32 against 26 at 480x270 and 34 against 27 at 640x360.
template <int S, bool kSrcF32>
__global__ void __launch_bounds__(kAtrousThreads, kAtrousBlocks) k_atrous(int W, int H, const void* src, const float4* gbuf,
                                                              uint2* __restrict__ dst) {
  frame_begin();
  extern __shared__ float4 sm[];
  atrous_tile<S>(sm, AtrousImage{W, H, src, kSrcF32, gbuf, dst}, blockIdx.x * kAtrousW, blockIdx.y * kAtrousH);
}

template <int S, bool kSrcF32>
static cudaError_t run(int W, int H, const void* src, const void* gbuf, void* dst, cudaStream_t st) {
  using G = AtrousGeom<S>;
  auto* fn = k_atrous<S, kSrcF32>;
  const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, G::smem);
  if (e != cudaSuccess) return e;
  const dim3 grid((W + kAtrousW - 1) / kAtrousW, (H + kAtrousH - 1) / kAtrousH);
  launch_after(fn, grid, kAtrousThreads, G::smem, st, W, H, src, (const float4*)gbuf, (uint2*)dst);
  return cudaGetLastError();
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
