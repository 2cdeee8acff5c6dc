// k_lights.cu -- the scene's emissive-face light list and per-brick light
// grid (scene.js:58-200, 435-461) built on the device, for scenes that are
// edited at run time (the reference builds them once on the CPU).
//
// Light list: every exposed face of an emissive voxel, voxels in z, y, x
// order and faces +x,-x,+y,-y,+z,-z within a voxel -- an ordered compaction:
// per-voxel face counts, a scan of per-block totals, then each block writes
// its lights at its offset.  Weights (emissiveFaceWeight) in double, as the
// reference's JavaScript numbers.
//
// Light grid: every brick cell ranks every light by power / max(d^2,
// (BRICK/2)^2) with a facing test and keeps the top 16, replaying the
// reference's insertion order and its Float32Array roundings exactly.
#include "vrt_device.cuh"
#include "vrt_internal.h"

namespace vrt {

constexpr int kLgK = 16, kLgStride = 2 + 2 * kLgK;

__device__ __forceinline__ double light_weight_d(uint32_t m) {
  const double e = (double)((m >> 24) & 0xffu) / 255.0;
  if (e <= 0.0) return 0.0;
  const double r = (double)(m & 0xffu) / 255.0;
  const double g = (double)((m >> 8) & 0xffu) / 255.0;
  const double b = (double)((m >> 16) & 0xffu) / 255.0;
  return e * (((0.2126 * r) * r + (0.7152 * g) * g) + (0.0722 * b) * b);
}

// Exposed-face bit mask (bit f = face f is a light) of voxel i.
__device__ __forceinline__ uint32_t light_faces(const uint32_t* __restrict__ vox, int N, long long i) {
  const uint32_t m = __ldg(vox + i);
  if (((m >> 24) & 0xffu) == 0u || m == 0u) return 0u;
  const int x = (int)(i % N), y = (int)((i / N) % N), z = (int)(i / ((long long)N * N));
  const int d[6][3] = {{1, 0, 0}, {-1, 0, 0}, {0, 1, 0}, {0, -1, 0}, {0, 0, 1}, {0, 0, -1}};
  uint32_t bits = 0u;
#pragma unroll
  for (int f = 0; f < 6; f++) {
    const int nx = x + d[f][0], ny = y + d[f][1], nz = z + d[f][2];
    const bool in = nx >= 0 && ny >= 0 && nz >= 0 && nx < N && ny < N && nz < N;
    if (!in || __ldg(vox + (size_t)nx + (size_t)ny * N + (size_t)nz * N * N) == 0u) bits |= 1u << f;
  }
  return bits;
}

// Block-wide exclusive scan of v over 1024 threads; returns the prefix, *total the sum.
__device__ __forceinline__ uint32_t block_scan_1024(uint32_t v, uint32_t* total) {
  __shared__ uint32_t warp_sums[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) warp_sums[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    uint32_t s = warp_sums[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += t;
    }
    warp_sums[lane] = s;   // inclusive over warps
  }
  __syncthreads();
  const uint32_t before = warp == 0 ? 0u : warp_sums[warp - 1];
  *total = warp_sums[31];
  return before + incl - v;
}

// A block covers kLightSpan voxels, four consecutive ones (of one row: N is a
// multiple of 8) per thread.
constexpr int kLightSpan = 4096;

// Exposed-face masks of voxels i..i+3, 6 bits each; words: the voxels.
__device__ __forceinline__ uint32_t light_faces4(const uint32_t* __restrict__ vox, int N, long long i, uint32_t* words) {
  const uint4 m = __ldg(reinterpret_cast<const uint4*>(vox + i));
  words[0] = m.x; words[1] = m.y; words[2] = m.z; words[3] = m.w;
  uint32_t bits = 0u;
  if ((m.x | m.y | m.z | m.w) >> 24) {
#pragma unroll
    for (int k = 0; k < 4; k++) bits |= light_faces(vox, N, i + k) << (6 * k);
  }
  return bits;
}

// Bound by the one read of the voxels (64 MB at 256^3): 75 us with one voxel
// per thread.
__global__ void __launch_bounds__(1024) k_light_count(const uint32_t* __restrict__ vox, int N,
                                                      uint32_t* __restrict__ bsum) {
  const long long n3 = (long long)N * N * N;
  const long long i = (long long)blockIdx.x * kLightSpan + 4 * threadIdx.x;
  uint32_t m[4];
  const uint32_t c = i < n3 ? (uint32_t)__popc(light_faces4(vox, N, i, m)) : 0u;
  uint32_t total;
  block_scan_1024(c, &total);
  if (threadIdx.x == 0) bsum[blockIdx.x] = total;
}

// Exclusive scan of the block totals by one block; total count to *count.
__global__ void __launch_bounds__(1024) k_light_offsets(uint32_t* __restrict__ bsum, int nb,
                                                        uint32_t* __restrict__ count) {
  __shared__ uint32_t carry;
  if (threadIdx.x == 0) carry = 0u;
  __syncthreads();
  for (int base = 0; base < nb; base += 1024) {
    const int i = base + threadIdx.x;
    const uint32_t v = i < nb ? bsum[i] : 0u;
    uint32_t total;
    const uint32_t ex = block_scan_1024(v, &total);
    const uint32_t c0 = carry;
    if (i < nb) bsum[i] = c0 + ex;
    __syncthreads();
    if (threadIdx.x == 0) carry = c0 + total;
    __syncthreads();
  }
  if (threadIdx.x == 0) *count = carry;
}

// boff[b]: the lights before block b (boff[blocks]: all of them).
__global__ void __launch_bounds__(1024) k_light_write(const uint32_t* __restrict__ vox, int N,
                                                      const uint32_t* __restrict__ boff, uint32_t* __restrict__ words,
                                                      double* __restrict__ weights) {
  if (boff[blockIdx.x] == boff[blockIdx.x + 1]) return;   // most blocks hold no light
  const long long n3 = (long long)N * N * N;
  const long long i = (long long)blockIdx.x * kLightSpan + 4 * threadIdx.x;
  uint32_t m[4];
  const uint32_t bits = i < n3 ? light_faces4(vox, N, i, m) : 0u;
  uint32_t total;
  uint32_t slot = boff[blockIdx.x] + block_scan_1024((uint32_t)__popc(bits), &total);
  if (!bits) return;
  const uint32_t x = (uint32_t)(i % N), y = (uint32_t)((i / N) % N), z = (uint32_t)(i / ((long long)N * N));
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const uint32_t f6 = (bits >> (6 * k)) & 63u;
    if (!f6) continue;
    const double w = light_weight_d(m[k]);
    for (uint32_t f = 0; f < 6; f++) {
      if (!((f6 >> f) & 1u)) continue;
      words[2 * (size_t)slot] = (x + (uint32_t)k) | (y << 9) | (z << 18) | (f << 27);
      words[2 * (size_t)slot + 1] = m[k];
      weights[slot] = w;
      slot++;
    }
  }
}

// One warp per cell, eight neighbouring cells per block.  The reference keeps
// the first 16 facing lights and then replaces the least of the 16 by any later
// light that ranks above it, so the result depends on the lights' order; but
// few lights replace anything.  The warp ranks 32 lights at a time and runs the
// replacements of those that pass in order (slot k of the 16 in lane k).  The
// block stages 256 lights at a time with the bounds of each 32 (lights are in
// z, y, x order, so 32 of them lie close together), and a warp passes over 32
// whose nearest corner and greatest weight cannot rank.  Distances are exact
// in fp32 (halves up to 512); tests that may pass over a light use bounds
// rounded outwards, and a light that passes them is ranked in doubles as the
// reference does.  9,614 lights at 256^3: 2757 -> 1023 us (a thread per cell, all
// in doubles, waited on one light after another); the serial replacements remain:
// lights come in z order, so cells of high z replace thousands of times.
constexpr int kGridCells = 8, kGridStage = 32 * kGridCells;
struct LightBounds { float lo[3], hi[3], w, pad; };

__global__ void __launch_bounds__(32 * kGridCells) k_light_grid(int N, const uint32_t* __restrict__ words,
                                                                const double* __restrict__ weights, int n,
                                                                uint32_t* __restrict__ grid) {
  __shared__ float4 s_at[kGridStage];       // centre, and the weight rounded up
  __shared__ double s_w[kGridStage];
  __shared__ int s_face[kGridStage];
  __shared__ LightBounds s_box[kGridCells];
  const unsigned full = 0xffffffffu;
  const int BG = N / kBrick, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int cell = blockIdx.x * kGridCells + warp;   // the cells fill the blocks only if there are 8 or more
  const bool real = cell < BG * BG * BG;
  const int bx = cell % BG, by = (cell / BG) % BG, bz = cell / (BG * BG);
  const float ccx = ((float)bx + 0.5f) * kBrick, ccy = ((float)by + 0.5f) * kBrick, ccz = ((float)bz + 0.5f) * kBrick;
  const float eps = (kBrick / 2.0f) * (kBrick / 2.0f);
  const float under = 1.0f - 1e-6f;         // keeps a rounded product below the exact one
  uint32_t topIdx = 0u;                     // lanes 0..15: the kept lights
  float topW = 0.0f;
  int count = 0, minAt = 0;
  float minW = 0.0f;
  for (int base = 0; base < n; base += kGridStage) {
    __syncthreads();
    {
      const int i = base + (int)threadIdx.x;
      float c[3] = {0.0f, 0.0f, 0.0f}, lo[3], hi[3], wu = 0.0f;
      if (i < n) {
        const uint32_t w0 = __ldg(words + 2 * (size_t)i);
        const int face = (int)((w0 >> 27) & 7u), axis = face >> 1, pos = (face & 1) == 0 ? 1 : 0;
#pragma unroll
        for (int a = 0; a < 3; a++) {
          const int v = (int)((w0 >> (9 * a)) & 0x1ffu);
          c[a] = axis == a ? (float)(v + pos) : (float)v + 0.5f;
        }
        const double w = __ldg(weights + i);
        wu = __double2float_ru(w);
        s_w[threadIdx.x] = w;
        s_face[threadIdx.x] = face;
        s_at[threadIdx.x] = make_float4(c[0], c[1], c[2], wu);
      }
#pragma unroll
      for (int a = 0; a < 3; a++) {         // centres are halves: reduce them as integers
        const int h = (int)(2.0f * c[a]);
        lo[a] = 0.5f * (float)__reduce_min_sync(full, i < n ? h : 1 << 20);
        hi[a] = 0.5f * (float)__reduce_max_sync(full, i < n ? h : -1);
      }
      const float wm = __uint_as_float(__reduce_max_sync(full, __float_as_uint(wu)));   // weights are >= 0
      if (lane == 0) s_box[warp] = LightBounds{{lo[0], lo[1], lo[2]}, {hi[0], hi[1], hi[2]}, wm, 0.0f};
    }
    __syncthreads();
    if (!real) continue;
    // the groups of 32 that may rank, one test per lane
    bool may = false;
    if (lane < kGridCells && base + 32 * lane < n) {
      const LightBounds b = s_box[lane];
      const float dx = fmaxf(fmaxf(b.lo[0] - ccx, ccx - b.hi[0]), 0.0f);
      const float dy = fmaxf(fmaxf(b.lo[1] - ccy, ccy - b.hi[1]), 0.0f);
      const float dz = fmaxf(fmaxf(b.lo[2] - ccz, ccz - b.hi[2]), 0.0f);
      const float d2 = dx * dx + dy * dy + dz * dz;
      may = count < kLgK || b.w > minW * fmaxf(d2, eps) * under;
    }
    for (unsigned groups = __ballot_sync(full, may); groups; groups &= groups - 1u) {
      const int k = 32 * (__ffs(groups) - 1) + lane, i = base + k;
      bool pass = false;
      float den = eps;
      if (i < n) {
        const float4 at = s_at[k];
        const float dx = ccx - at.x, dy = ccy - at.y, dz = ccz - at.z;
        const int face = s_face[k], axis = face >> 1;
        const float dn = axis == 0 ? dx : (axis == 1 ? dy : dz);
        den = fmaxf(dx * dx + dy * dy + dz * dz, eps);
        pass = ((face & 1) == 0 ? dn : -dn) > 0.0f && (count < kLgK || at.w > minW * den * under);
      }
      unsigned todo = __ballot_sync(full, pass);
      if (!todo) continue;
      const double w = pass ? s_w[k] / (double)den : 0.0;
      for (; todo; todo &= todo - 1u) {
        const int l = __ffs(todo) - 1;
        const double wl = __shfl_sync(full, w, l);
        const int slot = count < kLgK ? count : minAt;
        if (count == kLgK && !(wl > (double)minW)) continue;
        if (lane == slot) { topIdx = (uint32_t)(i - lane + l); topW = (float)wl; }
        if (count < kLgK) count++;
        if (count == kLgK) {                // the first of the least
          const uint32_t wb = lane < kLgK ? __float_as_uint(topW) : 0xffffffffu;
          const uint32_t m = __reduce_min_sync(full, wb);
          minW = __uint_as_float(m);
          minAt = __ffs(__ballot_sync(full, wb == m)) - 1;
        }
      }
    }
  }
  if (!real) return;
  uint32_t* g = grid + (size_t)cell * kLgStride;
  double wSum = 0.0;
  for (int k = 0; k < count; k++) wSum += (double)__shfl_sync(full, topW, k);
  if (lane == 0) {
    g[0] = (uint32_t)count;
    g[1] = __float_as_uint((float)wSum);
  }
  if (lane < kLgK) {
    g[2 + 2 * lane] = lane < count ? topIdx : 0u;
    g[3 + 2 * lane] = lane < count ? __float_as_uint(topW) : 0u;
  }
}

int light_blocks(int N) { return (int)(((long long)N * N * N + kLightSpan - 1) / kLightSpan); }

cudaError_t launch_light_count(const uint32_t* vox, int N, uint32_t* bsum, uint32_t* count, cudaStream_t st) {
  const int nb = light_blocks(N);
  k_light_count<<<nb, 1024, 0, st>>>(vox, N, bsum);
  k_light_offsets<<<1, 1024, 0, st>>>(bsum, nb, count);
  return cudaGetLastError();
}

cudaError_t launch_light_write(const uint32_t* vox, int N, const uint32_t* boff, uint32_t* words, double* weights,
                               cudaStream_t st) {
  k_light_write<<<light_blocks(N), 1024, 0, st>>>(vox, N, boff, words, weights);
  return cudaGetLastError();
}

cudaError_t launch_light_grid(int N, const uint32_t* words, const double* weights, int n, uint32_t* grid,
                              cudaStream_t st) {
  const int cells = (N / kBrick) * (N / kBrick) * (N / kBrick);
  k_light_grid<<<(cells + kGridCells - 1) / kGridCells, 32 * kGridCells, 0, st>>>(N, words, weights, n, grid);
  return cudaGetLastError();
}

}  // namespace vrt
