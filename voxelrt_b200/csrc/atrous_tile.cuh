// atrous_tile.cuh -- one a-trous iteration (atrous.wgsl:26-83) over a tile of
// 32 x 16 output pixels, shared by the single-image kernel (k_atrous.cu) and
// the batched one (k_batch.cu): 5x5 B3-spline taps at the step, weights
// normal^32 * exp(-(|dt| / (0.05 t + 0.01) + |dL| / sigmaL)),
// sigmaL = max(0.08, 2/sqrt(max(history,1))); sky, out-of-image taps and taps of
// zero normal weight skipped.  The two exponentials are one exp of the summed
// exponents with per-pixel reciprocals (within WGSL's accuracy for '/' and exp).
//
// Bound by arithmetic: 24 taps per pixel of up to 30 fp32 operations (a power
// of 32, an exponential, four sums), all of them part of the bit-exact
// definition.  So the layout serves the instruction count:
//  * Horizontal pixel pairs share packed fp32 instructions (f32x2).  The tile
//    and its halo are staged in shared memory by pairs, in planes of 16 bytes
//    per pair, so that a tap of both pixels is a few loads straight into
//    register pairs.  Taps at odd distances (step 1 only) take halves of two
//    neighbouring pairs.
//  * Each of the 256 threads computes one pair.  (Two pairs, `step` rows apart,
//    whose taps share four rows of five, take 30 tap loads per pair instead of 50, but half
//    the threads stage the tile and walk the taps: three iterations 27 against 15.6 us at 128x72,
//    28.4 / 20.7 at 320x180, 51 / 38 at 800x450, 172.4 / 172.1 at 1920x1080.)
//  * Normals along an axis (every G-buffer of a voxel world) are staged as one
//    code: the power of the dot product is then exactly 1 for equal codes and
//    0 otherwise, a compare and a select instead of ten multiplications.  A
//    tile with any other normal is staged again with the normals in full.
//  * No branches per tap: a tap that the definition skips (outside the image,
//    sky, a zero normal weight) adds a product with a weight of 0.  That
//    changes no bit while every staged colour is finite and not negative (nor
//    -0) and normals' components are at most 1.01; a tile with any other value
//    takes the form that keeps the sums of a skipped tap by a select (kOdd).
//  * The exponent is clamped at 87 instead of selecting 0 past it: the weight
//    is then at most 1.7e-38, which no sum can see while colours stay below
//    1e20 (same check; kOdd selects).
// floor() is a rounded-down addition of 1.5 * 2^23, exact for these exponents
// and without conversions; the signs in exp's polynomial are arranged for the
// negated argument, each product and sum rounding as in exp_nonpos_.
#pragma once
#include "image_core.cuh"

namespace vrt {

constexpr int kAtrousW = 32, kAtrousH = 16;               // a tile
constexpr int kAtrousThreads = kAtrousW * kAtrousH / 2;   // a pair each
constexpr int kAtrousBlocks = 3;                          // an SM

template <int S>
struct AtrousGeom {
  static constexpr int HX = 2 * S;                     // halo
  static constexpr int EW = (kAtrousW + 2 * HX) / 2;   // pairs per row
  static constexpr int NE = EW * (kAtrousH + 2 * HX);
  static constexpr int smem = NE * 64;                 // with the normals in full; 23 / 30 / 48 KB at steps 1 / 2 / 4
};

VRT_DI float2 f2(float x, float y) { return make_float2(x, y); }
VRT_DI float2 f2_fma(float2 a, float2 b, float2 c) {
  float2 r;
  asm("{\n\t.reg .b64 a, b, c, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tmov.b64 c, {%6, %7};\n\t"
      "fma.rn.f32x2 d, a, b, c;\n\tmov.b64 {%0, %1}, d;\n\t}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return r;
}

// A staged pair as loaded.  kUnit: the normal's code in x (0: none); else the
// normal in x, y, z.
struct TapPair { float2 x, y, z, w, r, g, b, l; };

template <bool kUnit>
VRT_DI TapPair load_pair(const float4* sm, int ne, int e) {
  TapPair p;
  const float4 a = sm[e], c = sm[ne + e], d = sm[2 * ne + e];
  p.x = f2(a.x, a.y);
  p.w = f2(a.z, a.w);
  p.r = f2(c.x, c.y);
  p.g = f2(c.z, c.w);
  p.b = f2(d.x, d.y);
  p.l = f2(d.z, d.w);
  if (!kUnit) {
    const float4 n = sm[3 * ne + e];
    p.y = f2(n.x, n.y);
    p.z = f2(n.z, n.w);
  }
  return p;
}
VRT_DI float2 mid(float2 a, float2 b) { return f2(a.y, b.x); }
VRT_DI TapPair between(const TapPair& p, const TapPair& q) {
  return TapPair{mid(p.x, q.x), mid(p.y, q.y), mid(p.z, q.z), mid(p.w, q.w),
                 mid(p.r, q.r), mid(p.g, q.g), mid(p.b, q.b), mid(p.l, q.l)};
}

// The centre pixels of a pair and their running sums.
struct CentrePair {
  float2 x, y, z, w, l, invD, invS, sr, sg, sb, ws;
};

// The tap `t` at kernel weight wk (passed negated: the exponential below
// comes out negated too).
template <bool kUnit, bool kOdd>
VRT_DI void tap_pair(CentrePair& c, const TapPair& t, float nwk) {
  float2 wn;   // -(kernel weight x normal weight)
  bool skip0 = false, skip1 = false;   // kOdd: the definition skips the tap
  if (kUnit) {
    skip0 = c.x.x != t.x.x;
    skip1 = c.x.y != t.x.y;
    wn = f2(skip0 ? 0.0f : nwk, skip1 ? 0.0f : nwk);
  } else {
    float2 nd = f2_fma(c.z, t.z, f2_fma(c.y, t.y, f2_mul(c.x, t.x)));
    nd = kOdd ? f2(fmax_(nd.x, 0.0f), fmax_(nd.y, 0.0f)) : f2(fmaxf(nd.x, 0.0f), fmaxf(nd.y, 0.0f));
    const float2 n2 = f2_mul(nd, nd), n4 = f2_mul(n2, n2), n8 = f2_mul(n4, n4), n16 = f2_mul(n8, n8),
                 n32 = f2_mul(n16, n16);
    wn = f2_mul(n32, f2(nwk, nwk));
    skip0 = n32.x == 0.0f || t.w.x < 0.0f;
    skip1 = n32.y == 0.0f || t.w.y < 0.0f;
  }
  const float2 dt = f2_sub(c.w, t.w), dl = f2_sub(c.l, t.l);
  float2 v = f2_fma(f2(fabsf(dt.x), fabsf(dt.y)), c.invD, f2(fabsf(dl.x) * c.invS.x, fabsf(dl.y) * c.invS.y));
  const bool far0 = !(v.x < 87.0f), far1 = !(v.y < 87.0f);
  if (!kOdd) v = f2(fminf(v.x, 87.0f), fminf(v.y, 87.0f));
  // exp_nonpos_(-v), negated
  const float2 k2 = f2_add_rd(f2_fma(v, f2(-1.44269502f, -1.44269502f), f2(0.5f, 0.5f)), f2(12582912.0f, 12582912.0f));
  const float2 kf = f2_sub(k2, f2(12582912.0f, 12582912.0f));
  float2 r = f2_fma(kf, f2(0.693145751953125f, 0.693145751953125f), v);
  r = f2_fma(kf, f2(1.42860677e-06f, 1.42860677e-06f), r);
  float2 p = f2_fma(r, f2(0.000198412701f, 0.000198412701f), f2(-0.00138888892f, -0.00138888892f));
  p = f2_fma(r, p, f2(0.00833333377f, 0.00833333377f));
  p = f2_fma(r, p, f2(-0.0416666679f, -0.0416666679f));
  p = f2_fma(r, p, f2(0.166666672f, 0.166666672f));
  p = f2_fma(r, p, f2(-0.5f, -0.5f));
  p = f2_fma(r, p, f2(1.0f, 1.0f));
  p = f2_fma(r, p, f2(-1.0f, -1.0f));
  float2 e = f2(__int_as_float(__float_as_int(p.x) + (__float_as_int(k2.x) << 23)),
                __int_as_float(__float_as_int(p.y) + (__float_as_int(k2.y) << 23)));
  if (kOdd) e = f2(far0 ? -0.0f : e.x, far1 ? -0.0f : e.y);
  const float2 w = f2_mul(wn, e);
  if (kOdd) {
    const float2 r2 = f2_fma(t.r, w, c.sr), g2 = f2_fma(t.g, w, c.sg), b2 = f2_fma(t.b, w, c.sb);
    if (!skip0) { c.sr.x = r2.x; c.sg.x = g2.x; c.sb.x = b2.x; c.ws.x = c.ws.x + w.x; }
    if (!skip1) { c.sr.y = r2.y; c.sg.y = g2.y; c.sb.y = b2.y; c.ws.y = c.ws.y + w.y; }
    return;
  }
  c.sr = f2_fma(t.r, w, c.sr);
  c.sg = f2_fma(t.g, w, c.sg);
  c.sb = f2_fma(t.b, w, c.sb);
  // scalar: a packed add of the packed product would be fused with it
  c.ws.x = c.ws.x + w.x;
  c.ws.y = c.ws.y + w.y;
}

// Image of one iteration.
struct AtrousImage {
  int W, H;
  const void* src;
  bool src_f32;
  const float4* gbuf;
  uint2* dst;
};

enum : int { kTileOdd = 1, kTileFullNormals = 2 };   // what staged values ask for

// Stages the tile at (x0, y0) (the halo's corner); returns kTile flags.
template <int S, bool kUnit>
VRT_DI int stage_tile(float4* sm, const AtrousImage& I, int x0, int y0) {
  using G = AtrousGeom<S>;
  constexpr int ne = G::NE;
  int flags = 0;
#pragma unroll 2
  for (int e = threadIdx.x; e < ne; e += kAtrousThreads) {
    const int qy = y0 + e / G::EW, qx = x0 + 2 * (e % G::EW);
    float4 g[2], c[2];
#pragma unroll
    for (int k = 0; k < 2; k++) {
      g[k] = make_float4(0.0f, 0.0f, 0.0f, -1.0f);   // outside the image: as sky
      c[k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      if ((unsigned)qy < (unsigned)I.H && (unsigned)(qx + k) < (unsigned)I.W) {
        const size_t q = (size_t)qy * I.W + (qx + k);
        g[k] = I.gbuf[q];
        c[k] = load_px(I.src, I.src_f32, q);
      }
    }
    float lum[2], code[2];
#pragma unroll
    for (int k = 0; k < 2; k++) {
      float4& gk = g[k];
      float4& ck = c[k];
      if (gk.w < 0.0f) {   // sky: drops out through its zero normal
        gk = make_float4(0.0f, 0.0f, 0.0f, -1.0f);
        ck = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      }
      // negative (and -0), infinite and NaN colours and distances all lie above the bound as bit patterns
      const uint32_t cb = max(max(__float_as_uint(ck.x), __float_as_uint(ck.y)), __float_as_uint(ck.z));
      if (cb >= 0x60ad78ecu || (__float_as_uint(gk.w) > 0x7f7fffffu && gk.w != -1.0f)) flags |= kTileOdd;   // 1e20
      lum[k] = luminance(ck.x, ck.y, ck.z);
      const float ax = fabsf(gk.x), ay = fabsf(gk.y), az = fabsf(gk.z);
      if (kUnit) {
        // components 0 or +-1, at most one of them not 0
        if (!(ax * ax == ax && ay * ay == ay && az * az == az && ax + ay + az <= 1.0f)) flags |= kTileFullNormals;
        code[k] = gk.x + 2.0f * gk.y + 3.0f * gk.z;
      } else if (!(ax <= 1.01f && ay <= 1.01f && az <= 1.01f)) {
        flags |= kTileOdd;
      }
    }
    sm[e] = kUnit ? make_float4(code[0], code[1], g[0].w, g[1].w) : make_float4(g[0].x, g[1].x, g[0].w, g[1].w);
    sm[ne + e] = make_float4(c[0].x, c[1].x, c[0].y, c[1].y);
    sm[2 * ne + e] = make_float4(c[0].z, c[1].z, lum[0], lum[1]);
    if (!kUnit) sm[3 * ne + e] = make_float4(g[0].y, g[1].y, g[0].z, g[1].z);
  }
  return flags;
}

// This thread's pair: pixels px, px + 1 of image row y, staged at pair column pc of row ly (the halo's corner is
// row 0).  alpha: their history lengths.  kOdd: the staged tile holds a value that asks for it.
template <int S, bool kUnit, bool kOdd>
VRT_DI void filter_pair(const float4* sm, const AtrousImage& I, int pc, int ly, int px, int y, const float (&alpha)[2]) {
  using G = AtrousGeom<S>;
  constexpr int ne = G::NE;
  CentrePair c;
  bool live = false;
  {
    const TapPair p = load_pair<kUnit>(sm, ne, (ly + G::HX) * G::EW + pc + G::HX / 2);
    c.x = p.x; c.y = p.y; c.z = p.z; c.w = p.w; c.l = p.l;
    if (kUnit) {   // a pixel without a normal matches no tap
      if (c.x.x == 0.0f) c.x.x = 8.0f;
      if (c.x.y == 0.0f) c.x.y = 8.0f;
    }
    const float cr[2] = {p.r.x, p.r.y}, cg[2] = {p.g.x, p.g.y}, cb[2] = {p.b.x, p.b.y}, gw[2] = {p.w.x, p.w.y};
    float invD[2], invS[2], sr[2], sg[2], sb[2];
#pragma unroll
    for (int k = 0; k < 2; k++) {
      live = live || !(gw[k] < 0.0f);   // in the image and not sky
      const float history = fmax_(alpha[k], 1.0f);
      const float sigmaL = fmax_(0.08f, 2.0f / __fsqrt_rn(history));
      invD[k] = 1.0f / (0.05f * gw[k] + 0.01f);
      invS[k] = 1.0f / sigmaL;
      sr[k] = (cr[k] * 0.375f) * 0.375f;
      sg[k] = (cg[k] * 0.375f) * 0.375f;
      sb[k] = (cb[k] * 0.375f) * 0.375f;
    }
    c.invD = f2(invD[0], invD[1]);
    c.invS = f2(invS[0], invS[1]);
    c.sr = f2(sr[0], sr[1]);
    c.sg = f2(sg[0], sg[1]);
    c.sb = f2(sb[0], sb[1]);
    c.ws = f2(0.140625f, 0.140625f);
  }
  if (live) {
#pragma unroll 1
    for (int j = 0; j < 5; j++) {   // tap rows (j - 2) S
      const float wy = j == 2 ? 0.375f : ((j == 1 || j == 3) ? 0.25f : 0.0625f);
      const int e = (ly + j * S) * G::EW + pc;
      TapPair prev;
#pragma unroll
      for (int dx = -2; dx <= 2; dx++) {
        TapPair tp;
        if (S > 1) {
          tp = load_pair<kUnit>(sm, ne, e + (G::HX + dx * S) / 2);
        } else if (dx & 1) {
          const TapPair next = load_pair<kUnit>(sm, ne, e + (dx + 3) / 2);
          tp = between(prev, next);
          prev = next;
        } else if (dx == -2) {
          prev = tp = load_pair<kUnit>(sm, ne, e);
        } else {
          tp = prev;
        }
        if (dx != 0 || j != 2) tap_pair<kUnit, kOdd>(c, tp, -(b3_weight(dx) * wy));
      }
    }
  }
#pragma unroll
  for (int k = 0; k < 2; k++) {
    if (px + k >= I.W || y >= I.H) continue;
    const size_t i = (size_t)y * I.W + (px + k);
    float4 v;
    if ((k ? c.w.y : c.w.x) < 0.0f) {
      v = load_px(I.src, I.src_f32, i);   // sky passes through
    } else {
      v.w = alpha[k];
      const float den = fmax_(k ? c.ws.y : c.ws.x, 1e-6f);
      v.x = (k ? c.sr.y : c.sr.x) / den;
      v.y = (k ? c.sg.y : c.sg.x) / den;
      v.z = (k ? c.sb.y : c.sb.x) / den;
    }
    I.dst[i] = pack_h4(v.x, v.y, v.z, v.w);
  }
}

// The tile at (x0, y0) (multiples of 32 and 16); all kAtrousThreads threads of
// the block call it.  sm: AtrousGeom<S>::smem bytes.
template <int S>
VRT_DI void atrous_tile(float4* sm, const AtrousImage& I, int x0, int y0) {
  using G = AtrousGeom<S>;
  const int pc = threadIdx.x & 15, ly = threadIdx.x >> 4, px = x0 + 2 * pc, y = y0 + ly;
  float alpha[2];   // arrives while the tile is staged; 1 outside the image
#pragma unroll
  for (int k = 0; k < 2; k++)
    alpha[k] = px + k < I.W && y < I.H ? load_px(I.src, I.src_f32, (size_t)y * I.W + (px + k)).w : 1.0f;
  int flags = stage_tile<S, true>(sm, I, x0 - G::HX, y0 - G::HX);
  bool odd = __syncthreads_or(flags & kTileOdd) != 0;
  const bool full = __syncthreads_or(flags & kTileFullNormals) != 0;
  if (!full) {
    if (!odd) filter_pair<S, true, false>(sm, I, pc, ly, px, y, alpha);
    else filter_pair<S, true, true>(sm, I, pc, ly, px, y, alpha);
    return;
  }
  flags = stage_tile<S, false>(sm, I, x0 - G::HX, y0 - G::HX);
  odd = __syncthreads_or(flags & kTileOdd) != 0;
  if (!odd) filter_pair<S, false, false>(sm, I, pc, ly, px, y, alpha);
  else filter_pair<S, false, true>(sm, I, pc, ly, px, y, alpha);
}

}  // namespace vrt
