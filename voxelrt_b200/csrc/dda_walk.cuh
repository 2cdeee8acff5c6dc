// dda_walk.cuh -- the two-level brick -> voxel DDA (voxel.wgsl:73-153) as a
// resumable walk for the queue tracer: test the current cell, then step.
//
// Issue slots bound this walk (its working set is in L1 / L2), and a warp runs
// every transition -- entering a brick, leaving it, ending -- that any of its
// lanes needs, so the walk is laid out for a short step that only notes a due
// transition (walk_step), and the transitions run for all lanes that wait for
// one every few steps (transition):
//
//  * One 32-bit word V holds the current level's linear cell index and its
//    step count, and a step adds one per-axis constant to it:
//      brick level: bits 0-21 the cell of the padded brick grid, bits 22-30 the
//        brick tests done, biased so that bit 31 becomes set at 3 BG + 2;
//      voxel level: bits 0-10 lx + 8 ly + 64 lz + 512 (the bias keeps a step
//        out of the brick from borrowing), bits 11 / 15 / 19 three four-bit
//        fields that count each axis up from its distance to the brick's face
//        behind the ray (a field's top bit set: the ray left on that axis),
//        bits 23-27 the voxel tests done, biased so that bit 28 becomes set at 24.
//    One AND with the level's guard bits is then the bounds check and the
//    iteration cap together, and the per-step counters cost nothing.
//  * The brick grid is padded by one cell on each side.  Border cells read as
//    occupied and their masks as full, so that a brick step needs no bounds
//    check: a ray that leaves the world "hits" the border, and finish() tells.
//  * Both levels' tests are one load at the same base (DScene::cells: the
//    padded bitmap, then 16 mask words per padded cell).
//  * Entering a brick floors through a rounded-down addition of 1.5 * 2^23
//    instead of conversions, and compares the cell of the result with the
//    walk's cell; only where they differ (the reference clamps there) is the
//    cell index taken apart.
//
// Every float operation and every decision is the reference's, so hits, t and
// the counters are bit-identical to the nested loops (vrt_device.cuh, trace()).
// kWide: grids over 128^3 bricks, whose cell index leaves no room for the
// count: the brick tests are counted in a word of their own.
#pragma once
#include "vrt_device.cuh"

namespace vrt {

// Normal of a hit on entry axis `vax` for direction rd (same value the DDA
// returns: -vmask * sign(rd)).
VRT_DI F3 hit_normal(int vax, F3 rd) {
  const int sx = rd.x > 0.0f ? 1 : (rd.x < 0.0f ? -1 : 0);
  const int sy = rd.y > 0.0f ? 1 : (rd.y < 0.0f ? -1 : 0);
  const int sz = rd.z > 0.0f ? 1 : (rd.z < 0.0f ? -1 : 0);
  return f3(face_normal_component(vax == 0, sx), face_normal_component(vax == 1, sy),
            face_normal_component(vax == 2, sz));
}

// Walk states.  kWalkOdd: a direction component below the bound at which
// safe_inv clamps its reciprocal (0 and NaN among them), or values so large that
// a point on the ray may lie far from its cell.
enum : int { kWalkVoxel = 1, kWalkOdd = 2, kWalkOcc = 4, kWalkOut = 8, kWalkDone = 16, kWalkWaits = 4 };

constexpr uint32_t kCntB = 1u << 22, kCntV = 1u << 23;
constexpr uint32_t kIdxB = kCntB - 1u;              // cell index of the narrow form's brick level
constexpr uint32_t kGuardB = 0x80000000u;
constexpr uint32_t kGuardV = (8u << 11) | (8u << 15) | (8u << 19) | (1u << 28);
constexpr uint32_t kStartV = 512u + 8u * kCntV;     // 32 - 24 tests
constexpr float kFloorMagic = 12582912.0f;          // 1.5 * 2^23
constexpr uint32_t kFloorBits = 0x4b400000u;        // its bit pattern

template <bool kWide>
struct Walk {
  F3 ro, d, tm, tmB;            // d = 1 / rd x (8 at brick level, 1 at voxel level); tm: next planes
  float t, tExit, tLim, maxT;   // tLim: tExit at brick level, infinity at voxel level
  uint32_t V, Vb;               // current level's word; the brick level's while walking voxels
  uint32_t dX, dY, dZ, last;    // the level's steps; the last step taken
  uint32_t bX, bY, bZ, vX, vY, vZ;   // the steps of the brick and of the voxel level
  uint32_t mirror;              // 7 in the four-bit field of each axis the ray walks down
  F3 cg;                        // kFloorMagic - (rd >= 0)
  uint32_t base, wm, gm;        // test word ((V >> 5) & wm) | base of the cells; guard bits
  uint32_t nb;                  // kWide: brick tests done
  int st;
  float tHit;
  uint32_t mat;

  VRT_DI bool walking() const { return st < kWalkWaits; }
  VRT_DI bool done() const { return (st & kWalkDone) != 0; }

  VRT_DI void brick_level() {
    dX = bX; dY = bY; dZ = bZ;
    gm = kWide ? 0u : kGuardB;
    wm = kWide ? 0x07ffffffu : kIdxB >> 5;
    base = 0u;
    tLim = tExit;
  }

  VRT_DI void init(const DScene& S, F3 roW, F3 rd, float maxTW) {
    ro = roW * kInvVoxel;
    maxT = maxTW * kInvVoxel;
    const float sgx = rd.x >= 0.0f ? 1.0f : -1.0f;
    const float sgy = rd.y >= 0.0f ? 1.0f : -1.0f;
    const float sgz = rd.z >= 0.0f ? 1.0f : -1.0f;
    const F3 inv = f3(safe_inv(sgx, rd.x), safe_inv(sgy, rd.y), safe_inv(sgz, rd.z));
    const F3 stepGE = f3(rd.x >= 0.0f ? 1.0f : 0.0f, rd.y >= 0.0f ? 1.0f : 0.0f, rd.z >= 0.0f ? 1.0f : 0.0f);
    const float G = (float)S.N;
    const F3 t0 = f3(__fsub_rn(0.0f, ro.x), __fsub_rn(0.0f, ro.y), __fsub_rn(0.0f, ro.z)) * inv;
    const F3 t1 = (f3(G, G, G) - ro) * inv;
    const F3 tmin3 = min3(t0, t1);
    const F3 tmax3 = max3(t0, t1);
    const float tEnter = fmax_(fmax_(tmin3.x, tmin3.y), fmax_(tmin3.z, 0.0f));
    tExit = fmin_(fmin_(tmax3.x, tmax3.y), fmin_(tmax3.z, maxT));
    V = kWide ? 0u : (512u - 3u * (uint32_t)S.BG - 2u) * kCntB;   // no tests yet
    nb = 0u;
    if (tEnter > tExit) { st = kWalkDone; return; }
    const float ax = fabsf(rd.x), ay = fabsf(rd.y), az = fabsf(rd.z);
    // A clamped reciprocal lets the point on the ray lag whole worlds behind the walk's cell, where descend()'s
    // comparison of linear indices could take it for another one.
    const bool plain = ax >= 1e-8f && ay >= 1e-8f && az >= 1e-8f && ax < 8.0f && ay < 8.0f && az < 8.0f &&
                       fabsf(ro.x) < 1048576.0f && fabsf(ro.y) < 1048576.0f && fabsf(ro.z) < 1048576.0f;
    st = plain ? 0 : kWalkOdd;
    t = tEnter;
    const F3 sp = ro + rd * (t + 1e-4f);
    // x / 8 as x * 0.125: the same real number, so the same rounding
    const int cx = iclamp_(ifloor_(sp.x * 0.125f), 0, S.BG - 1);
    const int cy = iclamp_(ifloor_(sp.y * 0.125f), 0, S.BG - 1);
    const int cz = iclamp_(ifloor_(sp.z * 0.125f), 0, S.BG - 1);
    tm = ((f3((float)cx, (float)cy, (float)cz) + stepGE) * 8.0f - ro) * inv;
    d = inv * 8.0f;
    const uint32_t P = (uint32_t)S.BG + 2u;
    V += (uint32_t)(cx + 1) + P * ((uint32_t)(cy + 1) + P * (uint32_t)(cz + 1));
    const uint32_t P2 = P * P, cb = kWide ? 0u : kCntB;
    const bool gx = rd.x >= 0.0f, gy = rd.y >= 0.0f, gz = rd.z >= 0.0f;
    bX = gx ? cb + 1u : cb - 1u;
    bY = gy ? cb + P : cb - P;
    bZ = gz ? cb + P2 : cb - P2;
    vX = gx ? kCntV + 2048u + 1u : kCntV + 2048u - 1u;
    vY = gy ? kCntV + 32768u + 8u : kCntV + 32768u - 8u;
    vZ = gz ? kCntV + 524288u + 64u : kCntV + 524288u - 64u;
    mirror = (gx ? 0u : 7u) | (gy ? 0u : 0x70u) | (gz ? 0u : 0x700u);
    cg = f3(gx ? kFloorMagic - 1.0f : kFloorMagic, gy ? kFloorMagic - 1.0f : kFloorMagic,
            gz ? kFloorMagic - 1.0f : kFloorMagic);
    if (!plain) {   // an axis whose component is 0 (or NaN) takes its steps in place
      if (!(ax > 0.0f)) { bX = cb; vX = kCntV; }
      if (!(ay > 0.0f)) { bY = cb; vY = kCntV; }
      if (!(az > 0.0f)) { bZ = cb; vZ = kCntV; }
    }
    brick_level();
    last = (tmin3.x >= tmin3.y && tmin3.x >= tmin3.z) ? dX : (tmin3.y >= tmin3.z ? dY : dZ);
  }

  // The reference's axis choice and step; true: the walk of this level ends.
  VRT_DI bool advance(const DScene& S) {
    const bool px = tm.x <= tm.y && tm.x <= tm.z;
    const bool py = !px && tm.y <= tm.z;
    t = px ? tm.x : (py ? tm.y : tm.z);
    last = px ? dX : (py ? dY : dZ);
    V += last;
    if (px) tm.x = t + fabsf(d.x);
    else if (py) tm.y = t + fabsf(d.y);
    else tm.z = t + fabsf(d.z);
    bool out = (V & gm) != 0u || t > tLim;
    if (kWide) {
      if (!(st & kWalkVoxel)) {
        nb++;
        out = out || nb >= 3u * (uint32_t)S.BG + 2u;
      }
    }
    return out;
  }

  // Up to kRun tests, each followed by a step where the cell is empty, until a
  // transition is due.
  template <int kRun>
  VRT_DI void walk_run(const DScene& S) {
    if (!walking()) return;
#pragma unroll
    for (int q = 0; q < kRun; q++) {
      const uint32_t word = __ldg(S.cells + (((V >> 5) & wm) | base));
      if ((word >> (V & 31u)) & 1u) { st |= kWalkOcc; return; }
      if (advance(S)) { st |= kWalkOut; return; }
    }
  }

  // The transition a waiting lane is due.  rd: the ray's direction.
  VRT_DI void transition(const DScene& S, F3 rd, DCount& c) {
    if (st & kWalkOut) {
      if (!(st & kWalkVoxel)) { st = kWalkDone; return; }
      // left the brick: the brick level's state comes back and takes its step
      c.inner += (V >> 23) - 8u;
      V = Vb;
      tm = tmB;
      const float2 d2 = f2_mul(make_float2(d.x, d.y), make_float2(8.0f, 8.0f));
      d = f3(d2.x, d2.y, d.z * 8.0f);
      st &= kWalkOdd;
      brick_level();
      if (advance(S)) st = kWalkDone;
    } else if (st & kWalkVoxel) {
      st |= kWalkDone;              // a voxel hit, or the border: finish() tells
    } else {
      descend(S, rd);
    }
  }

  // Coordinates of cell index idx in the padded grid, less 1.
  VRT_DI void cell_of(const DScene& S, uint32_t idx, int& bx, int& by, int& bz) const {
    const uint32_t P = (uint32_t)S.BG + 2u, P2 = P * P;
    uint32_t z = __umulhi(idx, S.rP2), r = idx - z * P2;
    if ((int)r < 0) { z--; r += P2; }   // the reciprocals are rounded up: at most one too many
    uint32_t y = __umulhi(r, S.rP), x = r - y * P;
    if ((int)x < 0) { y--; x += P; }
    bx = (int)x - 1; by = (int)y - 1; bz = (int)z - 1;
  }
  VRT_DI uint32_t cell(uint32_t v) const { return kWide ? v : v & kIdxB; }

  // Into the occupied (or border) cell (voxel.wgsl:104-109).
  VRT_DI void descend(const DScene& S, F3 rd) {
    const uint32_t P = (uint32_t)S.BG + 2u, P2 = P * P, idx = cell(V);
    const float te = t + 1e-4f;
    // not as a packed multiply and a packed add: the assembler fuses those into one rounding
    const float2 p2 = make_float2(ro.x + rd.x * te, ro.y + rd.y * te);
    const F3 p = f3(p2.x, p2.y, ro.z + rd.z * te);
    const float2 m2 = f2_add_rd(p2, make_float2(kFloorMagic, kFloorMagic));
    float mx = m2.x, my = m2.y, mz = __fadd_rd(p.z, kFloorMagic);
    uint32_t ix = __float_as_uint(mx), iy = __float_as_uint(my), iz = __float_as_uint(mz);
    // the cell of floor(p), from the patterns themselves (their constant part is a multiple of 8)
    const uint32_t near = (ix >> 3) + P * (iy >> 3) + P2 * (iz >> 3) - (kFloorBits / 8u - 1u) * (1u + P + P2);
    if (near != idx || (st & kWalkOdd)) {
      int bx, by, bz;
      cell_of(S, idx, bx, by, bz);
      const int vx = iclamp_(ifloor_(p.x), bx * kBrick, bx * kBrick + 7);
      const int vy = iclamp_(ifloor_(p.y), by * kBrick, by * kBrick + 7);
      const int vz = iclamp_(ifloor_(p.z), bz * kBrick, bz * kBrick + 7);
      mx = (float)vx + kFloorMagic; my = (float)vy + kFloorMagic; mz = (float)vz + kFloorMagic;
      ix = (uint32_t)vx; iy = (uint32_t)vy; iz = (uint32_t)vz;
    }
    Vb = V;
    tmB = tm;
    const float2 d2 = f2_mul(make_float2(d.x, d.y), make_float2(0.125f, 0.125f));
    d = f3(d2.x, d2.y, d.z * 0.125f);
    // (voxel + (rd >= 0)) - ro: the first difference is exact
    const float2 t2 = f2_mul(f2_sub(f2_sub(make_float2(mx, my), make_float2(cg.x, cg.y)), make_float2(ro.x, ro.y)), d2);
    tm = f3(t2.x, t2.y, ((mz - cg.z) - ro.z) * d.z);
    const uint32_t lx = ix & 7u, ly = iy & 7u, lz = iz & 7u;
    V = kStartV + (lx + 8u * ly + 64u * lz) + (((lx + 16u * ly + 256u * lz) ^ mirror) << 11);
    dX = vX; dY = vY; dZ = vZ;
    base = idx * 16u + S.mw;
    wm = 15u;
    gm = kGuardV;
    tLim = __int_as_float(0x7f800000);
    st = (st & kWalkOdd) | kWalkVoxel;
  }

  // Brick tests done so far (the reference's outer iterations).
  VRT_DI uint32_t brick_tests(const DScene& S, uint32_t v) const {
    return kWide ? nb : (v >> 22) - (512u - 3u * (uint32_t)S.BG - 2u);
  }

  // Entry axis of a hit: the axis of the last step (at either level), or of
  // the world's entry face; 3 for an axis whose direction component is 0,
  // whose normal is 0 in every component.
  VRT_DI int hit_axis(const DScene& S) const {
    const uint32_t P = (uint32_t)S.BG + 2u;
    int a = (int)last;
    int px = 1, py = (int)P, pz = (int)(P * P);
    if (a >= (int)kCntV) {            // a step in the brick
      a -= (int)kCntV;
      px = 2048; py = 32768; pz = 524288;
      a = (a + 512) & ~1023;          // the axis's field alone
    } else if (!kWide) {
      a -= (int)kCntB;
    }
    a = abs(a);
    return a == px ? 0 : (a == py ? 1 : (a == pz ? 2 : 3));
  }

  // The counters, tHit and mat of a finished walk; true when it hit a voxel
  // (vx, vy, vz) within maxT.
  VRT_DI bool finish(const DScene& S, DCount& c, int& vx, int& vy, int& vz) {
    tHit = -1.0f;
    mat = 0u;
    if (!(st & kWalkVoxel)) {
      c.outer += brick_tests(S, V);
      return false;
    }
    c.outer += brick_tests(S, Vb);
    int bx, by, bz;
    cell_of(S, cell(Vb), bx, by, bz);
    if (max(max((uint32_t)bx, (uint32_t)by), (uint32_t)bz) >= (uint32_t)S.BG) return false;   // left the world
    c.outer++;
    c.inner += (V >> 23) - 7u;
    vx = bx * kBrick + (int)(V & 7u);
    vy = by * kBrick + (int)((V >> 3) & 7u);
    vz = bz * kBrick + (int)((V >> 6) & 7u);
    c.vreads++;
    if (t > maxT) return false;
    mat = __ldg(S.vox + ((uint32_t)vx + (uint32_t)vy * (uint32_t)S.N + (uint32_t)vz * (uint32_t)(S.N * S.N)));
    tHit = t * kVoxelSize;
    return true;
  }
  VRT_DI void finish(const DScene& S, DCount& c) {
    int vx, vy, vz;
    finish(S, c, vx, vy, vz);
  }
};

}  // namespace vrt
