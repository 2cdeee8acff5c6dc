// wavefront_core.cuh -- building blocks of the wavefront path tracer shared by
// the single-session kernels (k_wavefront.cu) and the batched kernels
// (k_batch.cu): path-state layout, block-aggregated queue appends, the queue
// tracer, and per-vertex shading.
#pragma once
#include "dda_walk.cuh"
#include "vrt_device.cuh"
#include "vrt_internal.h"
#include <algorithm>
#include <cstring>

namespace vrt {


constexpr uint32_t kFlagShadow = 1u;     // a shadow ray of the previous vertex is pending
constexpr uint32_t kFlagTerminal = 2u;   // no bounce ray: finalize after the shadow ray
constexpr uint32_t kShadowBit = 0x80000000u;
constexpr uint32_t kFlagShadow2 = 4u;           // a second shadow ray of the previous vertex is pending

struct WfDev {
  float4* R0;      // ray origin of waves 1..: surf = pos + n*1e-3 (primary rays start at the camera)
  float4* R1;      // primary / bounce direction; w = RNG state bits in wave 0
  float4* R2;      // direction (xyz) and maxT (w) of the pending shadow ray
  float4* S0;      // radiance xyz, w = RNG state bits (waves 1..)
  float4* S1;      // throughput xyz, w = primary material bits
  float4* S2;      // pending sun contribution xyz, w = flags
  uint4* hit;      // x = t bits, y = material, z = entry axis, w = shadow occluded
  uint32_t* q0;    // ray queues (entry = path | kShadowBit for shadow rays), capacity 3P; a path's second
                   // shadow ray uses path index g + P (R0, R2 and hit hold 2P entries where it is used)
  uint32_t* q1;
  uint32_t* a0;    // active path lists, capacity P
  uint32_t* a1;
  int* ctr;        // per wave k: [4k] shadow rays (queue front), [4k+1] queue head, [4k+2] active count,
                   // [4k+3] bounce rays (queue back)
  int* act2;       // per wave k: paths at the back of the active list (a list in two parts: path i of the
                   // back part sits at acap - 1 - i)
  uint32_t qcap;   // queue capacity in entries: bounce ray i of a wave sits at qcap - 1 - i
  uint32_t acap;   // active-list capacity
};

// Ray queues: a wave's shadow rays are appended from the front, its bounce
// rays from the back (bounce ray i at qcap - 1 - i), so a tracer warp takes
// runs of one kind -- shadow rays of neighbouring paths share the sun
// direction and much of their walks.

VRT_DI uint32_t* queue_of(const WfDev& b, int wave) { return (wave & 1) ? b.q1 : b.q0; }
VRT_DI uint32_t* active_of(const WfDev& b, int wave) { return (wave & 1) ? b.a1 : b.a0; }

// Warp-aggregated append: one atomicAdd per warp, slots in lane order.  All
// 32 lanes must call it (pred false for lanes with nothing to append).
VRT_DI uint32_t warp_append(int* counter, bool pred) {
  const unsigned mask = __ballot_sync(0xffffffffu, pred);
  if (!mask) return 0u;
  const int lane = threadIdx.x & 31;
  const int leader = __ffs(mask) - 1;
  int base = 0;
  if (lane == leader) base = atomicAdd(counter, __popc(mask));
  base = __shfl_sync(0xffffffffu, base, leader);
  return (uint32_t)base + (uint32_t)__popc(mask & ((1u << lane) - 1u));
}

VRT_DI F3 xyz(float4 v) { return f3(v.x, v.y, v.z); }

// ---------------------------------------------------------------------------
// Job policies.  A "job" is one view (session) rendered in a wave: uniforms,
// scene, size and output buffers.  Path state is indexed by a global pixel id
// g (jobs are laid out back to back); outputs by the job-local pixel id.
// ---------------------------------------------------------------------------
struct JobOut {
  uint2* rad16;     // rgba16f demodulated radiance
  float4* rad32;    // optional fp32 copy
  uint32_t* alb8;   // rgba8 sqrt albedo
  float4* gbuf;     // rgba32f normal + distance of this frame
};

// One session: everything in kernel parameters.
struct SingleJob {
  Uni u;
  DScene S;
  JobOut out;
  CacheDev cc;             // radiance cache (cc.on == 0: plain path)
  float fclamp;
  int W, H;
  __host__ __device__ bool any_cache() const { return cc.on != 0; }
  VRT_DI const CacheDev& cache(int) const { return cc; }
  VRT_DI int job_of(uint32_t) const { return 0; }
  VRT_DI int job_of_warp(uint32_t) const { return 0; }
  VRT_DI int job_of_cached(uint32_t, int&, uint32_t&, uint32_t&) const { return 0; }
  VRT_DI const Uni& uni(int) const { return u; }
  VRT_DI DScene scene(int) const { return S; }
  VRT_DI JobOut outs(int) const { return out; }
  VRT_DI float clamp(int) const { return fclamp; }
  VRT_DI int width(int) const { return W; }
  VRT_DI int height(int) const { return H; }
  VRT_DI uint32_t first(int) const { return 0u; }
  bool wide() const { return S.BG > kNarrowBG; }
};

// Device job table entry of a batch (one per session in the batch).
struct JobDev {
  Uni u;
  DScene S;
  JobOut out;
  int W, H;
  uint32_t first;          // first global pixel of the job
  float fclamp;
  // image passes of the frame
  const void* acc_prev;    // history read by temporal (rgba16f / rgba32f)
  void* acc_cur;           // history written by temporal
  const float4* gbuf_prev;
  uint2* den0;             // a-trous ping-pong (dA, dB)
  uint2* den1;
  uint32_t* ldr;
  int acc_f32;
  int pad[3];
  CacheDev cache;          // radiance cache of the job's session (cache.on == 0: plain path)
};

// The last of n ascending values (the first is 0) that is not above v, which all lanes of the warp hold; all
// lanes call it.
VRT_DI int last_at_or_before(const uint32_t* __restrict__ a, int n, uint32_t v) {
  const int lane = threadIdx.x & 31;
  int c = 0;
  for (int base = 0; base < n; base += 32) {
    const unsigned m = __ballot_sync(0xffffffffu, base + lane < n && __ldg(a + base + lane) <= v);
    c += __popc(m);
    if (m != 0xffffffffu) break;
  }
  return c - 1;
}

// Many sessions: job table in device memory, job found by search on the sorted
// first-pixel array.
struct MultiJob {
  const JobDev* jobs;
  const uint32_t* firsts;  // n entries, ascending
  int n;
  int cache_jobs;          // jobs with the cache on
  int max_bg;              // largest brick grid side of the jobs' scenes
  bool wide() const { return max_bg > kNarrowBG; }
  __host__ __device__ bool any_cache() const { return cache_jobs != 0; }
  VRT_DI const CacheDev& cache(int j) const { return jobs[j].cache; }
  VRT_DI int job_of(uint32_t g) const {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (__ldg(firsts + mid) <= g) lo = mid;
      else hi = mid - 1;
    }
    return lo;
  }
  // job_of for a whole warp whose lanes hold consecutive pixels (all lanes call it; a pixel past the last
  // one gives some job): one load per 32 jobs instead of a dependent load per halving
  VRT_DI int job_of_warp(uint32_t g) const {
    const uint32_t g0 = __shfl_sync(0xffffffffu, g, 0);
    const int lo = last_at_or_before(firsts, n, g0);
    return __any_sync(0xffffffffu, lo + 1 < n && __ldg(firsts + lo + 1) <= g) ? job_of(g) : lo;
  }
  // job_of with the caller's last answer (job jc for pixels [lo, hi), lo <= hi; lo == hi: none)
  // tried first
  VRT_DI int job_of_cached(uint32_t g, int& jc, uint32_t& lo, uint32_t& hi) const {
    if (g - lo < hi - lo) return jc;
    jc = job_of(g);
    lo = __ldg(firsts + jc);
    hi = jc + 1 < n ? __ldg(firsts + jc + 1) : 0xffffffffu;
    return jc;
  }
  VRT_DI const Uni& uni(int j) const { return jobs[j].u; }
  VRT_DI DScene scene(int j) const { return jobs[j].S; }
  VRT_DI JobOut outs(int j) const { return jobs[j].out; }
  VRT_DI float clamp(int j) const { return jobs[j].fclamp; }
  VRT_DI int width(int j) const { return jobs[j].W; }
  VRT_DI int height(int j) const { return jobs[j].H; }
  VRT_DI uint32_t first(int j) const { return jobs[j].first; }
};

// ---------------------------------------------------------------------------
// radiance cache hooks (single session).  With the cache on, 1/16 of the
// pixels (one position of every 4x4 block, rotating per frame) trace full
// training paths of `train_bounces` bounces and record their first
// `rec_vertices` vertices; every other path ends at its first bounce hit
// (vertex 1): its emission is picked up there and the reflected radiance at
// that point is queried from the network after the waves.
// ---------------------------------------------------------------------------
enum : int { kRolePlain = 0, kRoleTrain = 1, kRoleQuery = 2 };

VRT_DI int cache_role(const CacheDev& c, uint32_t lp, int W) {
  if (!c.on) return kRolePlain;
  const uint32_t x = lp % (uint32_t)W, y = lp / (uint32_t)W;
  return ((x & 3u) == (c.phase & 3u) && (y & 3u) == (c.phase >> 2)) ? kRoleTrain : kRoleQuery;
}

VRT_DI uint32_t train_index(const CacheDev& c, uint32_t lp, int W) {
  const uint32_t x = lp % (uint32_t)W, y = lp / (uint32_t)W;
  return (y >> 2) * (uint32_t)c.TW + (x >> 2);
}

// Record slot of vertex k of a training path (nullptr: nothing to record).
VRT_DI float4* rec_slot(const CacheDev& c, int role, uint32_t lp, int W, uint32_t k) {
  if (role != kRoleTrain || (int)k >= c.rec_vertices) return nullptr;
  const uint32_t ti = train_index(c, lp, W);
  c.rec_n[ti] = (int)k + 1;
  return c.rec + ((size_t)ti * kCacheMaxRec + k) * 4;
}

VRT_DI float cache_target(float rfin, float rk, float tpk, float clampv) {
  float v = tpk > 1e-6f ? (rfin - rk) / tpk : 0.0f;
  v = fmax_(v, 0.0f);
  if (clampv > 0.0f) v = fmin_(v, clampv);
  return v;
}

// The counter that every thread of the block with want set appends to, when
// it is one counter (a single job's), or null when no thread appends; false
// when the threads append to different counters (several jobs of a batch in
// one block).  All threads of the block call it.
VRT_DI bool block_common_counter(int* mine, bool want, int*& common) {
  __shared__ int* s_c;
  if (threadIdx.x == 0) s_c = nullptr;
  __syncthreads();
  if (want) s_c = mine;   // any of the writers
  __syncthreads();
  common = s_c;
  return __syncthreads_and(!want || mine == common) != 0;
}

// One atomicAdd on ctr for the n entries of every thread of the block; the
// thread's first slot (its n slots are consecutive).  All threads call it.
VRT_DI uint32_t block_append1(int* ctr, int n) {
  __shared__ int s_cnt[8];
  __shared__ int s_base;
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int incl = n;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(full, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) s_cnt[w] = incl;
  __syncthreads();
  if (threadIdx.x == 0) {
    int tot = 0;
    const int nw = (int)(blockDim.x >> 5);   // blocks of up to 256 threads
    for (int k = 0; k < nw; k++) {
      const int v = s_cnt[k];
      s_cnt[k] = tot;
      tot += v;
    }
    s_base = tot ? atomicAdd(ctr, tot) : 0;
  }
  __syncthreads();
  const uint32_t slot = (uint32_t)(s_base + s_cnt[w] + incl - n);
  __syncthreads();   // s_cnt / s_base are rewritten by the block's next call
  return slot;
}

// Writes the nrec training samples of training path ti from sample slot
// `slot` on (slots at or past the buffer's capacity are dropped).
VRT_DI void cache_write_samples(const CacheDev& c, uint32_t ti, int nrec, int slot, F3 rfin) {
  for (int k = 0; k < nrec && slot < c.cand_cap; k++, slot++) {
    const float4* r = c.rec + ((size_t)ti * kCacheMaxRec + k) * 4;
    const float4 r0 = r[0], r1 = r[1], r2 = r[2], r3 = r[3];
    float* q = c.cand_q9 + (size_t)slot * 9;
    q[0] = r0.x; q[1] = r0.y; q[2] = r0.z;
    q[3] = r1.x; q[4] = r1.y; q[5] = r1.z;
    q[6] = r2.x; q[7] = r2.y; q[8] = r2.z;
    float* y = c.cand_y3 + (size_t)slot * 3;
    y[0] = cache_target(rfin.x, r0.w, r3.x, c.tclamp);
    y[1] = cache_target(rfin.y, r1.w, r3.y, c.tclamp);
    y[2] = cache_target(rfin.z, r2.w, r3.z, c.tclamp);
  }
}

// Training samples of finished training paths: for each recorded vertex k,
// the radiance the path gathered after vertex k's emission pickup per unit
// of the throughput that reached it, (R_final - R_k) / tp_k -- the reflected
// radiance estimate at x_k.  All threads of the block call it: one atomic per
// block when its samples go to one job's buffer; otherwise per warp, or per
// lane when a warp's lanes belong to different jobs.
VRT_DI void cache_emit_samples(const CacheDev& c, bool fin, uint32_t ti, F3 rfin) {
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int nrec = fin ? c.rec_n[ti] : 0;
  int* common = nullptr;
  int slot = 0;
  if (block_common_counter(c.cand_count, nrec > 0, common)) {
    if (!common) return;
    slot = (int)block_append1(common, nrec);
  } else {
    const unsigned any = __ballot_sync(full, nrec > 0);
    if (!any) return;
    const unsigned long long key = (unsigned long long)c.cand_count;
    const unsigned grp = __match_any_sync(full, nrec > 0 ? key : 0ull) & any;
    const bool one_job = nrec > 0 ? grp == any : true;
    if (__all_sync(full, one_job)) {
      int incl = nrec;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(full, incl, o);
        if (lane >= o) incl += v;
      }
      const int total = __shfl_sync(full, incl, 31);
      const int leader = __ffs(any) - 1;
      int base = 0;
      if (lane == leader) base = atomicAdd(c.cand_count, total);
      base = __shfl_sync(full, base, leader);
      slot = base + incl - nrec;
    } else if (nrec > 0) {
      slot = atomicAdd(c.cand_count, nrec);
    }
  }
  cache_write_samples(c, ti, nrec, slot, rfin);
}

// Appends a cache query of path g at its vertex 1.  All threads of the block
// call it; one atomic per block when its queries go to one job's buffer.
VRT_DI void cache_emit_query(const CacheDev& c, bool q, uint32_t g, F3 pos, F3 n, F3 alb) {
  const unsigned full = 0xffffffffu;
  int* common = nullptr;
  uint32_t slot = 0u;
  if (block_common_counter(c.qcount, q, common)) {
    if (!common) return;
    slot = block_append1(common, q ? 1 : 0);
  } else {
    const unsigned any = __ballot_sync(full, q);
    if (!any) return;
    const unsigned grp = __match_any_sync(full, q ? (unsigned long long)c.qcount : 0ull) & any;
    if (__all_sync(full, q ? grp == any : true)) slot = warp_append(c.qcount, q);
    else slot = q ? (uint32_t)atomicAdd(c.qcount, 1) : 0u;
  }
  if (q) {
    float* d = c.qbuf + (size_t)slot * 9;
    d[0] = pos.x; d[1] = pos.y; d[2] = pos.z;
    d[3] = n.x; d[4] = n.y; d[5] = n.z;
    d[6] = alb.x; d[7] = alb.y; d[8] = alb.z;
    c.qpix[slot] = g;
  }
}

// ---------------------------------------------------------------------------
// shading
// ---------------------------------------------------------------------------
VRT_DI void finalize(const JobOut& out, uint32_t lp, F3 radiance, uint32_t mat1bits, float fclamp) {
  const Mat mat1 = unpack_material(mat1bits);
  if (!(fclamp <= 0.0f)) radiance = min3(radiance, f3(fclamp, fclamp, fclamp));
  const F3 den = max3(mat1.albedo, f3(1e-3f, 1e-3f, 1e-3f));
  const float4 rad = make_float4(radiance.x / den.x, radiance.y / den.y, radiance.z / den.z, 1.0f);
  out.rad16[lp] = pack_h4(rad.x, rad.y, rad.z, rad.w);
  if (out.rad32) out.rad32[lp] = rad;
}

// Vertex k of a path (pathtrace.wgsl:297-320 loop body up to the trace call),
// path state at index g.  Returns whether the path stays active.
// kmax: the path's last vertex (the uniforms' bounce count for plain paths).
// rec (may be null): training record of this vertex, written after the
// emission pickup.
VRT_DI bool shade_vertex(const Uni& u, const WfDev& b, uint32_t g, uint32_t k, F3 pos, F3 n, Mat mat,
                         F3& radiance, F3& tp, uint32_t& rng, uint32_t mat1bits, bool& want_shadow,
                         bool& want_bounce, uint32_t kmax, float4* rec) {
  if (mat.emissive > 0.0f) radiance = radiance + (tp * mat.albedo) * (mat.emissive * kEmissiveScale);
  if (rec) {
    rec[0] = make_float4(pos.x, pos.y, pos.z, radiance.x);
    rec[1] = make_float4(n.x, n.y, n.z, radiance.y);
    rec[2] = make_float4(mat.albedo.x, mat.albedo.y, mat.albedo.z, radiance.z);
    rec[3] = make_float4(tp.x, tp.y, tp.z, 0.0f);
  }
  const F3 surf = pos + n * 1e-3f;
  const F3 l = sample_sun_dir(u, rng);
  const float ndl = dot3(n, l);
  uint32_t flags = 0u;
  F3 sunc = f3(0.0f, 0.0f, 0.0f);
  want_shadow = ndl > 0.0f && l.y > 0.0f;
  if (want_shadow) {
    const F3 sunRad = f3(u.sunRadiance[0], u.sunRadiance[1], u.sunRadiance[2]);
    sunc = (((tp * mat.albedo) * kInvPi) * ndl) * sunRad;
    flags |= kFlagShadow;
    b.R2[g] = make_float4(l.x, l.y, l.z, 1e4f);
  }
  want_bounce = false;
  if (k == kmax) {
    flags |= kFlagTerminal;
  } else {
    const F3 rd = cosine_hemisphere(n, rng);
    tp = tp * mat.albedo;
    bool alive = true;
    if (k >= 2u) {
      const float pr = clamp_(fmax_(tp.x, fmax_(tp.y, tp.z)), 0.05f, 0.95f);
      if (rand_(rng) > pr) alive = false;
      else tp = f3(tp.x / pr, tp.y / pr, tp.z / pr);
    }
    if (alive) {
      want_bounce = true;
      b.R1[g] = make_float4(rd.x, rd.y, rd.z, 0.0f);
    } else {
      flags |= kFlagTerminal;
    }
  }
  b.R0[g] = make_float4(surf.x, surf.y, surf.z, 0.0f);
  b.S0[g] = make_float4(radiance.x, radiance.y, radiance.z, __uint_as_float(rng));
  b.S1[g] = make_float4(tp.x, tp.y, tp.z, __uint_as_float(mat1bits));
  b.S2[g] = make_float4(sunc.x, sunc.y, sunc.z, __uint_as_float(flags));
  return want_shadow || want_bounce;
}

// Block-aggregated appends: each thread of a block of up to 256 adds nf entries to
// the list counted by c_front, nb to the list counted by c_back and, if act,
// one to the list counted by c_act; one atomicAdd per counter per block, since
// every block of the grid appends to the same counters.  Returns the thread's
// first slot in each (its nf / nb slots are consecutive).  All threads of the
// block call it (block-uniform control flow).  Entries of a block are in
// thread order; a path's results do not depend on the order of the queues.
VRT_DI void block_append(int* c_front, int* c_back, int* c_act, int nf, int nb, bool act, uint32_t& fslot,
                         uint32_t& bslot, uint32_t& aslot, int* c_act2 = nullptr, bool act2 = false,
                         uint32_t* a2slot = nullptr) {
  __shared__ int s_cnt[4][8];
  __shared__ int s_base[4];
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int incf = nf, incb = nb;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int vf = __shfl_up_sync(full, incf, o);
    const int vb = __shfl_up_sync(full, incb, o);
    if (lane >= o) { incf += vf; incb += vb; }
  }
  const unsigned ma = __ballot_sync(full, act);
  const unsigned m2 = c_act2 ? __ballot_sync(full, act2) : 0u;
  if (lane == 31) { s_cnt[0][w] = incf; s_cnt[1][w] = incb; }
  if (lane == 0) { s_cnt[2][w] = __popc(ma); s_cnt[3][w] = __popc(m2); }
  __syncthreads();
  if (threadIdx.x < (c_act2 ? 4 : 3)) {   // thread 0: front, 1: back, 2: list, 3: the list's back part
    int tot = 0;
    const int nw = (int)(blockDim.x >> 5);   // blocks of up to 256 threads
#pragma unroll
    for (int k = 0; k < 8; k++) {
      if (k >= nw) break;
      const int v = s_cnt[threadIdx.x][k];
      s_cnt[threadIdx.x][k] = tot;
      tot += v;
    }
    int* c = threadIdx.x == 0 ? c_front : (threadIdx.x == 1 ? c_back : (threadIdx.x == 2 ? c_act : c_act2));
    s_base[threadIdx.x] = tot ? atomicAdd(c, tot) : 0;
  }
  __syncthreads();
  fslot = (uint32_t)(s_base[0] + s_cnt[0][w] + incf - nf);
  bslot = (uint32_t)(s_base[1] + s_cnt[1][w] + incb - nb);
  aslot = (uint32_t)(s_base[2] + s_cnt[2][w]) + (uint32_t)__popc(ma & ((1u << lane) - 1u));
  if (c_act2) *a2slot = (uint32_t)(s_base[3] + s_cnt[3][w]) + (uint32_t)__popc(m2 & ((1u << lane) - 1u));
  __syncthreads();   // s_cnt / s_base are rewritten by the block's next call
}

// Appends the new rays (shadow ray of path g, its bounce ray) and the active
// path of wave `next`.  Block-uniform, see block_append.
VRT_DI void emit_block(const WfDev& b, int next, uint32_t g, bool shadow, bool bounce, bool keep) {
  uint32_t fs, bs, as;
  int* c = b.ctr + 4 * next;
  block_append(c, c + 3, c + 2, (int)shadow, (int)bounce, keep, fs, bs, as);
  uint32_t* q = queue_of(b, next);
  if (shadow) q[fs] = g | kShadowBit;
  if (bounce) q[b.qcap - 1u - bs] = g;
  if (keep) active_of(b, next)[as] = g;
}

// emit_block() with a second shadow ray of the path, traced as path g + P, and
// the active list in two parts: paths with `back` set go to its back.
VRT_DI void emit2_block(const WfDev& b, int next, uint32_t g, uint32_t P, bool shadow, bool shadow2, bool bounce,
                        bool keep, bool back) {
  uint32_t fs, bs, as, as2;
  int* c = b.ctr + 4 * next;
  block_append(c, c + 3, c + 2, (int)shadow2 + (int)shadow, (int)bounce, keep && !back, fs, bs, as, b.act2 + next,
               keep && back, &as2);
  uint32_t* q = queue_of(b, next);
  if (shadow2) q[fs++] = (g + P) | kShadowBit;
  if (shadow) q[fs] = g | kShadowBit;
  if (bounce) q[b.qcap - 1u - bs] = g;
  if (keep) active_of(b, next)[back ? b.acap - 1u - as2 : as] = g;
}

// ---------------------------------------------------------------------------
// kernels (templated on the job policy)
// ---------------------------------------------------------------------------
// generate: RNG stream, jitter, camera ray (pathtrace.wgsl:249-263)
template <class J>
__global__ void __launch_bounds__(256) k_wf_generate(J jobs, uint32_t P, WfDev b) {
  frame_begin();
  const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = jobs.job_of_warp(g);
  if (g >= P) return;
  const Uni& u = jobs.uni(j);
  const int W = jobs.width(j), H = jobs.height(j);
  const uint32_t lp = g - jobs.first(j);
  const uint32_t gx = lp % (uint32_t)W, gy = lp / (uint32_t)W;
  uint32_t rng = init_rng(gx, gy, u.params0[0]);
  const float jx = rand_(rng) - 0.5f;
  const float jy = rand_(rng) - 0.5f;
  const float uvx = (((float)gx + 0.5f) + jx) / (float)W;
  const float uvy = (((float)gy + 0.5f) + jy) / (float)H;
  const F3 rd = camera_ray(u, uvx, uvy);
  // the path state of wave 0 is this one word: no radiance yet, and the RNG state in the direction's free lane
  b.R1[g] = make_float4(rd.x, rd.y, rd.z, __uint_as_float(rng));
}

// The q-th pixel of a W x H image in tiles of kTileX x kTileY (row by row in
// the tile and over the tiles; what is left at the right and at the bottom keeps
// the same order in narrower and lower tiles).  A warp's primary rays so start
// through a compact part of the image and walk together: the primary wave of the
// 1080p frame 192 -> 177 us against rows of 32.
constexpr uint32_t kTileX = 8, kTileY = 4;
VRT_DI uint32_t tile_order(uint32_t q, uint32_t W, uint32_t H) {
  const uint32_t y0 = q / (kTileY * W) * kTileY, r = q - y0 * W;   // strip of rows, pixel in it
  const uint32_t h = min(kTileY, H - y0);
  const uint32_t x0 = r / (kTileX * h) * kTileX, t = r - x0 * h;   // tile of the strip, pixel in it
  const uint32_t w = min(kTileX, W - x0);
  return (y0 + t / w) * W + x0 + t % w;
}

constexpr int kTraceThreads = 128;
// Persistent queue tracer.  A pass of the warp bookkeeping (idle-lane ballot,
// refill, drain check) covers kPhases rounds of up to kRun DDA steps and the
// transitions due after them (dda_walk.cuh).  Lanes whose walk ended keep it
// until the next refill, which stores all their hits together.  kVarMaxT:
// shadow rays carry their own maxT in R2.w (otherwise every ray ends at 1e4 m,
// the plain path's bound).  kWide: scenes of more than 128^3 bricks.
//
// Bound by instruction issue: on the 1080p / 256^3 frame (2 bounces, 6.4 M
// rays, 32 cells each) the wave of vertex 0's shadow and bounce rays issues
// 297 M warp instructions at 78% of the issue slots, 41% of them on the ALU
// pipe; before the walk kept its transitions out of the step it was 444 M at
// 86%.  The four waves' trace: 1.319 -> 0.949 ms (deep paths, 6 bounces:
// 1.684 -> 1.210; the ReSTIR initial pass 1.918 -> 1.375).
template <class J, bool kWide, int kPhases, int kMinB, int kRun, bool kVarMaxT>
__global__ void __launch_bounds__(kTraceThreads, kMinB) k_wf_trace(J jobs, WfDev b, int wave, int implicit_n,
                                                              int refill_min, unsigned long long* stats) {
  frame_begin();
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  // The bounce rays (the queue's back) first: their walks are the longer ones, and a wave ends with its
  // longest walk (shadow rays first: 0.959 against 0.931 ms of trace per 1080p frame).
  const int nb = implicit_n > 0 ? 0 : b.ctr[4 * wave + 3];
  const int n = implicit_n > 0 ? implicit_n : nb + b.ctr[4 * wave];
  int* head = b.ctr + 4 * wave + 1;
  const uint32_t* queue = queue_of(b, wave);
  DCount c{0u, 0u, 0u, 0u};
  Walk<kWide> d;
  DScene S = jobs.scene(0);
  F3 rd = f3(0.0f, 0.0f, 0.0f);
  uint32_t entry = 0u;
  int jc = 0;                     // the lane's last job and its pixel range [jlo, jhi) (empty: none yet)
  uint32_t jlo = 0u, jhi = 0u;
  uint32_t passes = 0u;   // passes of the step loop with a lane walking (warp-uniform)
  // Lanes of a warp on different walks take turns, so the rays of a small wave are spread over all
  // resident warps: each warp uses as many lanes as it has rays to take.
  const int nwarps = (int)(gridDim.x * (kTraceThreads / 32));
  const int lanes = min(32, max(1, (n + nwarps - 1) / nwarps));
  const int refill = min(refill_min, lanes);
  const unsigned in_use = lanes == 32 ? full : (1u << lanes) - 1u;
  bool active = false, held = false, drained = false;   // held: the lane's ray is not stored yet
  while (true) {
    const unsigned idle = __ballot_sync(full, !active) & in_use;
    const int nidle = __popc(idle);
    if (nidle >= refill || drained) {
      // the lanes whose walk ended store their hits together
      if (held && !active) {
        d.finish(S, c);
        const uint32_t g = entry & ~kShadowBit;
        uint32_t* h = reinterpret_cast<uint32_t*>(b.hit + g);
        if (entry & kShadowBit) {
          h[3] = d.tHit >= 0.0f ? 1u : 0u;
        } else {
          *reinterpret_cast<uint2*>(h) = make_uint2(__float_as_uint(d.tHit), d.mat);
          h[2] = (uint32_t)d.hit_axis(S);
        }
        held = false;
      }
    }
    if (!drained && nidle >= refill) {
      int base = 0;
      if (lane == 0) base = atomicAdd(head, nidle);
      base = __shfl_sync(full, base, 0);
      if (base + nidle >= n) drained = true;
      if ((idle >> lane) & 1u) {
        const int slot = base + __popc(idle & ((1u << lane) - 1u));
        if (slot < n) {
          entry = implicit_n > 0 ? (uint32_t)slot
                                 : (slot < nb ? queue[b.qcap - 1u - (uint32_t)slot] : queue[slot - nb]);
          uint32_t g = entry & ~kShadowBit;
          const int j = jobs.job_of_cached(g, jc, jlo, jhi);   // consecutive rays mostly share a job
          S = jobs.scene(j);
          if (implicit_n > 0) {
            const uint32_t p0 = jobs.first(j);
            g = entry = p0 + tile_order(g - p0, (uint32_t)jobs.width(j), (uint32_t)jobs.height(j));
          }
          // primary rays start at the camera: its position comes from the job's
          // uniforms (k_wf_generate writes no R0, so no wave-0 shading kernel
          // may read R0 either); later waves read the origin their shading stored
          F3 ro;
          if (implicit_n > 0) {
            const Uni& uj = jobs.uni(j);
            ro = f3(uj.camPos[0], uj.camPos[1], uj.camPos[2]);
          } else {
            ro = xyz(b.R0[g]);
          }
          if (kVarMaxT) {
            float maxT = 1e4f;   // bounce rays; shadow rays carry theirs in R2.w
            if (entry & kShadowBit) {
              const float4 r2 = b.R2[g];
              rd = xyz(r2);
              maxT = r2.w;
            } else {
              rd = xyz(b.R1[g]);
            }
            d.init(S, ro, rd, maxT);
          } else {
            rd = (entry & kShadowBit) ? xyz(b.R2[g]) : xyz(b.R1[g]);
            d.init(S, ro, rd, 1e4f);
          }
          c.rays++;
          active = true;
          held = true;
        }
      }
    }
    if (!__any_sync(full, active)) {
      if (drained) break;
      continue;
    }
    passes++;
    if (active) {
#pragma unroll 1
      for (int k = 0; k < kPhases; k++) {
        d.template walk_run<kRun>(S);
        if (!d.walking() && !d.done()) d.transition(S, rd, c);
      }
      active = !d.done();
    }
  }
  if (stats) {
    block_flush_stats(stats, c, 0u);   // kStatRays..kStatVReads
    block_flush_one(stats + kStatTraceSlots, lane == 0 ? passes * (uint32_t)(32 * kPhases * kRun) : 0u);
  }
}

constexpr int kShadeThreads = 128;

// shade(0): primary hits over all pixels.  The shading kernels are bound by
// instruction issue (77% of the issue slots on a 1080p frame) and run 1280
// threads per SM (48 registers; 6 x 256 threads spill and gain nothing), in
// blocks of 128: the barriers of the block-wide appends then hold up four warps
// instead of eight (cache frames 1.040 -> 1.024 ms of path tracing against
// blocks of 256; plain frames equal).
template <class J>
__global__ void __launch_bounds__(kShadeThreads, 1280 / kShadeThreads) k_wf_shade_primary(J jobs, uint32_t P, WfDev b, unsigned long long* stats) {
  frame_begin();
  const bool any_cache = jobs.any_cache();
  const CacheDev* ccp = nullptr;
  const uint32_t stride = gridDim.x * blockDim.x;
  if (stats && blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(stats + kStatPixels, (unsigned long long)P);
  for (uint32_t base = blockIdx.x * blockDim.x; base < P; base += stride) {
    const uint32_t g = base + threadIdx.x;
    bool shadow = false, bounce = false, keep = false;
    bool fin_train = false;
    uint32_t ti = 0u;
    F3 rfin = f3(0.0f, 0.0f, 0.0f);
    const int j = jobs.job_of_warp(g);
    if (g < P) {
      const Uni& u = jobs.uni(j);
      const JobOut out = jobs.outs(j);
      const uint32_t lp = g - jobs.first(j);
      const uint4 h = b.hit[g];
      const float4 r1 = b.R1[g];
      const F3 rd = xyz(r1);
      const float t = __uint_as_float(h.x);
      if (t < 0.0f) {
        const F3 sky = sky_color(u, rd, true);
        out.rad16[lp] = pack_h4(sky.x, sky.y, sky.z, 1.0f);
        if (out.rad32) out.rad32[lp] = make_float4(sky.x, sky.y, sky.z, 1.0f);
        out.alb8[lp] = 0xffffffffu;
        out.gbuf[lp] = make_float4(-rd.x, -rd.y, -rd.z, -1.0f);
      } else {
        const Mat mat1 = unpack_material(h.y);
        const F3 ro = f3(u.camPos[0], u.camPos[1], u.camPos[2]);
        const F3 x1 = ro + rd * t;
        const F3 n1 = hit_normal((int)h.z, rd);
        out.alb8[lp] = sqrt_albedo8(h.y);
        out.gbuf[lp] = make_float4(n1.x, n1.y, n1.z, t);
        uint32_t rng = __float_as_uint(r1.w);
        F3 radiance = f3(0.0f, 0.0f, 0.0f), tp = f3(1.0f, 1.0f, 1.0f);
        const int W = jobs.width(j);
        const CacheDev& cc = jobs.cache(j);
        ccp = &cc;
        const int role = cache_role(cc, lp, W);
        const uint32_t kmax = role == kRolePlain ? u.params0[1] : (role == kRoleTrain ? cc.train_bounces : 1u);
        keep = shade_vertex(u, b, g, 0u, x1, n1, mat1, radiance, tp, rng, h.y, shadow, bounce, kmax,
                            rec_slot(cc, role, lp, W, 0u));
        if (!keep) {
          finalize(out, lp, radiance, h.y, jobs.clamp(j));
          if (role == kRoleTrain) { fin_train = true; ti = train_index(cc, lp, W); rfin = radiance; }
        }
      }
    }
    emit_block(b, 1, g, shadow, bounce, keep);
    if (any_cache) cache_emit_samples(fin_train ? *ccp : jobs.cache(0), fin_train, ti, rfin);
  }
}

// shade(k), k >= 1: resolve vertex k-1's shadow ray, then the bounce hit.
template <class J>
__global__ void __launch_bounds__(kShadeThreads, 1280 / kShadeThreads) k_wf_shade(J jobs, WfDev b, int wave) {
  frame_begin();
  const bool any_cache = jobs.any_cache();
  const int n = b.ctr[4 * wave + 2];
  const uint32_t* list = active_of(b, wave);
  const int stride = gridDim.x * blockDim.x;
  for (int base = blockIdx.x * blockDim.x; base < n; base += stride) {
    const int i = base + threadIdx.x;
    bool shadow = false, bounce = false, keep = false;
    bool fin_train = false, query = false;
    uint32_t ti = 0u;
    F3 rfin = f3(0.0f, 0.0f, 0.0f), qpos = rfin, qn = rfin, qalb = rfin;
    uint32_t g = 0u;
    int jc = 0;
    if (i < n) {
      g = list[i];
      const int j = jobs.job_of(g);
      jc = j;
      const uint32_t lp = g - jobs.first(j);
      const int W = jobs.width(j);
      const CacheDev& cc = jobs.cache(j);
      const int role = cache_role(cc, lp, W);
      const float4 s0 = b.S0[g];
      const float4 s1 = b.S1[g];
      const float4 s2 = b.S2[g];
      const uint4 h = b.hit[g];
      // loaded with the state above rather than after the terminal check, so a
      // path's reads are one round trip instead of two
      const float4 r1 = b.R1[g];
      const float4 r0 = b.R0[g];
      F3 radiance = xyz(s0);
      F3 tp = xyz(s1);
      uint32_t rng = __float_as_uint(s0.w);
      const uint32_t mat1bits = __float_as_uint(s1.w);
      const uint32_t flags = __float_as_uint(s2.w);
      if ((flags & kFlagShadow) && h.w == 0u) radiance = radiance + xyz(s2);
      bool done = (flags & kFlagTerminal) != 0u;
      if (!done) {
        const Uni& u = jobs.uni(j);
        const F3 rd = xyz(r1);
        const F3 surf = xyz(r0);
        const float t = __uint_as_float(h.x);
        if (t < 0.0f) {
          radiance = radiance + tp * sky_color(u, rd, false);
          done = true;
        } else {
          const F3 pos = surf + rd * t;
          const F3 nrm = hit_normal((int)h.z, rd);
          const Mat mat = unpack_material(h.y);
          if (role == kRoleQuery) {
            // path ends at vertex 1: emission here, reflected radiance from the cache
            if (mat.emissive > 0.0f) radiance = radiance + (tp * mat.albedo) * (mat.emissive * kEmissiveScale);
            b.S0[g] = make_float4(radiance.x, radiance.y, radiance.z, __uint_as_float(rng));
            query = true;
            qpos = pos; qn = nrm; qalb = mat.albedo;
          } else {
            const uint32_t kmax = role == kRolePlain ? u.params0[1] : cc.train_bounces;
            keep = shade_vertex(u, b, g, (uint32_t)wave, pos, nrm, mat, radiance, tp, rng, mat1bits, shadow, bounce,
                                kmax, rec_slot(cc, role, lp, W, (uint32_t)wave));
            done = !keep;
          }
        }
      }
      if (done) {
        finalize(jobs.outs(j), lp, radiance, mat1bits, jobs.clamp(j));
        if (role == kRoleTrain) { fin_train = true; ti = train_index(cc, lp, W); rfin = radiance; }
      }
    }
    emit_block(b, wave + 1, g, shadow, bounce, keep);
    if (any_cache) {
      const CacheDev& cc = jobs.cache(jc);
      cache_emit_query(cc, query, g, qpos, qn, qalb);
      cache_emit_samples(cc, fin_train, ti, rfin);
    }
  }
}

// The tail of a frame whose remaining paths are few (small frames, late waves,
// the radiance cache's training paths after every other path ended at its
// first bounce): each path of wave `wave`'s active list is finished here by one
// thread, or by two where all of them fit the grid so, tracing its pending
// shadow and bounce rays with the same resumable DDA the queue tracer runs
// (dda_walk.cuh: same walk, hits and counters) and shading each vertex as
// k_wf_shade does, until the path ends.  The per-wave form would launch a
// trace and a shade kernel for every remaining bounce, each waiting for the
// slowest of ~10^5 latency-bound walks; here each path runs its own
// sequence.  Same per-path arithmetic and RNG draws, so the same image.
// Few paths are spread over all warps, a few lanes each: lanes on different
// walks take turns.
// Bound by the latency of a path's walks, one after another.  Its shadow and
// bounce ray of a vertex are independent: with two lanes per path they walk
// together, and the odd lane leaves the path's state to the even one.  That pays
// while all paths fit the grid at once (kTailPairLimit per warp, 47 K); with more,
// a lane per path finishes sooner.  Path trace in ms, one lane / two where they fit
// / two always: 320x180 .122 / .111 / .117; 320x180 with 6 bounces .204 / .171 /
// .171; 400x225 .184 / .180 / .195; 1283x721 with 6 bounces .687 / .665 / .663;
// a 1080p cache frame (130 K paths) .980 / .975 / .997.
// (A per-lane state machine -- lanes stepping their walks together, each
// shading when its own ray ends and then taking the next path -- ran 447
// against 305 us per 1080p cache frame: some lane shades in nearly every pass,
// so the warp runs the shading code far more often than once per bounce.)
constexpr int kTailPairLimit = 16;
constexpr int kTailRun = 5;   // DDA steps between transitions
template <class J, bool kWide>
__global__ void __launch_bounds__(128, 5) k_wf_tail(J jobs, WfDev b, int wave, unsigned long long* stats) {
  frame_begin();
  const bool any_cache = jobs.any_cache();
  const int n = b.ctr[4 * wave + 2];
  const uint32_t* list = active_of(b, wave);
  // few paths are spread over all warps (as in k_wf_trace); every block runs every round
  const unsigned full = 0xffffffffu;
  const int nwarps = (int)(gridDim.x * (blockDim.x >> 5)), warp = (int)(blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5));
  const bool pair = n <= kTailPairLimit * nwarps;
  const int lane = threadIdx.x & 31, slot = pair ? lane >> 1 : lane;
  const int per = min(pair ? 16 : 32, max(1, (n + nwarps - 1) / nwarps));
  const bool owner = !pair || (lane & 1) == 0;    // of the path's state; the other lane of a pair walks its shadow rays
  const int ray0 = pair && owner ? 1 : 0, ray1 = pair && !owner ? 1 : 2;   // this lane's rays: 0 shadow, 1 bounce
  DCount c{0u, 0u, 0u, 0u};
  uint32_t passes = 0u;   // rounds of steps of this warp
  for (int base = 0; base < n; base += nwarps * per) {
    const int i = slot < per ? base + warp * per + slot : n;
    bool fin_train = false;
    uint32_t ti = 0u, g = 0u, lp = 0u;
    F3 rfin = f3(0.0f, 0.0f, 0.0f);
    int j = 0, role = kRolePlain;
    bool live = i < n;
    if (live) {
      g = list[i];
      j = jobs.job_of(g);
      lp = g - jobs.first(j);
      role = cache_role(jobs.cache(j), lp, jobs.width(j));
    }
    const DScene S = jobs.scene(j);
    for (int w = wave; __any_sync(full, live); w++) {
      uint32_t flags = 0u;
      F3 surf = f3(0.0f, 0.0f, 0.0f), rd = surf;
      bool lit = false;                            // the shadow ray met nothing
      Walk<kWide> d;
      uint32_t rounds = 0u;                        // of steps, of this lane
      if (live) {
        flags = __float_as_uint(b.S2[g].w);
        surf = xyz(b.R0[g]);
#pragma unroll 1
        for (int ray = ray0; ray < ray1; ray++) {
          if (!(ray == 0 ? (flags & kFlagShadow) != 0u : (flags & kFlagTerminal) == 0u)) continue;
          const float4 r = ray == 0 ? b.R2[g] : b.R1[g];
          rd = xyz(r);
          d.init(S, surf, rd, ray == 0 ? r.w : 1e4f);
          c.rays++;
          while (!d.done()) {
            rounds++;
            d.template walk_run<kTailRun>(S);
            if (!d.walking()) d.transition(S, rd, c);
          }
          d.finish(S, c);
          if (ray == 0) lit = !(d.tHit >= 0.0f);
        }
      }
      passes += __reduce_max_sync(full, rounds);   // lanes step together, so the longest walk counts
      if (pair) lit = __shfl_xor_sync(full, (int)lit, 1) != 0;   // the owner's answer from its pair
      if (live && owner) {
        const float4 s0 = b.S0[g];
        const float4 s1 = b.S1[g];
        F3 radiance = xyz(s0);
        F3 tp = xyz(s1);
        uint32_t rng = __float_as_uint(s0.w);
        const uint32_t mat1bits = __float_as_uint(s1.w);
        const int W = jobs.width(j);
        const CacheDev& cc = jobs.cache(j);
        const Uni& u = jobs.uni(j);
        if (lit) radiance = radiance + xyz(b.S2[g]);   // the previous vertex's sun
        bool done = (flags & kFlagTerminal) != 0u;
        if (!done) {
          if (d.tHit < 0.0f) {
            radiance = radiance + tp * sky_color(u, rd, false);
            done = true;
          } else {
            const F3 pos = surf + rd * d.tHit;
            const F3 nrm = hit_normal(d.hit_axis(S), rd);
            const Mat mat = unpack_material(d.mat);
            const uint32_t kmax = role == kRolePlain ? u.params0[1] : cc.train_bounces;
            bool shadow = false, bounce = false;
            done = !shade_vertex(u, b, g, (uint32_t)w, pos, nrm, mat, radiance, tp, rng, mat1bits, shadow, bounce,
                                 kmax, rec_slot(cc, role, lp, W, (uint32_t)w));
          }
        }
        if (done) {
          finalize(jobs.outs(j), lp, radiance, mat1bits, jobs.clamp(j));
          if (role == kRoleTrain) { fin_train = true; ti = train_index(cc, lp, W); rfin = radiance; }
          live = false;
        }
      }
      // the pair takes the owner's path state, written above
      if (pair) live = __shfl_sync(full, (int)live, lane & 30) != 0;
      __syncwarp();
    }
    if (any_cache) cache_emit_samples(jobs.cache(j), fin_train, ti, rfin);
  }
  if (stats) {
    block_flush_stats(stats, c, 0u);   // kStatRays..kStatVReads
    block_flush_one(stats + kStatTraceSlots, lane == 0 ? passes * (uint32_t)(32 * kTailRun) : 0u);
  }
}

// Zeroes the per-frame query and sample counters of every cache job.
template <class J>
__global__ void k_cache_reset(J jobs, int njobs) {
  frame_begin();
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= njobs) return;
  const CacheDev& c = jobs.cache(j);
  if (c.on) {
    *c.qcount = 0;
    *c.cand_count = 0;
  }
}

// Cache-terminated paths of up to kMaxMlpTasks jobs (blockIdx.y = entry):
// radiance += throughput at vertex 1 * predicted reflected radiance there,
// then the usual clamp / demodulation / store.
struct ResolveEntry {
  const int* qcount;
  const uint32_t* qpix;
  const int* cand_count;
  const float* pred;
  int cand_cap;
  int pad;
};
struct ResolveSet {
  int n;
  int pad[3];
  ResolveEntry e[kMaxMlpTasks];
};

template <class J>
__global__ void __launch_bounds__(256) k_cache_resolve(J jobs, WfDev b, const __grid_constant__ ResolveSet rs,
                                                       unsigned long long* stats) {
  frame_begin();
  const ResolveEntry& r = rs.e[blockIdx.y];
  const int n = *r.qcount;
  if (stats && blockIdx.x == 0 && threadIdx.x == 0) {
    atomicAdd(stats + kStatCacheQueries, (unsigned long long)n);
    atomicAdd(stats + kStatCacheSamples, (unsigned long long)min(*r.cand_count, r.cand_cap));
  }
  const int stride = gridDim.x * blockDim.x;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    const uint32_t g = r.qpix[i];
    const int j = jobs.job_of(g);
    const float4 s0 = b.S0[g];
    const float4 s1 = b.S1[g];
    const float* p = r.pred + 3 * (size_t)i;
    const F3 L = f3(fmax_(p[0], 0.0f), fmax_(p[1], 0.0f), fmax_(p[2], 0.0f));
    const F3 radiance = xyz(s0) + xyz(s1) * L;
    finalize(jobs.outs(j), g - jobs.first(j), radiance, __float_as_uint(s1.w), jobs.clamp(j));
  }
}

// ---------------------------------------------------------------------------
// host: one frame's wave sequence for a job set of P pixels
// ---------------------------------------------------------------------------
inline WfDev wf_view(const WavefrontBufs& w) {
  WfDev d;
  d.R0 = (float4*)w.R0; d.R1 = (float4*)w.R1; d.R2 = (float4*)w.R2;
  d.S0 = (float4*)w.S0; d.S1 = (float4*)w.S1; d.S2 = (float4*)w.S2;
  d.hit = (uint4*)w.hit;
  d.q0 = w.q[0]; d.q1 = w.q[1]; d.a0 = w.act[0]; d.a1 = w.act[1];
  d.ctr = w.ctr;
  d.act2 = w.ctr + 4 * (size_t)w.max_waves;
  d.qcap = (uint32_t)w.qcap;
  d.acap = (uint32_t)w.acap;
  return d;
}

// ---------------------------------------------------------------------------
// host: post-wave cache work of one job -- inference over its queries, the
// resolve of its cache-terminated paths, then its training steps.  Every
// per-frame quantity (counts, Adam step, sample draws) lives on the device,
// so the sequence can be captured in a CUDA graph and replayed.
// ---------------------------------------------------------------------------
// The MLP task of a cache job: inference (k < 0) or training step k.
inline MlpTask mlp_task_of(const CacheLaunch& cl, int k) {
  MlpTask t;
  std::memset(&t, 0, sizeof t);
  t.wb = cl.wb;
  t.extent = cl.extent;
  t.err = cl.err;
  if (k < 0) {
    t.q9 = cl.cd.qbuf;
    t.out3 = cl.pred;
    t.n_dev = cl.cd.qcount;
    t.n_max = cl.P;
  } else {
    t.q9 = cl.cd.cand_q9;
    t.y3 = cl.cd.cand_y3;
    t.n_dev = cl.cd.cand_count;
    t.n_max = cl.train_batch;
    t.pop_cap = cl.cd.cand_cap;
    t.seed = 0x9e3779b9u * (uint32_t)(k + 1);
    t.step = cl.step;
    t.partial = cl.partial;
    t.loss = cl.loss;
    t.grad = cl.grad;
    t.wm = cl.wm;
    t.m = cl.m;
    t.v = cl.v;
    t.wbw = cl.wb;
    t.lr = cl.lr;
  }
  return t;
}

// Post-wave cache work of `n` jobs, up to kMaxMlpTasks per launch: one
// inference launch over all their queries, one resolve launch, then per
// training step one gradient (+ reduction) and one Adam launch serving every
// job that still has steps to take.
template <class J>
cudaError_t launch_cache_post(const J& jobs, const WfDev& b, const CacheLaunch* cls, int n,
                              unsigned long long* stats, cudaStream_t st, uint32_t* launches) {
  uint32_t nl = 0;
  for (int c0 = 0; c0 < n; c0 += kMaxMlpTasks) {
    const int cn = std::min(kMaxMlpTasks, n - c0);
    MlpTaskSet ts;
    std::memset(&ts, 0, sizeof ts);
    ResolveSet rs;
    std::memset(&rs, 0, sizeof rs);
    int maxP = 1, steps = 0;
    for (int k = 0; k < cn; k++) {
      const CacheLaunch& cl = cls[c0 + k];
      ts.t[ts.n++] = mlp_task_of(cl, -1);
      rs.e[rs.n++] = ResolveEntry{cl.cd.qcount, cl.cd.qpix, cl.cd.cand_count, cl.pred, cl.cd.cand_cap, 0};
      maxP = std::max(maxP, cl.P);
      steps = std::max(steps, cl.train_steps);
    }
    cudaError_t e = mlp_infer_tasks(ts, st);
    if (e != cudaSuccess) return e;
    const int bx = std::max(1, std::min((maxP + 255) / 256, wf_sm_count() * 8 / cn));
    launch_after(k_cache_resolve<J>, dim3(bx, rs.n), 256, 0, st, jobs, b, rs, stats);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    nl += 2;
    for (int k = 0; k < steps; k++) {
      MlpTaskSet tr;
      std::memset(&tr, 0, sizeof tr);
      for (int q = 0; q < cn; q++)
        if (k < cls[c0 + q].train_steps) tr.t[tr.n++] = mlp_task_of(cls[c0 + q], k);
      if ((e = mlp_gradient_tasks(tr, st)) != cudaSuccess) return e;
      if ((e = mlp_adam_tasks(tr, st)) != cudaSuccess) return e;
      nl += 3;   // gradient, reduction, Adam
    }
  }
  if (launches) *launches += nl;
  return cudaSuccess;
}

template <class J, bool kWide, int kPhases, int kMinB, int kRun, bool kVarMaxT>
cudaError_t wf_launch_trace(const J& jobs, int blocks_per_sm, int sms, const WfDev& b, int w, int implicit_n,
                            int refill, unsigned long long* stats, cudaStream_t st) {
  auto* fn = k_wf_trace<J, kWide, kPhases, kMinB, kRun, kVarMaxT>;
  int per = blocks_per_sm * (256 / kTraceThreads);   // the tuning counts blocks of 256 threads
  if (per <= 0) {
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fn, kTraceThreads, 0);
    if (e != cudaSuccess || per < 1) per = 1;
  }
  launch_after(fn, sms * per, kTraceThreads, 0, st, jobs, b, w, implicit_n, refill, stats);
  return cudaGetLastError();
}

// Tracer variants (the autotuner's trace_variant).  A transition runs for
// every lane that waits for one, in about as many instructions as four steps,
// and nearly every step of a warp makes some lane due for one: more steps per
// round share a transition's cost among more lanes, and leave more lanes
// waiting.  Trace time of the 1080p / 256^3 frame by steps per round (9 blocks
// of 128 threads and 56 registers per SM, refill at 12 idle lanes): 1 step
// 1.251 ms, 3 0.987, 4 0.955, 5 0.949, 6 0.952.  8 blocks (64 registers, no
// spills) 0.971 at 4 steps; 10 (48 registers, spilling) 1.05 at 3.  Refill at 8
// / 10 / 12 / 14 idle lanes: 0.959 / 0.950 / 0.949 / 0.953 (later, from another
// view: 1.004 / 0.994 / 0.994 / 0.995, 16: 1.002).  Fetching the next
// cell's word before the checks that may end a level's walk: 0.990 against
// 0.971 (it costs a register that spills).
template <class J, bool kVarMaxT = false>
cudaError_t wf_dispatch_trace(int variant, const J& jobs, int tb, int sms, const WfDev& b, int w, int impl,
                              int refill, unsigned long long* stats, cudaStream_t st) {
  if (jobs.wide())   // scenes of more than 128^3 bricks: the default shape only
    return wf_launch_trace<J, true, 3, 9, 5, kVarMaxT>(jobs, tb, sms, b, w, impl, refill, stats, st);
  if (kVarMaxT)      // the ReSTIR passes: the default shape only
    return wf_launch_trace<J, false, 3, 9, 5, kVarMaxT>(jobs, tb, sms, b, w, impl, refill, stats, st);
  switch (variant) {
    case 1: return wf_launch_trace<J, false, 4, 9, 4, false>(jobs, tb, sms, b, w, impl, refill, stats, st);
    case 2: return wf_launch_trace<J, false, 3, 8, 4, false>(jobs, tb, sms, b, w, impl, refill, stats, st);
    case 3: return wf_launch_trace<J, false, 4, 9, 3, false>(jobs, tb, sms, b, w, impl, refill, stats, st);
    case 4: return wf_launch_trace<J, false, 2, 9, 4, false>(jobs, tb, sms, b, w, impl, refill, stats, st);
    case 5: return wf_launch_trace<J, false, 8, 9, 1, false>(jobs, tb, sms, b, w, impl, refill, stats, st);
    case 6: return wf_launch_trace<J, false, 4, 10, 3, false>(jobs, tb, sms, b, w, impl, refill, stats, st);
    case 7: return wf_launch_trace<J, false, 3, 9, 6, false>(jobs, tb, sms, b, w, impl, refill, stats, st);
    case 8: return wf_launch_trace<J, false, 3, 8, 6, false>(jobs, tb, sms, b, w, impl, refill, stats, st);
    default: return wf_launch_trace<J, false, 3, 9, 5, false>(jobs, tb, sms, b, w, impl, refill, stats, st);
  }
}

// Launches generate + (trace, shade) x waves; shade(b, w, blocks) launches
// the shading kernel of wave w.
constexpr int kPrimaryRefill = 32;   // idle lanes that trigger a refill in the primary wave (at least)

template <class J, class ShadeFn, bool kVarMaxT = false>
cudaError_t wf_run_waves(const J& jobs, uint32_t P, int waves, const WavefrontBufs& wb,
                         const WavefrontTuning& tune, unsigned long long* stats, cudaStream_t st, uint32_t* launches,
                         cudaEvent_t* trace_ev, int max_timed_waves, int* timed_waves, ShadeFn shade,
                         int tail_from = 0) {
  if (waves + 1 > wb.max_waves) return cudaErrorInvalidValue;
  const WfDev b = wf_view(wb);
  cudaError_t e = cudaMemsetAsync(wb.ctr, 0, (size_t)wb.max_waves * 20, st);
  if (e != cudaSuccess) return e;
  const int sms = wf_sm_count();
  const int refill = tune.refill_min > 0 ? tune.refill_min : 12;
  // shading blocks (the tuning counts them as blocks of 256 threads), no more than the pixels need: the full
  // grid's idle blocks cost 2 us of a 320x180 frame's 175
  const int sblocks = std::min(sms * (tune.shade_blocks_per_sm > 0 ? tune.shade_blocks_per_sm : 32) * (256 / kShadeThreads),
                               (int)((P + kShadeThreads - 1) / kShadeThreads));
  uint32_t nl = 0;
  launch_after(k_wf_generate<J>, (P + 255) / 256, 256, 0, st, jobs, P, b);
  nl++;
  int timed = 0;
  for (int w = 0; w < waves; w++) {
    if (tail_from > 0 && w == tail_from) {   // the remaining paths, a thread or two each
      // a resident grid of 128-thread blocks (a block's round waits for its slowest path); 5 per SM (96
      // registers): 0.125 ms of path trace at 58 K pixels and 1.050 of a 1080p cache frame, against 0.133
      // and 1.060 at 6, 0.146 and 1.082 at 8
      const int tblocks = sms * 5;
      if (jobs.wide()) launch_after(k_wf_tail<J, true>, tblocks, 128, 0, st, jobs, b, w, stats);
      else launch_after(k_wf_tail<J, false>, tblocks, 128, 0, st, jobs, b, w, stats);
      if ((e = cudaGetLastError()) != cudaSuccess) return e;
      nl++;
      break;
    }
    const bool tm = trace_ev && w < max_timed_waves;
    if (tm && (e = cudaEventRecord(trace_ev[2 * w], st)) != cudaSuccess) return e;
    const int impl = w == 0 ? (int)P : 0;
    const int tb = tune.trace_blocks_per_sm;
    // the coherent primary rays refill later, in whole warps: the four waves of a 1080p frame trace in 1.008 /
    // 1.003 / 0.998 / 0.994 ms with the primary wave's refill at 12 / 16 / 24 / 32 idle lanes, the others' at 12
    const int rf = w == 0 ? std::max(refill, kPrimaryRefill) : refill;
    e = wf_dispatch_trace<J, kVarMaxT>(tune.trace_variant, jobs, tb, sms, b, w, impl, rf, stats, st);
    if (e != cudaSuccess) return e;
    if (tm && (e = cudaEventRecord(trace_ev[2 * w + 1], st)) != cudaSuccess) return e;
    if (tm) timed++;
    nl++;
    if ((e = shade(b, w, sblocks)) != cudaSuccess) return e;
    nl++;
  }
  if (launches) *launches += nl;
  if (timed_waves) *timed_waves = timed;
  return cudaGetLastError();
}

// The wave whose remaining paths finish in k_wf_tail when the tuning leaves
// it open (0: none).  A wave has a floor of 25-35 us of trace and 5-8 of
// shading -- its longest walk, whatever its size -- which k_wf_tail pays once for all the
// waves it replaces, at a lower rate per ray; so the line lies at a number of
// paths, later the more pixels there are.  Path-trace pass in ms by tail wave
// (pixels, bounces: none / 1 / 2 / 3 / 4 / 5):
//   58 K, 2: .180 / .111 / .133 / .160      58 K, 6: .388 / .171 / .214 / .258 / .289
//  130 K, 2: .286 / .284 / .249 / .264     130 K, 6: .429 / .243 / .280 / .295 / .322
//  230 K, 2: .324 / .335 / .326 / .301     230 K, 4: .348 / .317 / .271 / .274 / .306
//  518 K, 2: .442 / .592 / .497 / .436     518 K, 6: .652 / .745 / .666 / .594 / .535 / .569
//  925 K, 6: .788 / 1.06 / .862 / .718 / .665 / .707
//  2.1 M, 2: 1.148 / 1.96 / 1.56 / 1.175   2.1 M, 6: 1.453 / 2.57 / 2.16 / 1.69 / 1.424 / 1.380
// (The tail's grid holds 95 K paths at once; a few more cost it a second round.)
// Cache-assisted frames (every path but the training paths ends at wave 1)
// always take wave 2, and with the cache on no frame takes wave 1 (frame_tail).
inline int auto_tail(uint32_t P, int waves, bool any_cache, bool all_cache) {
  if (all_cache) return 2;
  const bool deep = waves > 4;   // 3 bounces or more
  int w;
  if (P <= 120000u) w = any_cache ? 2 : 1;
  else if (P <= 200000u) w = 2;
  else if (P <= 300000u) w = deep ? 2 : 3;
  else if (P <= 700000u) w = deep ? 4 : 3;
  else if (P <= 1500000u) w = 4;
  else w = 5;
  return w < waves ? w : 0;
}

// The tail wave of a frame: as tuned, else automatic.  A path that the cache ends turns into a query in
// wave 1's shading, which the tail does not do, so with any such path in the frame the tail begins at wave 2.
inline int frame_tail(const WavefrontTuning& tune, uint32_t P, int waves, bool any_cache, bool all_cache) {
  const int w = tune.tail_wave >= 0 ? tune.tail_wave : auto_tail(P, waves, any_cache, all_cache);
  return any_cache && w == 1 ? 2 : w;
}

// The plain path's wave sequence (with the radiance cache's counter reset
// when any job has the cache on).
template <class J>
cudaError_t wf_launch_frame(const J& jobs, uint32_t P, int waves, const WavefrontBufs& wb,
                            const WavefrontTuning& tune, unsigned long long* stats, cudaStream_t st,
                            uint32_t* launches, cudaEvent_t* trace_ev, int max_timed_waves, int* timed_waves,
                            int njobs = 1, int tail_from = 0) {
  if (waves + 1 > wb.max_waves) return cudaErrorInvalidValue;
  if (jobs.any_cache()) {
    launch_after(k_cache_reset<J>, (njobs + 127) / 128, 128, 0, st, jobs, njobs);
    if (launches) (*launches)++;
  }
  return wf_run_waves(jobs, P, waves, wb, tune, stats, st, launches, trace_ev, max_timed_waves, timed_waves,
                      [&](const WfDev& b, int w, int sblocks) {
                        if (w == 0) launch_after(k_wf_shade_primary<J>, sblocks, kShadeThreads, 0, st, jobs, P, b, stats);
                        else launch_after(k_wf_shade<J>, sblocks, kShadeThreads, 0, st, jobs, b, w);
                        return cudaGetLastError();
                      }, tail_from);
}

}  // namespace vrt
