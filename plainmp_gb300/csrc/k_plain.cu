// Plain FP64 method: the reference's decisions and values (constraints/primitive_sphere_collision.cpp,
// ompl/motion_validator.cpp) in FP64, bit for bit (compiled --fmad=false), one configuration per warp or per
// four warps (pm_team.cuh).  FP32 only skips what it clears by more than its error bound.
#include <algorithm>

#include "pm_launch.h"
#include "pm_team.cuh"

using namespace pmd;

namespace {

#define PM_CUTOFF 0.1
#define PM_MAX_DOF (PM_MAX_CTRL + 6)

// Collision-free validity of one configuration (is_valid_dirty, primitive_sphere_collision.cpp:181-254) by
// the WPC warps of a team; wi: this warp's number.  Collision = OR over (group, primitive) of [gate AND OR over
// the group's spheres of test], and likewise over pairs, so the order of the tests is free.  `failed` (shared,
// zeroed by the caller) is set when one collides and ends the other warps' loops.
template <int WPC>
__device__ void valid_team(const TView& v, const Image& im, const TeamPose& P, int wi, volatile int* failed) {
  const unsigned FULL = 0xffffffffu;
  const PmTablesHdr* T = v.T;
  const int lane = threadIdx.x & 31;
  const int ng = T->n_groups, np = T->n_prims;
  // ---- groups against primitives, then the spheres of the pairs that FP32 does not clear
  for (int base = 32 * wi; base < ng * np; base += 32 * WPC) {  // warp-uniform
    if (__any_sync(FULL, *failed)) return;
    const int t = base + lane;
    const int gi = t / np, pi = t - gi * np;
    int n = 0;
    if (t < ng * np) {
      const PmGroupF& G = im.grp[gi];
      if (!G.only_self) {
        const PmPrimF& Q = im.prm[pi];
        const float* R = P.at32(G.slot);
        const float3 gc = xf(R, G.rel[0], G.rel[1], G.rel[2]);
        float g, sd, mag;
        if (Q.kind == PM_SDF_CLOUD) {
          const float lb = grid_field_lb16(v.C[Q.cloud], gc.x, gc.y, gc.z);
          g = lb - Q.a - G.radius;
          mag = fabsf(gc.x) + fabsf(gc.y) + fabsf(gc.z) + lb;
        } else {
          clearance(Q, v.C, gc.x, gc.y, gc.z, G.radius, G.tiny, 0.f, g, sd, mag);
        }
        if (!(g > margin32(mag) + cast_error(R, G.gn))) n = G.count;
      }
    }
    bool hit = false;
    warp_spread(n, [&](int owner, int j, bool have) {
      const int g2 = __shfl_sync(FULL, gi, owner), p2 = __shfl_sync(FULL, pi, owner);
      const PmPrim& Q = v.P[p2];
      const PmGroup& G = v.G[g2];
      const int k = G.begin + j;
      bool open = false, search = false;
      int known = -1;
      if (have) {
        const PmSphereF& S = im.sph[k];
        const float* R = P.at32(G.slot);
        const float3 c = xf(R, S.x, S.y, S.z);
        const float ek = cast_error(R, S.sn);
        if (Q.kind == PM_SDF_CLOUD) {
          const FieldLB f = grid_field32(v.C[Q.cloud], c.x, c.y, c.z);
          search = !(f.lb - (float)Q.a - S.r > margin32(fabsf(c.x) + fabsf(c.y) + fabsf(c.z) + f.lb) + ek);
          known = f.idx;
        } else {
          float g, sd, mag;
          clearance(im.prm[p2], v.C, c.x, c.y, c.z, S.r, S.tiny, 0.f, g, sd, mag);
          open = !(g > margin32(mag) + ek);
        }
      }
      if (open) {  // FP64: gate AND test
        const DPose lp = P.at(G.slot);
        const DM3 R = qmat(lp.q);
        const D3 c = add(mv(R, v.rel(k)), lp.t);
        const double r = v.sr[k];
        hit = !outside_aabb(Q, c, r) && !prim_outside(Q, nullptr, c, r) &&
              gate_open(Q, add(mv(R, D3{G.rel[0], G.rel[1], G.rel[2]}), lp.t), G.radius);
      }
      D3 c{0, 0, 0}, gc{0, 0, 0};
      bool gate = true;
      if (search) {
        const DPose lp = P.at(G.slot);
        const DM3 R = qmat(lp.q);
        c = add(mv(R, v.rel(k)), lp.t);
        gc = add(mv(R, D3{G.rel[0], G.rel[1], G.rel[2]}), lp.t);
        search = !outside_aabb(Q, c, v.sr[k]) && !outside_aabb(Q, gc, G.radius);
        if (search && known >= 0) {
          // a point of the cloud inside both spheres settles the search and the gate: the nearest points
          // are no farther, and rounding is monotone
          const PmGridDev& Gd = v.C[Q.cloud];
          const D3 p{Gd.px[known], Gd.py[known], Gd.pz[known]};
          const D3 d = sub(p, c), e = sub(p, gc);
          gate = sqrt(sqn(e)) - Q.a > G.radius;
          hit = hit || (!(sqrt(sqn(d)) - Q.a > v.sr[k]) && !gate);
        }
      }
      if (__any_sync(FULL, hit)) return false;
      for (unsigned bal = __ballot_sync(FULL, search); bal != 0; bal &= bal - 1) {  // warp-uniform
        const int src = __ffs(bal) - 1;
        const int ps = __shfl_sync(FULL, p2, src), ks = __shfl_sync(FULL, k, src), gs = __shfl_sync(FULL, g2, src);
        const PmPrim& Qs = v.P[ps];
        const D3 cs = shfl_d3(c, src), gcs = shfl_d3(gc, src);
        const int hint = __shfl_sync(FULL, known, src);
        int near = -1;
        if (!cloud_outside_warp(Qs, v.C, cs, v.sr[ks], &near, hint)) {
          const PmGridDev& Gd = v.C[Qs.cloud];
          const D3 e = sub(D3{Gd.px[near], Gd.py[near], Gd.pz[near]}, gcs);
          const double rg = v.G[gs].radius;
          hit = !(sqrt(sqn(e)) - Qs.a > rg);
          if (!hit) hit = !cloud_outside_warp(Qs, v.C, gcs, rg, nullptr);
          if (hit) return false;
        }
      }
      return true;
    });
    if (__any_sync(FULL, hit)) {
      if (lane == 0) *failed = 1;
      return;
    }
  }
  // ---- self pairs: the group spheres, then the sphere pairs of the group pairs that FP32 does not clear
  for (int base = 32 * wi; base < T->n_pairs; base += 32 * WPC) {  // warp-uniform
    if (__any_sync(FULL, *failed)) return;
    const int t = base + lane;
    bool near = false;
    int ga = 0, gb = 0;
    if (t < T->n_pairs) {
      ga = v.pairs[2 * t];
      gb = v.pairs[2 * t + 1];
      const PmGroupF &G1 = im.grp[ga], &G2 = im.grp[gb];
      const float *R1 = P.at32(G1.slot), *R2 = P.at32(G2.slot);
      const float3 a = xf(R1, G1.rel[0], G1.rel[1], G1.rel[2]), b = xf(R2, G2.rel[0], G2.rel[1], G2.rel[2]);
      const float dx = a.x - b.x, dy = a.y - b.y, dz = a.z - b.z;
      const float mag = fabsf(a.x) + fabsf(a.y) + fabsf(a.z) + fabsf(b.x) + fabsf(b.y) + fabsf(b.z);
      near = !(sqrtf(fmaf(dx, dx, fmaf(dy, dy, dz * dz))) - (G1.radius + G2.radius) >
               2.0f * margin32(mag) + cast_error(R1, G1.gn) + cast_error(R2, G2.gn));
    }
    for (unsigned bal = __ballot_sync(FULL, near); bal != 0; bal &= bal - 1) {  // warp-uniform
      const int src = __ffs(bal) - 1;
      const int a = __shfl_sync(FULL, ga, src), b = __shfl_sync(FULL, gb, src);
      const PmGroup &G1 = v.G[a], &G2 = v.G[b];
      const float *R1 = P.at32(G1.slot), *R2 = P.at32(G2.slot);
      const int n = G1.count * G2.count;
      bool hit = false;
      for (int u = lane; u < n; u += 32) {
        const int i = G1.begin + u / G2.count, j = G2.begin + u % G2.count;
        const PmSphereF &S1 = im.sph[i], &S2 = im.sph[j];
        const float3 ci = xf(R1, S1.x, S1.y, S1.z), cj = xf(R2, S2.x, S2.y, S2.z);
        const float ex = ci.x - cj.x, ey = ci.y - cj.y, ez = ci.z - cj.z;
        const float mag = fabsf(ci.x) + fabsf(ci.y) + fabsf(ci.z) + fabsf(cj.x) + fabsf(cj.y) + fabsf(cj.z);
        if (sqrtf(fmaf(ex, ex, fmaf(ey, ey, ez * ez))) - (S1.r + S2.r) >
            2.0f * margin32(mag) + cast_error(R1, S1.sn) + cast_error(R2, S2.sn))
          continue;
        const DPose p1 = P.at(G1.slot), p2 = P.at(G2.slot);
        const DM3 M1 = qmat(p1.q), M2 = qmat(p2.q);
        const D3 c1 = add(mv(M1, D3{G1.rel[0], G1.rel[1], G1.rel[2]}), p1.t), c2 = add(mv(M2, D3{G2.rel[0], G2.rel[1], G2.rel[2]}), p2.t);
        const double ors = G1.radius + G2.radius;
        if (sqn(sub(c1, c2)) > ors * ors) continue;
        const double rs = v.sr[i] + v.sr[j];
        hit = hit || sqn(sub(add(mv(M1, v.rel(i)), p1.t), add(mv(M2, v.rel(j)), p2.t))) < rs * rs;
      }
      if (__any_sync(FULL, hit)) {
        if (lane == 0) *failed = 1;
        return;
      }
    }
  }
}

// Dynamic shared memory of a block of nc configurations.
inline size_t team_smem(const PmTablesHdr& h, int nc) { return (size_t)nc * h.n_slots * (kRec * sizeof(double) + kRec32 * sizeof(float)); }

// ConstraintBase::update_kintree (primitive.hpp:38-62) on the model state by a block of at least two warps: the
// control joints' rows on the first warp's lanes (of a repeated joint the last value counts), the base row on
// the second warp.  q: the joint values, then the base's.
__device__ void update_state_block(double* state, const PmSlot* __restrict__ recs, const double* __restrict__ q, int n, int accurate,
                                   int base_type) {
  const int tid = threadIdx.x;
  if (tid < 32) {
    for (int i = tid; i < n; i += 32) {
      bool last = true;
      for (int j = i + 1; j < n; j++) last = last && recs[j].link != recs[i].link;
      if (!last) continue;
      DQ lq;
      D3 lt;
      bool lid;
      joint_local(recs[i], q[i], accurate == 0, lq, lt, lid);
      double* r = state + (int64_t)PM_STATE_LINK_ROW(recs[i].link) * PM_STATE_STRIDE;
      r[0] = lq.x;
      r[1] = lq.y;
      r[2] = lq.z;
      r[3] = lq.w;
      r[4] = lt.x;
      r[5] = lt.y;
      r[6] = lt.z;
      r[7] = lid ? 1.0 : 0.0;
    }
  } else if (tid == 32 && base_type != PM_BASE_FIXED) {
    const double* qb = q + n;
    DQ bq;
    D3 t;
    if (base_type == PM_BASE_FLOATING) {
      t = D3{qb[0], qb[1], qb[2]};
      bq = quat_from_rpy(qb[3], qb[4], qb[5]);
    } else {
      t = D3{qb[0], qb[1], 0.0};
      bq = quat_from_rpy(0, 0, qb[2]);
    }
    double* r = state + PM_STATE_BASE_ROW * PM_STATE_STRIDE;
    r[0] = bq.x;
    r[1] = bq.y;
    r[2] = bq.z;
    r[3] = bq.w;
    r[4] = t.x;
    r[5] = t.y;
    r[6] = t.z;
    r[7] = 0.0;
  }
}

__global__ void k_update_state(double* state, const PmSlot* recs, const double* q, int n, int accurate, int base_type) {
  update_state_block(state, recs, q, n, accurate, base_type);
}

// NC configurations per block, WPC warps each.  Batches run 4 configurations of a warp each at 64 registers:
// 1,500, 4,096 and 16,384 chain states take 40, 62 and 191 us, with 8 at 128 registers 48, 70 and 207, with 4
// at 128 registers 38, 69 and 208, with 2 at 64 registers 40, 77 and 232.  One configuration takes 4 warps at 128.
// UPDATE (one configuration): a second block leaves the model in its state, as is_valid of the reference does.
// The rows it writes (control joints' links, the base row unless the base is fixed) are not among those that
// the check reads (links without a control joint, a fixed base).
template <int NC, int WPC, bool UPDATE = false>
__global__ void __launch_bounds__(NC * WPC * 32, (NC > 1 ? 1024 : 512) / (NC * WPC * 32))
    k_is_valid64(const PmTablesHdr* __restrict__ T, double* state, const double* __restrict__ q, int64_t B, uint8_t* __restrict__ out,
                 const PmSlot* __restrict__ recs, int accurate) {
  extern __shared__ __align__(16) double team_mem[];
  __shared__ int failed[NC];
  if (UPDATE && blockIdx.x == 1) {
    update_state_block(state, recs, q, T->n_ctrl, accurate, T->base_type);
    return;
  }
  const TView v(T);
  const Image im(T);
  const int nsl = T->n_slots, qd = T->q_dim;
  const int64_t c0 = (int64_t)blockIdx.x * NC;
  const int ncfg = (int)min((int64_t)NC, B - c0);
  if (threadIdx.x < NC) failed[threadIdx.x] = 0;
  float* p32 = reinterpret_cast<float*>(team_mem + (size_t)NC * nsl * kRec);
  fk64_block<NC * WPC * 32>(v, state, [&](int c, int col) { return q[(c0 + c) * qd + col]; }, ncfg, T->base_type == PM_BASE_FIXED,
                            kNorm2Valid, team_mem, p32);
  const int c = (threadIdx.x >> 5) / WPC, wi = (threadIdx.x >> 5) % WPC;
  if (c < ncfg) valid_team<WPC>(v, im, TeamPose{team_mem + (size_t)c * nsl * kRec, p32 + (size_t)c * nsl * kRec32}, wi, failed + c);
  __syncthreads();
  if (threadIdx.x < ncfg) out[c0 + threadIdx.x] = failed[threadIdx.x] ? 0 : 1;
}

// Step ratio of checkMotion on the edge a -> b (motion_validator.cpp:17-79).  inv: 1 / width, computed once a block
// (FP64 divisions were most of the time of an edge without length).
__device__ double edge_step(int type, const double* a, const double* b, const double* width, const double* inv, double resolution, int dim) {
  if (type == 0) {  // BoxMotionValidator::determine_step_ratio (:89-111)
    double diff_long = 0.0, max_diff = -INFINITY;
    int li = 0;
    for (int i = 0; i < dim; i++) {
      const double diff = b[i] - a[i];
      const double asd = fabs(diff) * inv[i];
      if (asd > max_diff) {
        max_diff = asd;
        li = i;
        diff_long = diff;
      }
    }
    return fabs(diff_long) < 1e-6 ? INFINITY : width[li] / fabs(diff_long);
  }
  double dist = 0.0;  // EuclideanMotionValidator (:118-126)
  for (int i = 0; i < dim; i++) {
    const double d = a[i] - b[i];
    dist += d * d;
  }
  return resolution / sqrt(dist);
}
// Waypoints to check, or 0 where the step ratio decides: `valid` is the answer then.  NaN / non-positive ratios,
// and edges needing more than 2^26 waypoints, are reported invalid instead of looping (the reference has no bound
// here).
__device__ int edge_waypoints(double sr, bool& valid) {
  valid = sr == INFINITY;
  if (valid || !(sr > 0.0) || 1.0 / sr > 67108864.0) return 0;
  return (int)(floor(1 / sr) + 1);
}
// Coordinate of waypoint k of n: b for k = 0, then the interior points in visiting order (:45-78).
__device__ __forceinline__ double edge_value(double a, double b, double sr, int n, int k, const int16_t* __restrict__ seq) {
  if (k == 0) return b;
  return a + (b - a) * (n < 128 ? (double)seq[n * 128 + (k + 1)] * sr : (double)k * sr);
}

// CustomValidatorBase::checkMotion, a block per edge: its waypoints in the reference's visiting order, NC at a
// time, a warp each; the first round with a collision ends it.
// n_checked (a sum) and counts (per edge), each optional, count the waypoints up to and including the first
// that collides, as the reference visits them.  The endpoints go to shared memory first: small calls pass them
// in page-locked host memory.
template <int NC>
__global__ void __launch_bounds__(NC * 32, 512 / (NC * 32)) k_check_motion64(const PmTablesHdr* __restrict__ T, const double* __restrict__ state,
                                                            const double* __restrict__ s1, const double* __restrict__ s2, int type,
                                                            const double* __restrict__ width, double resolution,
                                                            const int16_t* __restrict__ seq, uint8_t* __restrict__ out,
                                                            unsigned long long* n_checked, unsigned long long* counts) {
  extern __shared__ __align__(16) double team_mem[];
  __shared__ int failed[NC];
  __shared__ double ends[2][PM_MAX_DOF], inv[PM_MAX_DOF];
  __shared__ double step;
  __shared__ int n_way;  // waypoints to check (0: decided already)
  const TView v(T);
  const Image im(T);
  const int64_t e = blockIdx.x;
  const int dim = T->q_dim, nsl = T->n_slots;
  const double *a = ends[0], *b = ends[1];
  for (int i = threadIdx.x; i < dim; i += NC * 32) {
    ends[0][i] = s1[e * dim + i];
    ends[1][i] = s2[e * dim + i];
    if (type == 0) inv[i] = 1.0 / width[i];
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    bool valid;
    step = edge_step(type, a, b, width, inv, resolution, dim);
    n_way = edge_waypoints(step, valid);
    if (counts) counts[e] = 0;
    if (n_way == 0) out[e] = valid;
  }
  __syncthreads();
  const double sr = step;
  const int n = n_way;
  if (n == 0) return;  // block-uniform
  float* p32 = reinterpret_cast<float*>(team_mem + (size_t)NC * nsl * kRec);
  int k0 = 0, checked = n;
  bool ok = true;
  for (; k0 < n && ok; k0 += NC) {  // block-uniform
    const int ncfg = min(NC, n - k0);
    if (threadIdx.x < NC) failed[threadIdx.x] = 0;
    auto qf = [&](int c, int col) { return edge_value(a[col], b[col], sr, n, k0 + c, seq); };
    fk64_block<NC * 32>(v, state, qf, ncfg, T->base_type == PM_BASE_FIXED, kNorm2Valid, team_mem, p32);
    const int c = threadIdx.x >> 5;
    if (c < ncfg) valid_team<1>(v, im, TeamPose{team_mem + (size_t)c * nsl * kRec, p32 + (size_t)c * nsl * kRec32}, 0, failed + c);
    __syncthreads();
    for (int i = 0; i < ncfg && ok; i++)
      if (failed[i]) {
        ok = false;
        checked = k0 + i + 1;
      }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    out[e] = ok ? 1 : 0;
    if (n_checked) atomicAdd(n_checked, (unsigned long long)checked);
    if (counts) counts[e] = checked;
  }
}

// The same for 16 edges per SM and more, G (2 to 64) edges a block: the waypoints of its edges in a row, NC at a time,
// leaving out those of an edge that has collided.  A block an edge, as above, has NC - 1 warps idle where edges are
// of one waypoint, and starts a block for each edge without length: 100,000 chain edges of one waypoint took 7.4 ms,
// 1.41 this way; of no length 1.01 ms, 0.10; 20,000 of three 1.66 ms, 0.84; 1,000 of twenty 0.24 ms either way.
// (Up to 32 a block 1.34 and 0.13 ms for the first two, up to 128 1.50 and 0.10.)
constexpr int kEdgesPerBlock = 64;
static_assert(kEdgesPerBlock % 32 == 0, "whole warps");
template <int NC>
__global__ void __launch_bounds__(NC * 32, 512 / (NC * 32)) k_check_motions64(const PmTablesHdr* __restrict__ T, const double* __restrict__ state,
                                                            const double* __restrict__ s1, const double* __restrict__ s2, int64_t E, int G,
                                                            int type, const double* __restrict__ width, double resolution,
                                                            const int16_t* __restrict__ seq, uint8_t* __restrict__ out,
                                                            unsigned long long* n_checked, unsigned long long* counts) {
  extern __shared__ __align__(16) double team_mem[];
  __shared__ int failed[NC];
  __shared__ double step[kEdgesPerBlock], inv[PM_MAX_DOF];
  __shared__ int n_way[kEdgesPerBlock];   // waypoints of an edge (0: decided already)
  __shared__ int checked[kEdgesPerBlock];  // up to its first collision (0: none yet)
  __shared__ int task_e[NC], task_k[NC], n_task;
  static_assert(kEdgesPerBlock <= NC * 32, "a thread an edge");
  const TView v(T);
  const Image im(T);
  const int tid = threadIdx.x;
  const int64_t e0 = (int64_t)blockIdx.x * G;
  const int ge = (int)min((int64_t)G, E - e0);
  const int dim = T->q_dim, nsl = T->n_slots;
  if (type == 0)
    for (int i = tid; i < dim; i += NC * 32) inv[i] = 1.0 / width[i];
  __syncthreads();
  if (tid < ge) {
    const int64_t e = e0 + tid;
    bool valid;
    step[tid] = edge_step(type, s1 + e * dim, s2 + e * dim, width, inv, resolution, dim);
    n_way[tid] = edge_waypoints(step[tid], valid);
    checked[tid] = 0;
    if (n_way[tid] == 0) out[e] = valid;
  }
  __syncthreads();
  float* p32 = reinterpret_cast<float*>(team_mem + (size_t)NC * nsl * kRec);
  int ce = 0, ck = 0;  // thread 0: the next edge and waypoint
  for (;;) {  // block-uniform
    if (tid == 0) {
      int m = 0;
      while (m < NC && ce < ge) {
        if (ck >= n_way[ce] || checked[ce]) {
          ce++;
          ck = 0;
        } else {
          task_e[m] = ce;
          task_k[m] = ck++;
          failed[m++] = 0;
        }
      }
      n_task = m;
    }
    __syncthreads();
    const int ncfg = n_task;
    if (ncfg == 0) break;
    auto qf = [&](int c, int col) {
      const int i = task_e[c];
      const int64_t at = (e0 + i) * dim + col;
      return edge_value(s1[at], s2[at], step[i], n_way[i], task_k[c], seq);
    };
    fk64_block<NC * 32>(v, state, qf, ncfg, T->base_type == PM_BASE_FIXED, kNorm2Valid, team_mem, p32);
    const int c = tid >> 5;
    if (c < ncfg) valid_team<1>(v, im, TeamPose{team_mem + (size_t)c * nsl * kRec, p32 + (size_t)c * nsl * kRec32}, 0, failed + c);
    __syncthreads();
    if (tid == 0)
      for (int i = 0; i < ncfg; i++)
        if (failed[i] && !checked[task_e[i]]) checked[task_e[i]] = task_k[i] + 1;
  }
  if (tid < kEdgesPerBlock) {  // whole warps
    unsigned long long n = 0;
    if (tid < ge) {
      if (n_way[tid] > 0) {
        n = checked[tid] ? checked[tid] : n_way[tid];
        out[e0 + tid] = checked[tid] ? 0 : 1;
      }
      if (counts) counts[e0 + tid] = n;
    }
    for (int o = 16; o > 0; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
    if ((tid & 31) == 0 && n > 0 && n_checked) atomicAdd(n_checked, n);
  }
}

// The smallest of a warp's values and its place in the reference's order (ties go to the earlier term).
struct Least {
  double val;
  unsigned long long order;
  __device__ __forceinline__ void take(double v, unsigned long long o) {
    if (v < val || (v == val && o < order)) {
      val = v;
      order = o;
    }
  }
  __device__ __forceinline__ void share() {
    for (int o = 16; o > 0; o >>= 1) {
      const double ov = __shfl_xor_sync(0xffffffffu, val, o);
      const unsigned long long oo = __shfl_xor_sync(0xffffffffu, order, o);
      take(ov, oo);
    }
  }
};
constexpr unsigned long long kNoTerm = ~0ull;

// Column d of get_attached_point_jacobian (algorithm.cpp:346-433) for the point p of a slot's link.
__device__ D3 attached_column(const TView& v, const TeamPose& P, int plink_slot, const D3& p, int d) {
  const int nc = v.T->n_ctrl;
  if (d < nc) {
    const PmJoint& J = v.J[d];
    if (J.slot < 0 || !((v.S[plink_slot].relevant >> d) & 1ull)) return D3{0.0, 0.0, 0.0};
    const DPose tc = P.at(J.slot);
    const D3 wa = qrot(tc.q, D3{J.axis[0], J.axis[1], J.axis[2]});
    return J.prismatic ? wa : cross(wa, sub(p, tc.t));
  }
  const int k = d - nc;  // FLOATING: x y z roll pitch yaw; PLANAR: x y yaw
  const bool floating = v.T->base_type == PM_BASE_FLOATING;
  const int n_trans = floating ? 3 : 2;
  if (k < n_trans) return D3{k == 0 ? 1.0 : 0.0, k == 1 ? 1.0 : 0.0, k == 2 ? 1.0 : 0.0};
  // the angle columns by the reference's forward differences
  const double eps = 1e-7;
  DPose te;
  te.q = DQ{0, 0, 0, 1};
  te.t = p;
  const DPose tb = P.at(v.T->root_slot);
  const DPose tbe = pose_mul(pose_inverse(tb), te);
  const D3 rpy = get_rpy(tb.q);
  const int ang = floating ? k - 3 : 2;
  DPose tw = tb;
  tw.q = quat_from_rpy(ang == 0 ? rpy.x + eps : rpy.x, ang == 1 ? rpy.y + eps : rpy.y, ang == 2 ? rpy.z + eps : rpy.z);
  const D3 dp = sub(pose_mul(tw, tbe).t, te.t);
  return D3{dp.x / eps, dp.y / eps, dp.z / eps};
}

// evaluate_ext_collision (primitive_sphere_collision.cpp:256-322) by one warp: the least value of a sphere
// against a primitive below the cutoff, and its gradient row.  FP32 finds an upper bound of that value (each
// term's distance plus its error; the nearest point that the field stores, for a cloud), then FP64 evaluates
// the terms whose lower bound does not exceed it: one to three of a few hundred.
__device__ double eval_ext_warp(const TView& v, const Image& im, const TeamPose& P, double* grad) {
  const unsigned FULL = 0xffffffffu;
  const PmTablesHdr* T = v.T;
  const int lane = threadIdx.x & 31;
  const int ng = T->n_groups, np = T->n_prims, dof = T->q_dim;
  const float stretch = T->stretch;
  Least best{PM_CUTOFF, kNoTerm};
  float upper = (float)PM_CUTOFF;  // no term above it can be the least
  for (int pass = 0; pass < 2; pass++) {  // 0: the bound; 1: the values
    for (int base = 0; base < ng * np; base += 32) {  // warp-uniform
      const int t = base + lane;
      const int gi = t / np, pi = t - gi * np;
      int n = 0;
      if (t < ng * np) {
        const PmGroupF& G = im.grp[gi];
        if (!G.only_self) {
          const PmPrimF& Q = im.prm[pi];
          const float* R = P.at32(G.slot);
          const float3 gc = xf(R, G.rel[0], G.rel[1], G.rel[2]);
          float g, sd, mag;
          if (Q.kind == PM_SDF_CLOUD) {
            const float lb = grid_field_lb16(v.C[Q.cloud], gc.x, gc.y, gc.z);
            sd = g = lb - Q.a - G.radius;
            mag = fabsf(gc.x) + fabsf(gc.y) + fabsf(gc.z) + lb;
          } else {
            clearance(Q, v.C, gc.x, gc.y, gc.z, G.radius, G.tiny, 0.f, g, sd, mag);
          }
          // sd bounds the values of the group's spheres from below: beyond the cutoff its gate is closed,
          // beyond the bound none of them is the least.  The ground's gate tests more than the distance
          // (g), and only the cutoff counts for it.  (g of a box or cylinder ends at -radius inside it.)
          const bool by_gate = Q.kind == PM_SDF_GROUND;
          if (!((by_gate ? g : sd) > (by_gate ? (float)PM_CUTOFF : upper) + margin32(mag) + cast_error(R, G.gn) + stretch * G.radius)) n = G.count;
        }
      }
      warp_spread(n, [&](int owner, int j, bool have) {
        const int g2 = __shfl_sync(FULL, gi, owner), p2 = __shfl_sync(FULL, pi, owner), t2 = __shfl_sync(FULL, t, owner);
        const PmPrim& Q = v.P[p2];
        const PmGroup& G = v.G[g2];
        const int k = G.begin + j;
        bool open = false, search = false;
        int known = -1;
        if (have) {
          const PmSphereF& S = im.sph[k];
          const float* R = P.at32(G.slot);
          const float3 c = xf(R, S.x, S.y, S.z);
          const float ek = cast_error(R, S.sn) + stretch * im.grp[g2].radius;
          if (Q.kind == PM_SDF_CLOUD) {
            const PmGridDev& Gd = v.C[Q.cloud];
            const float qmag = fabsf(c.x) + fabsf(c.y) + fabsf(c.z);
            const FieldLB f = grid_field32(Gd, c.x, c.y, c.z, true);
            search = !(f.lb - (float)Q.a - S.r > upper + margin32(qmag + f.lb) + ek);
            known = f.idx;
            if (pass == 0 && f.idx >= 0) {
              const float ex = f.np.x - c.x, ey = f.np.y - c.y, ez = f.np.z - c.z;
              const float ub = sqrtf(fmaf(ex, ex, fmaf(ey, ey, ez * ez)));
              upper = fminf(upper, ub - (float)Q.a - S.r + margin32(qmag + ub) + ek);
            }
          } else {
            float g, sd, mag;
            clearance(im.prm[p2], v.C, c.x, c.y, c.z, S.r, S.tiny, 0.f, g, sd, mag);
            const float m = margin32(mag) + ek;
            open = !(sd > upper + m);
            if (pass == 0 && Q.kind != PM_SDF_GROUND) upper = fminf(upper, sd + m);
          }
        }
        if (pass == 0) return true;
        const unsigned long long order = (unsigned long long)t2 << 32 | (unsigned)k;
        const double r = v.sr[k];
        D3 c{0, 0, 0}, gc{0, 0, 0};
        if (open || search) {
          const DPose lp = P.at(G.slot);
          const DM3 R = qmat(lp.q);
          c = add(mv(R, v.rel(k)), lp.t);
          gc = add(mv(R, D3{G.rel[0], G.rel[1], G.rel[2]}), lp.t);
          const bool far = outside_aabb(Q, c, r + PM_CUTOFF) || outside_aabb(Q, gc, G.radius + PM_CUTOFF);
          open = open && !far && !prim_outside(Q, nullptr, gc, G.radius + PM_CUTOFF);
          search = search && !far;
          if (open) best.take(prim_eval(Q, nullptr, c) - r, order);
        }
        for (unsigned bal = __ballot_sync(FULL, search); bal != 0; bal &= bal - 1) {  // warp-uniform
          const int src = __ffs(bal) - 1;
          const int ps = __shfl_sync(FULL, p2, src), hint = __shfl_sync(FULL, known, src);
          const PmPrim& Qs = v.P[ps];
          const D3 cs = shfl_d3(c, src), gcs = shfl_d3(gc, src);
          const double rs = shfl_d(r, src), rg = shfl_d(G.radius, src);
          const bool scales = isnan(P.at32(v.G[__shfl_sync(FULL, g2, src)].slot)[3]);  // the group sphere may not hold its spheres
          const unsigned long long os = __shfl_sync(FULL, order, src);
          // only a value up to the smallest so far matters: search slightly beyond its reach
          const double reach = ((double)upper + Qs.a + rs) * (1.0 + 1e-6) + 1e-6;
          if (!(reach > 0.0)) continue;
          const NNResult64 nn = warp_nearest64(v.C[Qs.cloud], cs, reach * reach, hint);
          if (nn.idx < 0) continue;
          const double val = sqrt(nn.d2) - Qs.a - rs;
          // below the cutoff the gate is open, but for rounding at the cutoff itself
          if ((scales || val > PM_CUTOFF - 1e-6 - stretch * rg) && cloud_outside_warp(Qs, v.C, gcs, rg + PM_CUTOFF, nullptr)) continue;
          if (val < PM_CUTOFF) best.take(val, os);  // the same on every lane
          upper = fminf(upper, (float)val + 1e-6f * (1.0f + fabsf((float)val)));
        }
        return true;
      });
    }
    if (pass == 0)
      for (int o = 16; o > 0; o >>= 1) upper = fminf(upper, __shfl_xor_sync(FULL, upper, o));
  }
  if (!(best.val < PM_CUTOFF)) best = Least{PM_CUTOFF, kNoTerm};
  best.share();
  if (best.order == kNoTerm) {
    for (int d = lane; d < dof; d += 32) grad[d] = 0.0;
    return best.val;
  }
  const int t = (int)(best.order >> 32), k = (int)(best.order & 0xffffffffu);
  const PmGroup& G = v.G[t / np];
  const PmPrim& Q = v.P[t % np];
  const D3 sc = P.point(G.slot, v.rel(k));
  const double r = v.sr[k];
  double g3[3];
  if (Q.kind == PM_SDF_CLOUD) {
    double d3[3] = {INFINITY, INFINITY, INFINITY};
    warp_nearest64<3>(v.C[Q.cloud], sc, INFINITY, -1, d3);
    for (int i = 0; i < 3; i++) g3[i] = (((sqrt(d3[i]) - Q.a) - r) - best.val) / 1e-6;
  } else {  // a lane per axis
    D3 pc = sc;
    if (lane == 0) pc.x += 1e-6;
    if (lane == 1) pc.y += 1e-6;
    if (lane == 2) pc.z += 1e-6;
    const double g = ((prim_eval(Q, nullptr, pc) - r) - best.val) / 1e-6;
    for (int i = 0; i < 3; i++) g3[i] = shfl_d(g, i);
  }
  for (int d = lane; d < dof; d += 32) {
    const D3 j = attached_column(v, P, G.slot, sc, d);
    grad[d] = j.x * g3[0] + j.y * g3[1] + j.z * g3[2];
  }
  return best.val;
}

// evaluate_self_collision (primitive_sphere_collision.cpp:324-383) by one warp, in the same two passes.
__device__ double eval_self_warp(const TView& v, const Image& im, const TeamPose& P, double* grad) {
  const unsigned FULL = 0xffffffffu;
  const PmTablesHdr* T = v.T;
  const int lane = threadIdx.x & 31;
  const int dof = T->q_dim;
  const float stretch = T->stretch;
  Least best{PM_CUTOFF, kNoTerm};
  float upper = (float)PM_CUTOFF;
  for (int pass = 0; pass < 2; pass++) {
    for (int base = 0; base < T->n_pairs; base += 32) {  // warp-uniform
      const int t = base + lane;
      bool near = false;
      int ga = 0, gb = 0;
      if (t < T->n_pairs) {
        ga = v.pairs[2 * t];
        gb = v.pairs[2 * t + 1];
        const PmGroupF &G1 = im.grp[ga], &G2 = im.grp[gb];
        const float *R1 = P.at32(G1.slot), *R2 = P.at32(G2.slot);
        const float3 a = xf(R1, G1.rel[0], G1.rel[1], G1.rel[2]), b = xf(R2, G2.rel[0], G2.rel[1], G2.rel[2]);
        const float dx = a.x - b.x, dy = a.y - b.y, dz = a.z - b.z;
        const float mag = fabsf(a.x) + fabsf(a.y) + fabsf(a.z) + fabsf(b.x) + fabsf(b.y) + fabsf(b.z);
        near = !(sqrtf(fmaf(dx, dx, fmaf(dy, dy, dz * dz))) - (G1.radius + G2.radius) >
                 upper + 2.0f * margin32(mag) + cast_error(R1, G1.gn) + cast_error(R2, G2.gn) + stretch * (G1.radius + G2.radius));
      }
      for (unsigned bal = __ballot_sync(FULL, near); bal != 0; bal &= bal - 1) {  // warp-uniform
        const int src = __ffs(bal) - 1;
        const int a = __shfl_sync(FULL, ga, src), b = __shfl_sync(FULL, gb, src);
        const PmGroup &G1 = v.G[a], &G2 = v.G[b];
        const float *R1 = P.at32(G1.slot), *R2 = P.at32(G2.slot);
        const int n = G1.count * G2.count;
        for (int u = lane; u < n; u += 32) {
          const int i = G1.begin + u / G2.count, j = G2.begin + u % G2.count;
          const PmSphereF &S1 = im.sph[i], &S2 = im.sph[j];
          const float3 ci = xf(R1, S1.x, S1.y, S1.z), cj = xf(R2, S2.x, S2.y, S2.z);
          const float ex = ci.x - cj.x, ey = ci.y - cj.y, ez = ci.z - cj.z;
          const float mag = fabsf(ci.x) + fabsf(ci.y) + fabsf(ci.z) + fabsf(cj.x) + fabsf(cj.y) + fabsf(cj.z);
          const float d32 = sqrtf(fmaf(ex, ex, fmaf(ey, ey, ez * ez))) - (S1.r + S2.r);
          const float m = 2.0f * margin32(mag) + cast_error(R1, S1.sn) + cast_error(R2, S2.sn) + stretch * (im.grp[a].radius + im.grp[b].radius);
          if (pass == 0) {
            upper = fminf(upper, d32 + m);
            continue;
          }
          if (d32 > upper + m) continue;
          const DPose p1 = P.at(G1.slot), p2 = P.at(G2.slot);
          const DM3 M1 = qmat(p1.q), M2 = qmat(p2.q);
          const D3 c1 = add(mv(M1, D3{G1.rel[0], G1.rel[1], G1.rel[2]}), p1.t);
          const D3 c2 = add(mv(M2, D3{G2.rel[0], G2.rel[1], G2.rel[2]}), p2.t);
          const double orm = G1.radius + G2.radius + PM_CUTOFF;
          if (sqn(sub(c1, c2)) > orm * orm) continue;
          const double d = nrm(sub(add(mv(M1, v.rel(i)), p1.t), add(mv(M2, v.rel(j)), p2.t))) - (v.sr[i] + v.sr[j]);
          if (d < PM_CUTOFF) best.take(d, (unsigned long long)(base + src) << 42 | (unsigned long long)(i - G1.begin) << 21 | (unsigned)(j - G2.begin));
        }
        __syncwarp();
      }
    }
    if (pass == 0)
      for (int o = 16; o > 0; o >>= 1) upper = fminf(upper, __shfl_xor_sync(FULL, upper, o));
  }
  best.share();
  if (best.order == kNoTerm) {
    for (int d = lane; d < dof; d += 32) grad[d] = 0.0;
    return best.val;
  }
  const int pr = (int)(best.order >> 42);
  const PmGroup &G1 = v.G[v.pairs[2 * pr]], &G2 = v.G[v.pairs[2 * pr + 1]];
  const int i = G1.begin + (int)(best.order >> 21 & 0x1fffffu), j = G2.begin + (int)(best.order & 0x1fffffu);
  const D3 c1 = P.point(G1.slot, v.rel(i)), c2 = P.point(G2.slot, v.rel(j));
  const D3 cd = sub(c1, c2);
  const double ni = 1.0 / nrm(cd);
  for (int d = lane; d < dof; d += 32) {
    const D3 a = attached_column(v, P, G1.slot, c1, d), b = attached_column(v, P, G2.slot, c2, d);
    grad[d] = cd.x * ni * (a.x - b.x) + cd.y * ni * (a.y - b.y) + cd.z * ni * (a.z - b.z);
  }
  return best.val;
}

// NC configurations per block, two warps each: one for the row against the environment, one for the
// self-collision row.
template <int NC>
__global__ void __launch_bounds__(NC * 64, 512 / (NC * 64)) k_evaluate64(const PmTablesHdr* __restrict__ T, const double* __restrict__ state,
                                                        const double* __restrict__ q, int64_t B, int high_accuracy,
                                                        double* __restrict__ vals, double* __restrict__ jac) {
  extern __shared__ __align__(16) double team_mem[];
  const TView v(T);
  const Image im(T);
  const int nsl = T->n_slots, qd = T->q_dim;
  const int64_t c0 = (int64_t)blockIdx.x * NC;
  const int ncfg = (int)min((int64_t)NC, B - c0);
  float* p32 = reinterpret_cast<float*>(team_mem + (size_t)NC * nsl * kRec);
  fk64_block<NC * 64>(v, state, [&](int c, int col) { return q[(c0 + c) * qd + col]; }, ncfg, !high_accuracy, kNorm2Eval, team_mem, p32);
  const int c = threadIdx.x >> 6;
  if (c >= ncfg) return;
  const TeamPose P{team_mem + (size_t)c * nsl * kRec, p32 + (size_t)c * nsl * kRec32};
  const int ext = T->n_prims > 0 ? 1 : 0, m = ext + (T->n_pairs > 0 ? 1 : 0);
  const bool self = (threadIdx.x >> 5) & 1;
  if (self ? T->n_pairs <= 0 : !ext) return;
  const int row = self ? ext : 0;
  double* g = jac + ((c0 + c) * m + row) * (int64_t)qd;
  const double val = self ? eval_self_warp(v, im, P, g) : eval_ext_warp(v, im, P, g);
  if ((threadIdx.x & 31) == 0) vals[(c0 + c) * m + row] = val;
}

// Per-sphere signed distances in two launches: the FP64 sphere centres (one thread per configuration:
// the FK), then the SDF of every (configuration, sphere) in its own thread or warp, so the nearest-point
// searches of a batch run side by side instead of one configuration's 120 in a row.
__global__ void k_sphere_centres64(const PmTablesHdr* __restrict__ T, const double* __restrict__ state, const double* __restrict__ q,
                                   int64_t B, int high_accuracy, double* __restrict__ centres) {
  int64_t b = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (b >= B) return;
  TView v(T);
  DPose pose[PM_MAX_SLOTS];
  fk64(T, state, q + b * T->q_dim, !high_accuracy, pose);
  const int ns = T->n_spheres;
  for (int gi = 0; gi < T->n_groups; gi++) {
    const PmGroup& g = v.G[gi];
    DM3 R = qmat(pose[g.slot].q);
    for (int k = g.begin; k < g.begin + g.count; k++) {
      D3 c = add(mv(R, v.rel(k)), pose[g.slot].t);
      centres[(b * ns + k) * 3 + 0] = c.x;
      centres[(b * ns + k) * 3 + 1] = c.y;
      centres[(b * ns + k) * 3 + 2] = c.z;
    }
  }
}
// f(primitive) for each point cloud among n primitives, on every lane of the warp; until f returns false.
template <class F>
__device__ __forceinline__ void each_cloud(const PmPrim* prims, int n, const F& f) {
  for (int base = 0; base < n; base += 32) {
    const int k = base + (threadIdx.x & 31);
    // every lane loads: a branch around the load parts the lanes, and all that follows issues twice (k_sphere_sdf64
    // over 4,096 chain states and the cloud 810 -> 1605 us)
    const bool is_cloud = prims[min(k, n - 1)].kind == PM_SDF_CLOUD && k < n;
    __syncwarp();
    for (unsigned bal = __ballot_sync(0xffffffffu, is_cloud); bal != 0; bal &= bal - 1)
      if (!f(prims[base + __ffs(bal) - 1])) return;
  }
}

// The primitives by a thread per sphere, the point clouds by a warp per sphere (CLOUD), for the cooperative search;
// `fold`: the other kernel has written the distances to the primitives.  (Both by the warp: every lane evaluated
// every primitive, and 4,096 chain states against the cloud and 1,000 boxes took 621 ms, split in two 21.)
template <bool CLOUD>
__global__ void k_sphere_sdf64(const PmTablesHdr* __restrict__ T, const double* __restrict__ centres, int64_t n, bool fold,
                               double* __restrict__ dist) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (CLOUD) i >>= 5;
  if (i >= n) return;
  TView v(T);
  const double r = v.sr[(int)(i % T->n_spheres)];
  const D3 c{centres[3 * i], centres[3 * i + 1], centres[3 * i + 2]};
  double d = fold ? dist[i] : INFINITY;
  if (CLOUD) {
    each_cloud(v.P, T->n_prims, [&](const PmPrim& P) {
      d = fmin(d, cloud_eval_warp(P, v.C, c) - r);
      return true;
    });
  } else {
    for (int pi = 0; pi < T->n_prims; pi++)
      if (v.P[pi].kind != PM_SDF_CLOUD) d = fmin(d, prim_eval(v.P[pi], v.C, c) - r);
  }
  __syncwarp();  // every lane has read dist[i]
  if (!CLOUD || (threadIdx.x & 31) == 0) dist[i] = d;
}

__global__ void k_spheres_of_state(const PmTablesHdr* __restrict__ T, const double* __restrict__ state, int groups,
                                   double* __restrict__ out4) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  TView v(T);
  DPose pose[PM_MAX_SLOTS];
  // the state already holds the local transforms of every joint
  const PmSlot* S = v.S;
  bool dummy;
  DPose base = state_pose(state, PM_STATE_BASE_ROW, dummy);
  for (int i = 0; i < T->n_slots; i++) {
    if (S[i].parent < 0) {
      pose[i] = base;
      continue;
    }
    bool lid;
    DPose l = state_pose(state, PM_STATE_LINK_ROW(S[i].link), lid);
    pose[i] = compose(pose[S[i].parent], l.q, l.t, lid);
  }
  int k = 0;
  for (int gi = 0; gi < T->n_groups; gi++) {
    const PmGroup& g = v.G[gi];
    DM3 R;
    D3 gc = group_centre(v, g, pose[g.slot], R);
    if (groups) {
      out4[4 * gi + 0] = gc.x;
      out4[4 * gi + 1] = gc.y;
      out4[4 * gi + 2] = gc.z;
      out4[4 * gi + 3] = g.radius;
      continue;
    }
    for (int s = g.begin; s < g.begin + g.count; s++, k++) {
      D3 c = add(mv(R, v.rel(s)), pose[g.slot].t);
      out4[4 * k + 0] = c.x;
      out4[4 * k + 1] = c.y;
      out4[4 * k + 2] = c.z;
      out4[4 * k + 3] = v.sr[s];
    }
  }
}

// ------------------------------------------------------------------ model state
// build_cache_until for selected links (algorithm.cpp:160-210)
__global__ void k_link_poses(const double* __restrict__ state, const int32_t* __restrict__ parents, const int32_t* __restrict__ links,
                             int n, double* __restrict__ out7) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int chain[256];
  int depth = 0;
  int h = links[i];
  while (h >= 0 && parents[h] >= 0 && depth < 256) {
    chain[depth++] = h;
    h = parents[h];
  }
  bool dummy;
  DPose p = state_pose(state, PM_STATE_BASE_ROW, dummy);
  while (depth > 0) {
    int l = chain[--depth];
    bool lid;
    DPose loc = state_pose(state, PM_STATE_LINK_ROW(l), lid);
    p = compose(p, loc.q, loc.t, lid);
  }
  double* o = out7 + 7 * i;
  o[0] = p.t.x;
  o[1] = p.t.y;
  o[2] = p.t.z;
  o[3] = p.q.x;
  o[4] = p.q.y;
  o[5] = p.q.z;
  o[6] = p.q.w;
}

// ------------------------------------------------------------------ SDF utilities
// The primitives by a thread per point, the point clouds by a warp per point (CLOUD), for the cooperative search;
// `fold`: the other kernel has written the outcome of the primitives.  (Both by the warp: 100,000 points against a
// cloud and 200 boxes took 53.5 ms, split in two 2.5.)
template <bool CLOUD>
__global__ void k_sdf_points(const PmPrim* __restrict__ prims, int n_prims, const PmGridDev* __restrict__ clouds, int is_union, bool fold,
                             const double* __restrict__ pts, const double* __restrict__ radii, int64_t n, double* eval_out,
                             uint8_t* outside_out) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (CLOUD) i >>= 5;
  if (i >= n) return;
  const bool writer = !CLOUD || (threadIdx.x & 31) == 0;
  D3 p{pts[3 * i], pts[3 * i + 1], pts[3 * i + 2]};
  if (eval_out) {
    double v = fold ? eval_out[i] : (is_union ? 1.7976931348623157e308 : 0.0);
    auto take = [&](double e) { v = is_union ? fmin(v, e) : e; };
    const int m = is_union ? n_prims : min(n_prims, 1);
    if (CLOUD) {
      each_cloud(prims, m, [&](const PmPrim& P) {
        take(cloud_eval_warp(P, clouds, p));
        return true;
      });
    } else {
      for (int k = 0; k < m; k++)
        if (prims[k].kind != PM_SDF_CLOUD) take(prim_eval(prims[k], clouds, p));
    }
    __syncwarp();  // every lane has read eval_out[i]
    if (writer) eval_out[i] = v;
  }
  if (outside_out) {
    bool o = !fold || outside_out[i] != 0;
    if (CLOUD) {
      if (o) each_cloud(prims, n_prims, [&](const PmPrim& P) { return o = cloud_outside_warp(P, clouds, p, radii[i], nullptr); });
    } else {
      for (int k = 0; k < n_prims && o; k++)
        if (prims[k].kind != PM_SDF_CLOUD) o = prim_outside(prims[k], clouds, p, radii[i]);
    }
    __syncwarp();
    if (writer) outside_out[i] = o ? 1 : 0;
  }
}

// KDTree::query / sqdist: one warp per query (warp_nearest64).
__global__ void __launch_bounds__(256) k_cloud_nearest(const PmGridDev* __restrict__ grid, const double* __restrict__ pts, int64_t n,
                                                       double* sq, double* near3) {
  const int64_t i = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  if (i >= n) return;
  const int lane = threadIdx.x & 31;
  const D3 p{pts[3 * i], pts[3 * i + 1], pts[3 * i + 2]};
  const NNResult64 r = warp_nearest64(*grid, p);
  if (lane == 0 && sq) sq[i] = r.d2;
  if (lane < 3 && near3) near3[3 * i + lane] = r.idx < 0 ? NAN : (lane == 0 ? grid->px : (lane == 1 ? grid->py : grid->pz))[r.idx];
}

inline unsigned grid_for(int64_t n, int bs) { return (unsigned)((n + bs - 1) / bs); }

// Launches a kernel of nc configurations per block, wpc warps each.
template <class K, class... A>
cudaError_t team_launch(K kern, int64_t blocks, int nc, int wpc, const PmTablesHdr& h, cudaStream_t s, A... args) {
  const size_t sm = team_smem(h, nc);  // with the static part it may pass 48 KB long before it does alone
  const cudaError_t e = pmg::raise_smem(reinterpret_cast<const void*>(kern), sm);
  if (e != cudaSuccess) return e;
  kern<<<(unsigned)blocks, nc * wpc * 32, sm, s>>>(args...);
  return cudaGetLastError();
}

}  // namespace

namespace pmg {

cudaError_t launch_update_state(double* state, const PmSlot* recs, const double* q, int n, int accurate, int base_type, cudaStream_t s) {
  k_update_state<<<1, 64, 0, s>>>(state, recs, q, n, accurate, base_type);
  return cudaGetLastError();
}
cudaError_t launch_link_poses(const double* state, const int32_t* parents, const int32_t* links, int n, double* out7,
                              cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  k_link_poses<<<grid_for(n, 64), 64, 0, s>>>(state, parents, links, n, out7);
  return cudaGetLastError();
}
cudaError_t launch_is_valid64(const PmTablesHdr* T, const PmTablesHdr& h, const double* state, const double* q, int64_t B,
                              uint8_t* out, cudaStream_t s) {
  if (B <= 0) return cudaSuccess;
  int n_sm = 0;
  cudaError_t e = sm_count(&n_sm);
  if (e != cudaSuccess) return e;
  double* st = const_cast<double*>(state);  // written only with UPDATE
  prof_begin("k_is_valid64", s);
  if (B <= 4 * (int64_t)n_sm)
    e = team_launch(k_is_valid64<1, 4>, B, 1, 4, h, s, T, st, q, B, out, (const PmSlot*)nullptr, 0);
  else
    e = team_launch(k_is_valid64<4, 1>, (B + 3) / 4, 4, 1, h, s, T, st, q, B, out, (const PmSlot*)nullptr, 0);
  prof_end("k_is_valid64", s);
  return e;
}
cudaError_t launch_is_valid64_update(const PmTablesHdr* T, const PmTablesHdr& h, double* state, const PmSlot* recs, const double* q,
                                     int accurate, uint8_t* out, cudaStream_t s) {
  return team_launch(k_is_valid64<1, 4, true>, 2, 1, 4, h, s, T, state, q, (int64_t)1, out, recs, accurate);
}
cudaError_t launch_evaluate64(const PmTablesHdr* T, const PmTablesHdr& h, const double* state, const double* q, int64_t B,
                              int high_accuracy, double* vals, double* jac, cudaStream_t s) {
  if (B <= 0) return cudaSuccess;
  int n_sm = 0;
  const cudaError_t e = sm_count(&n_sm);
  if (e != cudaSuccess) return e;
  if (B <= 4 * (int64_t)n_sm) return team_launch(k_evaluate64<1>, B, 1, 2, h, s, T, state, q, B, high_accuracy, vals, jac);
  return team_launch(k_evaluate64<4>, (B + 3) / 4, 4, 2, h, s, T, state, q, B, high_accuracy, vals, jac);
}
cudaError_t launch_sphere_dist64(const PmTablesHdr* T, const PmTablesHdr& h, const double* state, const double* q, int64_t B,
                                 int high_accuracy, double* dist, double* centres, cudaStream_t s) {
  if (B <= 0 || h.n_spheres <= 0) return cudaSuccess;
  k_sphere_centres64<<<grid_for(B, 128), 128, 0, s>>>(T, state, q, B, high_accuracy, centres);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess || !dist) return e;
  const int64_t n = B * h.n_spheres;
  const bool prims = h.n_prims > h.n_clouds || h.n_clouds == 0;
  if (prims) k_sphere_sdf64<false><<<grid_for(n, 128), 128, 0, s>>>(T, centres, n, false, dist);
  if (h.n_clouds > 0) k_sphere_sdf64<true><<<grid_for(n, 8), 256, 0, s>>>(T, centres, n, prims, dist);
  return cudaGetLastError();
}
cudaError_t launch_spheres_of_state(const PmTablesHdr* T, const double* state, int groups, double* out4, cudaStream_t s) {
  k_spheres_of_state<<<1, 1, 0, s>>>(T, state, groups, out4);
  return cudaGetLastError();
}
cudaError_t launch_check_motion64(const PmTablesHdr* T, const PmTablesHdr& h, const double* state, const double* s1,
                                  const double* s2, int64_t E, int type, const double* width, double resolution, const int16_t* seq,
                                  uint8_t* out, unsigned long long* n_checked, unsigned long long* counts, cudaStream_t s) {
  if (E <= 0) return cudaSuccess;
  int n_sm = 0;
  cudaError_t e = sm_count(&n_sm);
  if (e != cudaSuccess) return e;
  if (E <= n_sm)
    return team_launch(k_check_motion64<16>, E, 16, 1, h, s, T, state, s1, s2, type, width, resolution, seq, out, n_checked, counts);
  // more edges a block while 8 blocks per SM (4 rounds of resident ones) are left; below two, the block an edge that
  // keeps its endpoints in shared memory (1,024 chain edges of 1 to 120 waypoints: 417 us, 432 with the other kernel)
  const int G = (int)std::min<int64_t>(std::max<int64_t>(E / (8 * (int64_t)n_sm), 1), kEdgesPerBlock);
  if (G == 1)
    return team_launch(k_check_motion64<8>, E, 8, 1, h, s, T, state, s1, s2, type, width, resolution, seq, out, n_checked, counts);
  return team_launch(k_check_motions64<8>, (E + G - 1) / G, 8, 1, h, s, T, state, s1, s2, E, G, type, width, resolution, seq, out, n_checked,
                     counts);
}
cudaError_t launch_sdf_points(const PmPrim* prims, int n_prims, const PmGridDev* clouds, int n_clouds, int is_union,
                              const double* pts, const double* radii, int64_t n, double* eval_out, uint8_t* outside_out, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  const bool others = n_prims > n_clouds || n_clouds == 0;
  if (others) k_sdf_points<false><<<grid_for(n, 128), 128, 0, s>>>(prims, n_prims, clouds, is_union, false, pts, radii, n, eval_out, outside_out);
  if (n_clouds > 0) k_sdf_points<true><<<grid_for(n, 8), 256, 0, s>>>(prims, n_prims, clouds, is_union, others, pts, radii, n, eval_out, outside_out);
  return cudaGetLastError();
}
cudaError_t launch_cloud_nearest(const PmGridDev* grid, const double* pts, int64_t n, double* sq, double* near3,
                                 cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  k_cloud_nearest<<<grid_for(n, 8), 256, 0, s>>>(grid, pts, n, sq, near3);
  return cudaGetLastError();
}

}  // namespace pmg
