// One configuration per warp (or few warps) in FP64: the block's FK into shared memory, and the helpers of
// the checks that run on it (k_plain.cu).
//
// GB300 issues about 20 G FP64 warp instructions a second however few lanes take part.  A thread per
// configuration ran FK and every test at 2 to 7 active lanes, and a batch of a few hundred left most SMs
// idle.  Here a block's FK runs level by level over the slot tree, four lanes per (configuration, slot),
// one component each; the checks spread groups, primitives, spheres and pairs over lanes, clear what FP32
// clears for certain (pm_clear.cuh) and give FP64 what is left, a warp's worth at a time.  Every FP64 value
// comes from the operand pairs, signs and summation order of the reference (pm_math.cuh).
#pragma once
#include "pm_clear.cuh"
#include "pm_view.cuh"
#include "pm_warp.cuh"

namespace pmd {

constexpr int kRec = 8;    // doubles per slot: quaternion x y z w, translation, identity flag of the local transform
constexpr int kRec32 = 12; // floats per slot: the rows of (R, t)

// Poses of one configuration (kRec / kRec32 per slot).
struct TeamPose {
  const double* rec;
  const float* p32;
  __device__ __forceinline__ DPose at(int slot) const {
    const double* r = rec + (size_t)slot * kRec;
    return DPose{DQ{r[0], r[1], r[2], r[3]}, D3{r[4], r[5], r[6]}};
  }
  __device__ __forceinline__ const float* at32(int slot) const { return p32 + (size_t)slot * kRec32; }
  // a point of the slot's link frame in the world (create_group_sphere_position_cache's expression)
  __device__ __forceinline__ D3 point(int slot, const D3& rel) const {
    const DPose p = at(slot);
    return add(mv(qmat(p.q), rel), p.t);
  }
};

// The FP32 records of the tables' image in global memory.
struct Image {
  const PmSphereF* sph;
  const PmGroupF* grp;
  const PmPrimF* prm;
  __device__ explicit Image(const PmTablesHdr* T) {
    auto a16 = [](size_t x) { return (x + 15) & ~(size_t)15; };
    const char* p = pm_at<char>(T, T->off_img) + a16(sizeof(PmSlotF) * T->n_slots) + 32;
    sph = reinterpret_cast<const PmSphereF*>(p);
    p += a16(sizeof(PmSphereF) * T->n_spheres);
    grp = reinterpret_cast<const PmGroupF*>(p);
    p += a16(sizeof(PmGroupF) * T->n_groups);
    prm = reinterpret_cast<const PmPrimF*>(p);
  }
};

// Bound on the distance between the FP32 centre xf(p32, s) and the FP64 one, |s| = sn: the FP32 rounding of
// the quaternion (2u) moves R s by at most (8 * 2u + 24u) |s|, that of t by u |t|_1 (the rounding of R s + t
// itself is part of margin32).
__device__ __forceinline__ float cast_error(const float* P, float sn) {
  return kU * (64.0f * sn + 4.0f * (fabsf(P[3]) + fabsf(P[7]) + fabsf(P[11]))) + 1e-9f;
}

// FK of configurations 0 .. ncfg - 1 by NT threads (a block, or the one warp of a block: WARP) into rec
// [ncfg][n_slots][kRec]; qf(c, col) gives a joint or base value.  The pose of a slot replaces its local
// transform in place.  Poses are bit for bit those of fk64.
template <int NT, bool WARP, class QF>
__device__ void fk64_levels(const TView& v, const double* __restrict__ state, const QF& qf, int ncfg, bool taylor, double* rec) {
  const unsigned FULL = 0xffffffffu;
  const PmTablesHdr* T = v.T;
  const int tid = WARP ? threadIdx.x & 31 : threadIdx.x, nsl = T->n_slots, nc = T->n_ctrl;
  auto sync = [] {
    if (WARP) {
      __syncwarp();
    } else {
      __syncthreads();
    }
  };
  for (int t = tid; t < ncfg * nsl; t += NT) {
    const int c = t / nsl, i = t - c * nsl;
    const PmSlot& s = v.S[i];
    DPose p;
    bool lid = false;
    if (s.parent < 0) {
      if (T->base_type == PM_BASE_FIXED) {
        p = state_pose(state, PM_STATE_BASE_ROW, lid);
      } else if (T->base_type == PM_BASE_FLOATING) {
        p.t = D3{qf(c, nc), qf(c, nc + 1), qf(c, nc + 2)};
        p.q = quat_from_rpy(qf(c, nc + 3), qf(c, nc + 4), qf(c, nc + 5));
      } else {
        p.t = D3{qf(c, nc), qf(c, nc + 1), 0.0};
        p.q = quat_from_rpy(0, 0, qf(c, nc + 2));
      }
    } else if (s.mode == PM_FK_STATE) {
      p = state_pose(state, PM_STATE_LINK_ROW(s.link), lid);
    } else {
      joint_local(s, qf(c, s.qcol), taylor, p.q, p.t, lid);
    }
    double* r = rec + (size_t)t * kRec;
    r[0] = p.q.x;
    r[1] = p.q.y;
    r[2] = p.q.z;
    r[3] = p.q.w;
    r[4] = p.t.x;
    r[5] = p.t.y;
    r[6] = p.t.z;
    r[7] = lid ? 1.0 : 0.0;
  }
  // the levels (starts, then slot | parent << 16) in shared memory: two dependent loads a level otherwise
  __shared__ int32_t lev[2 * PM_MAX_SLOTS + 1];
  for (int i = tid; i < T->n_levels + 1 + nsl; i += NT) lev[i] = pm_at<int32_t>(T, T->off_lev)[i];
  const int32_t* order = lev + T->n_levels + 1;
  const int quad = tid >> 2, k = tid & 3, w0 = (tid >> 5) << 3;  // the lane's quad and component, the warp's first quad
  const int i1 = k == 0 ? 1 : (k == 1 ? 2 : 0), i2 = k == 0 ? 2 : (k == 1 ? 0 : 1);  // the cyclic next two of x y z
  sync();
  for (int l = 1; l < T->n_levels; l++) {
    const int s0 = lev[l], nl = lev[l + 1] - s0, tasks = ncfg * nl;
    for (int t0 = 0; t0 + w0 < tasks; t0 += NT / 4) {  // warp-uniform
      const bool on = t0 + quad < tasks;
      const int t = on ? t0 + quad : tasks - 1;
      const int c = t / nl, sp = order[s0 + t - c * nl];  // slot and parent, 16 bits each
      double* o = rec + ((size_t)c * nsl + (sp & 0xffff)) * kRec;
      const double* a = rec + ((size_t)c * nsl + (sp >> 16)) * kRec;
      // component k of qmul(a, o): x y z: aw o_k + a_k ow + a_i1 o_i2 - a_i2 o_i1;
      //                            w:     aw ow - ax ox - ay oy - az oz
      const bool w = k == 3;
      const double p1 = a[w ? 0 : k] * o[w ? 0 : 3], p2 = a[w ? 1 : i1] * o[w ? 1 : i2], p3 = a[w ? 2 : i2] * o[w ? 2 : i1];
      double q = ((a[3] * o[k] + neg_if(w, p1)) + neg_if(w, p2)) - p3;
      if (o[7] != 0.0) q = a[k];
      // component k < 3 of add(a.t, qrot(a, o.t)): uv = 2 cross(a, t); ((t + w uv) + cross(a, uv)) + a.t
      const int kk = w ? 0 : k;
      double uv = a[i1] * o[4 + i2] - a[i2] * o[4 + i1];
      uv = uv + uv;
      const double u1 = __shfl_sync(FULL, uv, i1, 4), u2 = __shfl_sync(FULL, uv, i2, 4);
      const double cr = a[i1] * u2 - a[i2] * u1;
      const double tr = a[4 + kk] + ((o[4 + kk] + a[3] * uv) + cr);
      __syncwarp();
      if (on) {
        o[k] = q;
        if (!w) o[4 + k] = tr;
      }
    }
    sync();
  }
}

// fk64_levels by a block of NT threads, and the poses in FP32 (p32 [ncfg][n_slots][kRec32]).
// The FP32 bounds (cast_error, margin32) are those of rotations, and so is that a group's sphere holds its spheres.
// A quaternion off unit norm (URDF axes and base poses are taken as they are given) scales: R stretches by up to
// 1 + 2 (|q|^2 - 1), or shrinks where |q| < 1.  Where |q|^2 exceeds `norm2` the FP32 translation is NaN, so that every
// FP32 comparison of the slot's spheres fails and FP64 decides.
// Validity needs the bounds alone, which have 1 % to spare (the Taylor form is within 1e-5 of unit norm a joint);
// evaluate also that the spheres leave the group's sphere by no more than the tables' stretch of its radius.
constexpr float kNorm2Valid = 1.01f;
constexpr float kNorm2Eval = 1.0011f;
template <int NT, class QF>
__device__ void fk64_block(const TView& v, const double* __restrict__ state, const QF& qf, int ncfg, bool taylor, float norm2, double* rec,
                           float* p32) {
  fk64_levels<NT, false>(v, state, qf, ncfg, taylor, rec);
  for (int t = threadIdx.x; t < ncfg * v.T->n_slots; t += NT) {
    const double* r = rec + (size_t)t * kRec;
    float* f = p32 + (size_t)t * kRec32;
    const float x = (float)r[0], y = (float)r[1], z = (float)r[2], w = (float)r[3];
    const float tx = 2.f * x, ty = 2.f * y, tz = 2.f * z;
    const bool scales = !(x * x + y * y + (z * z + w * w) <= norm2);
    float4* row = reinterpret_cast<float4*>(f);
    row[0] = make_float4(1.f - (ty * y + tz * z), ty * x - tz * w, tz * x + ty * w, scales ? NAN : (float)r[4]);
    row[1] = make_float4(ty * x + tz * w, 1.f - (tx * x + tz * z), tz * y - tx * w, scales ? NAN : (float)r[5]);
    row[2] = make_float4(tz * x - ty * w, tz * y + tx * w, 1.f - (tx * x + ty * y), scales ? NAN : (float)r[6]);
  }
  __syncthreads();
}

// Spreads items over the warp's lanes: lane l of the warp brings n_l >= 0 items; f(owner lane, index among
// the owner's items, have) runs for 32 of all items at a time on every lane (have: the lane got one; a lane
// past the end is given the last item, so that owner and index are valid on every lane).  f returns whether to
// go on (the same on every lane).
template <class F>
__device__ __forceinline__ void warp_spread(int n, const F& f) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  int incl = n;
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(FULL, incl, o);
    if (lane >= o) incl += u;
  }
  const int total = __shfl_sync(FULL, incl, 31);
  for (int t0 = 0; t0 < total; t0 += 32) {  // warp-uniform
    const int u = min(t0 + lane, total - 1);
    int lo = 0, hi = 31;  // owner: the first lane whose inclusive count exceeds u
    for (int it = 0; it < 5; it++) {
      const int mid = (lo + hi) >> 1;
      if (__shfl_sync(FULL, incl, mid) <= u) lo = mid + 1;
      else hi = mid;
    }
    const int excl = __shfl_sync(FULL, incl - n, lo);
    if (!f(lo, u - excl, t0 + lane < total)) return;
  }
}

__device__ __forceinline__ double shfl_d(double v, int src) { return __shfl_sync(0xffffffffu, v, src); }
__device__ __forceinline__ D3 shfl_d3(const D3& v, int src) { return D3{shfl_d(v.x, src), shfl_d(v.y, src), shfl_d(v.z, src)}; }

// Whether group g's gate for primitive P opens at the margin (0, or the cutoff of evaluate): the reference's
// outside_aabb and is_outside of the group sphere.  Not for point clouds.
__device__ __forceinline__ bool gate_open(const PmPrim& P, const D3& gc, double r) {
  return !outside_aabb(P, gc, r) && !prim_outside(P, nullptr, gc, r);
}

}  // namespace pmd
