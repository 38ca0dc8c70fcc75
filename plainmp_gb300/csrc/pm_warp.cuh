// Warp-cooperative searches of the point-cloud grid that several kernels share: the field's starting
// candidate of a query and the exact FP64 nearest neighbour.  Every lane of the warp calls them with the
// same query.
#pragma once
#include "pm_sdf.cuh"

namespace pmd {

__device__ __forceinline__ unsigned long long nn_key(float d2, int idx) {
  return ((unsigned long long)__float_as_uint(d2) << 32) | (unsigned)idx;
}

// Starting candidate of a warp search, in two steps so that the loads can be issued early: the field
// record (nearest point and index) of one of the 8 fine-cell centres around q on lanes 0-7 (index -1
// elsewhere and outside the grid), and q's own cell-list range on lane 8 (int bits in x, y; -1 none);
// then the best of the 8 shared by the warp ((INFINITY, -1) if none) and the list range.
// sub: the lane's position in its query's group of lanes (the lane itself for a whole warp; 0-15 for
// a half warp).
__device__ __forceinline__ float4 field_corner_record(const PmGridDev& G, float qx, float qy, float qz, int sub) {
  const int lane = sub;
  float4 rec = make_float4(__int_as_float(-1), __int_as_float(-1), 0.f, __int_as_float(-1));
  if (lane < 8 && G.n_points > 0) {
    const float inv = G.inv_cell32;
    const float qa[3] = {qx, qy, qz};
    const int nc[3] = {G.nbx * PM_GRID_B, G.nby * PM_GRID_B, G.nbz * PM_GRID_B};
    int cc[3];
    bool ok = true;
    for (int a = 0; a < 3; a++) {
      const float t = floorf((qa[a] - G.o32[a]) * inv - 0.5f) + (float)((lane >> a) & 1);
      ok = ok && t >= 0.f && t <= (float)(nc[a] - 1);
      cc[a] = ok ? (int)t : 0;
    }
    if (ok) rec = __ldg(G.cell_np + cc[0] + nc[0] * (cc[1] + (int64_t)nc[1] * cc[2]));
  } else if (lane == 8 && G.n_points > 0) {
    int2 rng;
    if (cell_list_of(G, qx, qy, qz, rng)) rec = make_float4(__int_as_float(rng.x), __int_as_float(rng.y), 0.f, __int_as_float(-1));
  }
  return rec;
}
struct FieldStart {
  NNResult32 nn;  // the best of the 8 corner records
  int2 rng;       // q's cell-list range (-1: none)
};
// width: 32 (one query per warp) or 16 (one per half warp; every lane calls it).
__device__ __forceinline__ FieldStart field_corner_candidate(const float4& rec, float qx, float qy, float qz, int width = 32) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & (width - 1);
  const int idx = __float_as_int(rec.w);
  unsigned long long key = ~0ull;
  if (lane < 8 && idx >= 0) {  // the FP32 expression of every walk (point_d2_32)
    const float dx = rec.x - qx, dy = rec.y - qy, dz = rec.z - qz;
    key = nn_key(fmaf(dx, dx, fmaf(dy, dy, dz * dz)), idx);
  }
  for (int o = 4; o > 0; o >>= 1) {
    const unsigned long long k2 = __shfl_xor_sync(FULL, key, o);
    key = k2 < key ? k2 : key;
  }
  key = __shfl_sync(FULL, key, 0, width);
  const int rx = __shfl_sync(FULL, __float_as_int(rec.x), 8, width), ry = __shfl_sync(FULL, __float_as_int(rec.y), 8, width);
  FieldStart f{{INFINITY, -1}, make_int2(rx, ry)};
  if (key != ~0ull) {
    f.nn.d2 = __uint_as_float((unsigned)(key >> 32));
    f.nn.idx = (int)(unsigned)(key & 0xffffffffu);
  }
  return f;
}

// Warp-cooperative exact FP64 nearest neighbour below maxd2: the minimum over points of
// fl(dx*dx + (dy*dy + dz*dz)) in FP64, as grid_nearest64 (among equal values the smallest sorted index).
//
// An FP64 warp instruction costs the same however few lanes take part and GB300 issues about 20 G of them
// a second, so the search runs in FP32 and FP64 sees only points that FP32 cannot tell apart from the
// nearest one.  A box or point is skipped when its FP32 squared distance exceeds thr(d2) of a point known
// to the warp: thr adds the FP32 error of both distances (2.5 tabs, tabs = 4e-7 (|q|_1 + |p|_1 max), and
// 1e-5 relative; the rounding of the points, of q and of the distance arithmetic stays below 1.5e-7 of
// the same magnitudes), so the skipped point's FP64 distance is larger.  A lane keeps one candidate
// unevaluated; one surely nearer replaces it, one that is neither surely nearer nor surely farther gets
// its FP64 distance at once (coincident and equidistant points), and the candidates that the warp's
// final threshold leaves are evaluated together at the end.  One FP64 distance per query then remains,
// against every box and point of the walk: 100,000 uniform queries in a 2.5 m cube around the 200k-point
// cloud took 26.1 ms with one thread per query in FP64 (the FP64 pipe 82 % busy with 3.3 of 32 lanes),
// and take 0.36 ms this way.
//
// Where q's fine cell has a cell list, the list is scanned, nearest first, 32 entries at a time.
// Elsewhere the super-block with the nearest box is searched first, then those within the threshold.
// hint: a point index whose distance starts the search (e.g. the FP32 nearest point), or -1.
//
// STEPS = 3: the squared distances of q + h e_x, q + h e_y, q + h e_z, h = 1e-6 (the forward differences of a
// gradient), in one search: a point that FP32 rules out for q by 2h more is ruled out for all three, and the
// points that are left get three FP64 distances.  d3 receives them; maxd2 must be INFINITY.
constexpr double kStep = 1e-6;
template <int STEPS = 0>
__device__ inline NNResult64 warp_nearest64(const PmGridDev& G, const D3& q, double maxd2 = INFINITY, int hint = -1, double* d3 = nullptr) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  NNResult64 r{maxd2, -1};
  if (G.n_points <= 0 || !(maxd2 > 0.0) || !isfinite(q.x) || !isfinite(q.y) || !isfinite(q.z)) return r;  // as grid_nearest64
  const float qx = (float)q.x, qy = (float)q.y, qz = (float)q.z;
  float pmax = 0.f;
  for (int a = 0; a < 3; a++) pmax += fmaxf(fabsf(G.box_lo32[a]), fabsf(G.box_hi32[a]));
  const float mag = fabsf(qx) + fabsf(qy) + fabsf(qz) + pmax;
  if (!(mag < 1e15f)) {  // FP32 squares would overflow: the FP64 walk, one lane's result for all
    r = grid_nearest64(G, q, maxd2);
    for (int i = 0; i < STEPS; i++) d3[i] = grid_nearest64(G, D3{i == 0 ? q.x + kStep : q.x, i == 1 ? q.y + kStep : q.y, i == 2 ? q.z + kStep : q.z}).d2;
    return r;
  }
  const float tabs = 4e-7f * mag + (STEPS ? 1e-6f : 1e-12f);  // 2.5 tabs >= 2h
  auto thr = [&](float d2) {
    const float sb = sqrtf(d2) * (1.0f + 1e-5f) + 2.5f * tabs;
    return sb * sb * (1.0f + 1e-6f);
  };
  double best = maxd2;  // the lane's smallest evaluated FP64 distance, and its point
  int bidx = -1;
  float c32 = INFINITY;  // the lane's unevaluated candidate
  int cand = -1;
  float t = thr((float)maxd2);
  double b3[STEPS > 0 ? STEPS : 1];
  for (int i = 0; i < STEPS; i++) b3[i] = INFINITY;
  auto exact = [&](int p) {
    const double px = G.px[p], py = G.py[p], pz = G.pz[p];
    for (int i = 0; i < STEPS; i++) {
      const D3 d{px - (i == 0 ? q.x + kStep : q.x), py - (i == 1 ? q.y + kStep : q.y), pz - (i == 2 ? q.z + kStep : q.z)};
      const double d2 = d.x * d.x + (d.y * d.y + d.z * d.z);
      if (d2 < b3[i]) b3[i] = d2;
    }
    if (STEPS > 0) return;
    const D3 d{px - q.x, py - q.y, pz - q.z};
    const double d2 = d.x * d.x + (d.y * d.y + d.z * d.z);
    if (d2 < best || (d2 == best && bidx >= 0 && p < bidx)) {
      best = d2;
      bidx = p;
    }
  };
  auto offer = [&](float d2, int p) {
    if (d2 > t) return;
    const float l = thr(d2);
    t = fminf(t, l);
    if (cand < 0 || l < c32) {
      c32 = d2;
      cand = p;
    } else {
      exact(p);
    }
  };
  auto offer_point = [&](int p) {
    const float4 pt = __ldg(G.p32 + p);
    const float dx = pt.x - qx, dy = pt.y - qy, dz = pt.z - qz;
    offer(fmaf(dx, dx, fmaf(dy, dy, dz * dz)), p);
  };
  auto share = [&]() { t = __uint_as_float(__reduce_min_sync(FULL, __float_as_uint(t))); };  // t >= 0: its bits order like it
  auto box2 = [&](const float4& lo, const float4& hi) {
    const float gx = gap32(qx, lo.x, hi.x), gy = gap32(qy, lo.y, hi.y), gz = gap32(qz, lo.z, hi.z);
    return fmaf(gx, gx, fmaf(gy, gy, gz * gz));
  };
  // start: the nearest points of the 8 fine-cell centres around q (one lane each), and the hint
  const float4 rec = field_corner_record(G, qx, qy, qz, lane);
  const int2 rng = make_int2(__shfl_sync(FULL, __float_as_int(rec.x), 8), __shfl_sync(FULL, __float_as_int(rec.y), 8));
  if (lane < 8) {
    const int p = __float_as_int(rec.w);
    const float dx = rec.x - qx, dy = rec.y - qy, dz = rec.z - qz;
    if (p >= 0) offer(fmaf(dx, dx, fmaf(dy, dy, dz * dz)), p);
  } else if (lane == 8 && hint >= 0 && hint < G.n_points) {
    offer_point(hint);
  }
  share();
  if (rng.x >= 0) {
    const float unit = G.cell32 * (1.0f / (float)PM_CL_UNITS);
    for (int base = rng.x; base < rng.y; base += 32) {  // warp-uniform
      const int k = base + lane;
      bool beyond = true;  // this entry, and (sorted) every later one, lies beyond the threshold
      int2 pr = make_int2(0, 0);
      if (k < rng.y) {
        const uint32_t e = __ldg(G.cl_ent + k);
        const float lbd = (float)(e >> 24) * unit;
        beyond = lbd * lbd * (1.0f - 1e-5f) > t;
        if (!beyond) {
          const int o = (int)(e & 0xffffffu);
          const float4 lo = __ldg(G.cell_rec + 2 * o), hi = __ldg(G.cell_rec + 2 * o + 1);
          if (!(box2(lo, hi) > t)) pr = make_int2(__float_as_int(lo.w), __float_as_int(hi.w));
        }
      }
      const bool stop = __shfl_sync(FULL, beyond ? 1 : 0, 31) != 0;
      // the points of the surviving cells, spread over the lanes (a warp scan of their counts)
      const int n = pr.y - pr.x;
      int incl = n;
      for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(FULL, incl, o);
        if (lane >= o) incl += u;
      }
      const int total = __shfl_sync(FULL, incl, 31);
      for (int t0 = 0; t0 < total; t0 += 32) {  // warp-uniform
        const int u = t0 + lane;
        int lo = 0, hi = 31;  // owner: the first lane whose inclusive count exceeds u
        for (int it = 0; it < 5; it++) {
          const int mid = (lo + hi) >> 1;
          if (__shfl_sync(FULL, incl, mid) <= u) lo = mid + 1;
          else hi = mid;
        }
        const int first = __shfl_sync(FULL, pr.x, lo), excl = __shfl_sync(FULL, incl - n, lo);
        if (u < total) offer_point(first + (u - excl));
      }
      share();
      if (stop) break;
    }
  } else {
    // one super-block: its occupied blocks nearest first, each block's cells over the lanes
    auto visit = [&](int b0, int b1) {
      for (int base = b0; base < b1; base += 32) {  // warp-uniform
        const int k = base + lane;
        float lb = INFINITY;
        int2 occ = make_int2(0, 0);
        if (k < b1) {
          const float4 lo = __ldg(G.sb_blk + 2 * k), hi = __ldg(G.sb_blk + 2 * k + 1);
          occ = make_int2(__float_as_int(lo.w), __float_as_int(hi.w));
          lb = box2(lo, hi);
        }
        for (;;) {  // warp-uniform: the nearest block left
          const unsigned m = __reduce_min_sync(FULL, __float_as_uint(lb));
          const unsigned who = __ballot_sync(FULL, __float_as_uint(lb) == m);
          if (!(__uint_as_float(m) <= t) || m == 0x7f800000u) break;
          const int src = __ffs(who) - 1;
          const int c0 = __shfl_sync(FULL, occ.x, src), c1 = __shfl_sync(FULL, occ.y, src);
          if (lane == src) lb = INFINITY;
          for (int c = c0 + lane; c < c1; c += 32) {
            const float4 lo = __ldg(G.cell_rec + 2 * (int64_t)c), hi = __ldg(G.cell_rec + 2 * (int64_t)c + 1);
            if (box2(lo, hi) > t) continue;
            for (int p = __float_as_int(lo.w); p < __float_as_int(hi.w); p++) offer_point(p);
          }
          __syncwarp();
          share();
        }
      }
    };
    float lb0 = INFINITY;
    int j0 = -1;
    int2 r0 = make_int2(0, 0);
    for (int j = lane; j < G.n_sb; j += 32) {
      const float4 lo = __ldg(G.sb_rec + 2 * j), hi = __ldg(G.sb_rec + 2 * j + 1);
      const float lb = box2(lo, hi);
      if (lb < lb0) {
        lb0 = lb;
        j0 = j;
        r0 = make_int2(__float_as_int(lo.w), __float_as_int(hi.w));
      }
    }
    const unsigned m = __reduce_min_sync(FULL, __float_as_uint(lb0));
    const int who = __ffs(__ballot_sync(FULL, __float_as_uint(lb0) == m)) - 1;
    j0 = __shfl_sync(FULL, j0, who);
    const int f0 = __shfl_sync(FULL, r0.x, who), f1 = __shfl_sync(FULL, r0.y, who);
    if (j0 >= 0 && __uint_as_float(m) <= t) {
      visit(f0, f1);
      for (int base = 0; base < G.n_sb; base += 32) {  // warp-uniform
        const int j = base + lane;
        float lb = INFINITY;
        int2 br = make_int2(0, 0);
        if (j < G.n_sb && j != j0) {
          const float4 lo = __ldg(G.sb_rec + 2 * j), hi = __ldg(G.sb_rec + 2 * j + 1);
          lb = box2(lo, hi);
          br = make_int2(__float_as_int(lo.w), __float_as_int(hi.w));
        }
        for (unsigned bal = __ballot_sync(FULL, lb <= t && lb < INFINITY); bal != 0; bal &= bal - 1) {
          const int src = __ffs(bal) - 1;
          const float l = __shfl_sync(FULL, lb, src);
          const int b0 = __shfl_sync(FULL, br.x, src), b1 = __shfl_sync(FULL, br.y, src);
          if (l <= t) visit(b0, b1);  // t is the warp's
        }
      }
    }
  }
  if (cand >= 0 && !(c32 > t)) exact(cand);
  __syncwarp();
  // the warp's minima: values >= 0, so their words order like them
  auto least = [&](double d, unsigned& hi, unsigned& lo) {
    hi = __reduce_min_sync(FULL, (unsigned)__double2hiint(d));
    lo = __reduce_min_sync(FULL, (unsigned)__double2hiint(d) == hi ? (unsigned)__double2loint(d) : 0xffffffffu);
    return __hiloint2double((int)hi, (int)lo);
  };
  unsigned mh, ml;
  if (STEPS > 0) {
    for (int i = 0; i < STEPS; i++) d3[i] = least(b3[i], mh, ml);
    return r;
  }
  r.d2 = least(best, mh, ml);
  r.idx = (int)__reduce_min_sync(FULL, (unsigned)__double2hiint(best) == mh && (unsigned)__double2loint(best) == ml ? (unsigned)bidx : 0xffffffffu);
  return r;
}

// is_outside(p, r) of a point cloud (primitive_sdf.hpp:597-603) with the warp search: only
// whether a point lies within r + radius matters (see prim_outside).  Warp-uniform arguments.
__device__ __forceinline__ bool cloud_outside_warp(const PmPrim& P, const PmGridDev* clouds, const D3& p, double r, int* near,
                                                   int hint = -1) {
  const double reach = (r + P.a) * (1.0 + 1e-12) + 1e-12;
  const NNResult64 nn = warp_nearest64(clouds[P.cloud], p, reach * reach, hint);
  if (near) *near = nn.idx;
  if (nn.idx < 0) return true;
  return sqrt(nn.d2) - P.a > r;
}

// prim_eval of a point cloud with the warp search.  Warp-uniform arguments; every lane gets the value.
__device__ __forceinline__ double cloud_eval_warp(const PmPrim& P, const PmGridDev* clouds, const D3& p) {
  return sqrt(warp_nearest64(clouds[P.cloud], p).d2) - P.a;
}

}  // namespace pmd
