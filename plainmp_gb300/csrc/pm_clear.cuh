// FP32 clearances of spheres against the primitives, with the margin inside which a decision is left to FP64.
#pragma once
#include "pm_grid.cuh"

namespace pmd {

constexpr float kU = 5.9604645e-8f;  // 2^-24
// Margin of an FP32 clearance: 64 units of roundoff of the magnitudes involved, plus 1 um.  The
// error analysis of the FP32 evaluation (pose rounding, one dot product, one square root)
// gives about 52 units for the box, the largest case.
__device__ __forceinline__ float margin32(float mag) { return 1e-6f + 64.0f * kU * (1.0f + mag); }

// A pose in FP32: the rows (R_i0 R_i1 R_i2 t_i) as float4 (P on a 16-byte boundary).
__device__ __forceinline__ float3 xf(const float* P, float x, float y, float z) {  // R v + t
  const float4* p = reinterpret_cast<const float4*>(P);
  const float4 a = p[0], b = p[1], c = p[2];
  return make_float3(fmaf(a.x, x, fmaf(a.y, y, fmaf(a.z, z, a.w))), fmaf(b.x, x, fmaf(b.y, y, fmaf(b.z, z, b.w))),
                     fmaf(c.x, x, fmaf(c.y, y, fmaf(c.z, z, c.w))));
}

// Clearance g (the reference reports a collision iff g <= 0, up to its own rounding), the
// evaluate()-based signed distance sd (minus r) and the magnitude for the margin.
__device__ __forceinline__ void clearance(const PmPrimF& P, const PmGridDev* clouds, float cx, float cy, float cz, float r, bool tiny,
                                          float extra, float& g, float& sd, float& mag) {
  const float dx = cx - P.pos[0], dy = cy - P.pos[1], dz = cz - P.pos[2];
  mag = fabsf(cx) + fabsf(cy) + fabsf(cz) + P.mag;
  switch (P.kind) {
    case PM_SDF_BOX: {
      float lx, ly, lz;
      if (P.aa) {
        lx = dx;
        ly = dy;
        lz = dz;
      } else {
        lx = fmaf(dx, P.rot[0], fmaf(dy, P.rot[3], dz * P.rot[6]));
        ly = fmaf(dx, P.rot[1], fmaf(dy, P.rot[4], dz * P.rot[7]));
        lz = fmaf(dx, P.rot[2], fmaf(dy, P.rot[5], dz * P.rot[8]));
      }
      const float sx = fabsf(lx) - P.a, sy = fabsf(ly) - P.b, sz = fabsf(lz) - P.c;
      const float mx = fmaxf(sx, 0.f), my = fmaxf(sy, 0.f), mz = fmaxf(sz, 0.f);
      const float ext = sqrtf(fmaf(mx, mx, fmaf(my, my, mz * mz)));
      const float ms = fmaxf(sx, fmaxf(sy, sz));
      g = tiny ? ms - r : ext - r;
      sd = ext + fminf(ms, 0.f) - r;
      return;
    }
    case PM_SDF_CYLINDER: {
      float lx, ly, lz;
      if (P.za) {
        lx = dx;
        ly = dy;
        lz = dz;
      } else {
        lx = fmaf(dx, P.rot[0], fmaf(dy, P.rot[3], dz * P.rot[6]));
        ly = fmaf(dx, P.rot[1], fmaf(dy, P.rot[4], dz * P.rot[7]));
        lz = fmaf(dx, P.rot[2], fmaf(dy, P.rot[5], dz * P.rot[8]));
      }
      const float zs = fabsf(lz) - P.c;
      const float rs = sqrtf(fmaf(lx, lx, ly * ly)) - P.a;
      const float a = fmaxf(rs, 0.f), b = fmaxf(zs, 0.f);
      const float ext = sqrtf(fmaf(a, a, b * b));
      g = tiny ? fmaxf(zs - r, rs) : ext - r;
      sd = ext + fminf(fmaxf(rs, zs), 0.f) - r;
      return;
    }
    case PM_SDF_SPHERE: {
      const float d = sqrtf(fmaf(dx, dx, fmaf(dy, dy, dz * dz))) - P.a;
      g = tiny ? d : d - r;
      sd = d - r;
      return;
    }
    case PM_SDF_GROUND: {  // the reference's AABB (z in [0, 0]) is part of its decision
      g = fmaxf(fabsf(cz) - r, cz + P.a - r);
      sd = cz + P.a - r;
      return;
    }
    case PM_SDF_CLOUD: {
      const float reach = P.a + r + extra;
      NNResult32 nn = grid_nearest32(clouds[P.cloud], cx, cy, cz, reach * reach);
      if (nn.idx < 0) {
        g = reach - P.a - r;  // nothing closer than reach
        sd = 3.0e38f;
        mag = fabsf(cx) + fabsf(cy) + fabsf(cz);
        return;
      }
      const float d = sqrtf(nn.d2);
      g = d - P.a - r;
      sd = g;
      mag = fabsf(cx) + fabsf(cy) + fabsf(cz) + d;
      return;
    }
  }
  g = 3.0e38f;
  sd = 3.0e38f;
}

}  // namespace pmd
