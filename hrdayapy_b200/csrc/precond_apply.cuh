// What the flexible CG needs of the preconditioner: the point-wise part of
//   z = M(r) = omega D^-1 r + s y[parent] + zc[aggregate],
// so that its passes can form z where they use it instead of storing it, and
// the coarse solve from sums of r over line segments, which the r update
// takes while r is in registers.
#pragma once
#include "hp_common.cuh"

struct HpPrecond;

namespace hp {
namespace pc {

struct ZArgs {
  float omega;
  const float* zbox;   // coarse correction per aggregate box (0 without a coarse level)
  int sh, nbj, nbk;    // aggregate edge 2^sh, boxes along j and k
  const float* y;      // network output (half grid), or null
  const float* scale;  // y's scale (scale[2])
  int H, W;            // half grid along j and k
};

// z at an unknown cell with unpadded coordinates (i, j, k), in the order and
// rounding of prolong_kernel.
__device__ __forceinline__ float z_value(const ZArgs& z, float inv, float r, int i, int j, int k) {
  const float t = __fmul_rn(z.omega, inv);
  const float zc =
      z.zbox ? z.zbox[((i >> z.sh) * z.nbj + (j >> z.sh)) * z.nbk + (k >> z.sh)] : 0.0f;
  if (!z.y) return __fmaf_rn(t, r, zc);
  const float sy =
      __fmul_rn(z.scale[2], z.y[((int64_t)(i >> 1) * z.H + (j >> 1)) * z.W + (k >> 1)]);
  const float v = __fmaf_rn(t, r, sy);
  return __fadd_rn(v, zc);
}

// Segments of the r update: seg[(i nj + j) n_seg + k / len] is the sum of r
// over len consecutive cells of a line.  Null without a coarse level, and for
// aggregates of an edge below SEG_MIN: the r update sums four lanes before it
// looks at len, and the sums would take as many bytes as r itself.  There r is
// summed per aggregate by a pass of its own.
constexpr int SEG_MIN = 4;
struct SegArgs {
  double* seg;
  int len, n_seg, nj;
};

SegArgs precond_segments(const HpPrecond* h);
ZArgs precond_z(const HpPrecond* h, int use_net);
// zbox = A_c^-1 Q^T r from the segment sums (from r where there are none), then
// the network on r (use_net).
hp_status precond_update(HpPrecond* h, const uint8_t* label, const float* invd, const float* r,
                         int use_net, cudaStream_t s);
// The same from r itself (a residual that no r update has summed).
hp_status precond_begin(HpPrecond* h, const uint8_t* label, const float* invd, const float* r,
                        int use_net, cudaStream_t s);
uint64_t precond_serial(const HpPrecond* h);

}  // namespace pc
}  // namespace hp
