// rpd_clip_box.cuh -- the box and radius by which the thread-per-cell clipper
// (rpd_clip_thread.cu) passes over list entries.
#pragma once

#include <cuda_runtime.h>

#include <cmath>

namespace rpd {

// mid and half extent of a box around a cell's vertices (about the tet's
// centroid), and a bound of their distance to the seed
struct CullBox {
  float3 mid, half;
  float R;
};

// Fits b to vertices within [lo, hi] and r of the seed, with `slack` around
// them; true if some of them were outside b.  A group of entries is passed over
// by the box it met, and clips follow for those left of it: as long as they
// leave every vertex in that box, what was passed over stays so.  The fitted box
// is therefore kept inside b (the slack is for the vertices the next clips
// make, not to be gained anew by each of them), to the rounding of mid and half
// (2 u of the extent a clip; the test of an entry allows for 40).  With vertices
// outside b nothing of it counts any more and the group is looked over again.
__host__ __device__ __forceinline__ bool fit_box(CullBox& b, float3 lo, float3 hi, float r,
                                                 float slack) {
  const float3 bl = make_float3(b.mid.x - b.half.x, b.mid.y - b.half.y, b.mid.z - b.half.z);
  const float3 bh = make_float3(b.mid.x + b.half.x, b.mid.y + b.half.y, b.mid.z + b.half.z);
  const bool outside = lo.x < bl.x || hi.x > bh.x || lo.y < bl.y || hi.y > bh.y || lo.z < bl.z ||
                       hi.z > bh.z || r > b.R;
  lo = make_float3(lo.x - slack, lo.y - slack, lo.z - slack);
  hi = make_float3(hi.x + slack, hi.y + slack, hi.z + slack);
  r += slack;
  if (!outside) {
    lo = make_float3(fmaxf(lo.x, bl.x), fmaxf(lo.y, bl.y), fmaxf(lo.z, bl.z));
    hi = make_float3(fminf(hi.x, bh.x), fminf(hi.y, bh.y), fminf(hi.z, bh.z));
    r = fminf(r, b.R);
  }
  b.mid = make_float3(0.5f * (lo.x + hi.x), 0.5f * (lo.y + hi.y), 0.5f * (lo.z + hi.z));
  b.half = make_float3(0.5f * (hi.x - lo.x), 0.5f * (hi.y - lo.y), 0.5f * (hi.z - lo.z));
  b.R = r;
  return outside;
}

}  // namespace rpd
