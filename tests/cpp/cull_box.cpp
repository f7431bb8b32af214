// fit_box of rpd_clip_box.cuh for n vertex boxes in a row (7 floats each: lo,
// hi, r): outside[i], and the fitted boxes (lo, hi, R)
#include "../../libmat_gb300/csrc/rpd_clip_box.cuh"

extern "C" void fit_boxes(const float* v, int n, float slack, unsigned char* outside, float* out) {
  rpd::CullBox b;
  b.mid = make_float3(0.f, 0.f, 0.f);
  b.half = make_float3(INFINITY, INFINITY, INFINITY);
  b.R = INFINITY;
  for (int i = 0; i < n; ++i, v += 7, out += 7) {
    outside[i] = rpd::fit_box(b, make_float3(v[0], v[1], v[2]), make_float3(v[3], v[4], v[5]),
                              v[6], slack);
    const float o[7] = {b.mid.x - b.half.x, b.mid.y - b.half.y, b.mid.z - b.half.z,
                        b.mid.x + b.half.x, b.mid.y + b.half.y, b.mid.z + b.half.z, b.R};
    for (int k = 0; k < 7; ++k) out[k] = o[k];
  }
}
