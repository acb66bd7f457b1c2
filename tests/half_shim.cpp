// Host build of the MIXED form on half cells (snapshot-raytracer_gb300/csrc/
// srt_scheme.cuh, kHalf) beside planes, for tests/test_half_cells_host.py. Fields are
// halo-padded float arrays in the order B_x, B_y, B_z, phi.
#include <vector>
#include "srt_adjoint.cuh"

namespace {

struct Half {
  srt::Geom G;
  srt::FieldPtrs planes = {}, half = {};
  std::vector<float2> data[4];
  Half(const float* const* f, int n0, int n1, int n2) {
    const int n[3] = {n0, n1, n2};
    for (int i = 0; i < 3; ++i) {
      G.n[i] = n[i];
      G.invn[i] = 1.0f / (float)n[i];
    }
    const int64_t px = n0 + 3, py = n1 + 3, rows = py - 1;
    G.px = px;
    G.pxy = px * py;
    G.pxy2 = px * rows;
    for (int c = 0; c < 4; ++c) {
      data[c].resize((size_t)(px * rows * (n2 + 3)));
      for (int64_t q = 0; q < (int64_t)data[c].size(); ++q) {
        const int64_t j = q / px % rows;
        const float* v = f[c] + q % px + px * (j + py * (q / (px * rows)));
        data[c][q] = make_float2(v[0], j > 0 ? srt::diff2(v[-px], v[0], v[px]) : NAN);  // row 0 is never read
      }
      half.pr[c] = data[c].data();
    }
    planes.phi = f[3];
    for (int c = 0; c < 3; ++c) planes.b[c] = f[c];
  }
};

}  // namespace

// Maps and guard flags of pixels [0, count) from planes (maps[0 ..], flagged[0 ..])
// and from half cells (the second halves); and for each pixel's direction the cotangent
// of one right-hand side at affine parameter s and state d for the cotangent fb.
extern "C" void half_compare(const float* const* f, int n0, int n1, int n2, long long nside, long long count, int n_steps,
                             float s, const float* d, const float* fb, float* maps, int* flagged, float* yb) {
  const Half H(f, n0, n1, n2);
  float x0[3];
  srt::mixed_observer(H.G, x0);
  const srt::AccNone none[3];
  for (long long r = 0; r < count; ++r) {
    const srt::RayDir dir = srt::ray_dir_pix(nside, r);
    float m[2];
    flagged[r] = srt::trace_ray_mixed<srt::kPlanes>(H.planes, H.G, dir, n_steps, maps + 6 * r, m);
    flagged[count + r] = srt::trace_ray_mixed<srt::kHalf>(H.half, H.G, dir, n_steps, maps + 6 * (count + r), m);
    srt::MixedRay R;
    float y[srt::kMixedState];
    srt::init_mixed(dir, R, y);
    srt::StageView<float> V;
    srt::stage_view_mixed(d, s, R, H.G, x0, V);
    srt::rhs_vjp<float, srt::AccNone, srt::AccNone, srt::kPlanes>(V, H.planes, H.G, fb, yb + 19 * r, none, none[0]);
    srt::rhs_vjp<float, srt::AccNone, srt::AccNone, srt::kHalf>(V, H.half, H.G, fb, yb + 19 * (count + r), none, none[0]);
  }
}
