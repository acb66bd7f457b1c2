// Host build of the MIXED form on each field layout (planes, row pairs, cells, four taps;
// snapshot-raytracer_gb300/csrc/srt_scheme.cuh, srt_adjoint.cuh) for
// tests/test_layouts_host.py. Fields are halo-padded float arrays (extents
// n + 3, voxel (i, j, k) at (i+1) + px ((j+1) + py (k+1))), in the order B_x,
// B_y, B_z, phi.
#include <vector>
#include "srt_adjoint.cuh"

namespace {

struct Layouts {
  srt::Geom G;
  srt::FieldPtrs F[6];  // by layout
  std::vector<float2> pair[4];
  std::vector<float4> cell[4];
  Layouts(const float* const* f, int n0, int n1, int n2) {
    const int n[3] = {n0, n1, n2};
    for (int i = 0; i < 3; ++i) {
      G.n[i] = n[i];
      G.invn[i] = 1.0f / (float)n[i];
    }
    const int px = n0 + 3, py = n1 + 3, pz = n2 + 3;
    G.px = px;
    G.pxy = (int64_t)px * py;
    G.pxy2 = (int64_t)px * (py - 1);
    for (auto& p : F) p = {};
    for (int c = 0; c < 4; ++c) {
      pair[c].resize((size_t)px * (py - 1) * pz);
      cell[c].resize((size_t)px * py * pz);
      for (int k = 0; k < pz; ++k)
        for (int j = 0; j < py; ++j)
          for (int i = 0; i < px; ++i) {
            // periodic neighbours, as the layout kernel takes them
            float v[3][3];
            for (int b = 0; b < 3; ++b)
              for (int a = 0; a < 3; ++a) {
                const int vi = ((i + a - 2) % n0 + n0) % n0, vj = ((j + b - 2) % n1 + n1) % n1;
                v[b][a] = f[c][(vi + 1) + px * ((vj + 1) + (int64_t)py * k)];
              }
            cell[c][i + px * (j + (size_t)py * k)] = srt::cell_of(v);
            if (j + 1 < py)
              pair[c][i + px * (j + (size_t)(py - 1) * k)] =
                  make_float2(f[c][i + px * (j + (int64_t)py * k)], f[c][i + px * (j + 1 + (int64_t)py * k)]);
          }
      F[srt::kPairs].pr[c] = pair[c].data();
      F[srt::kCells].cell[c] = cell[c].data();
    }
    F[srt::kPlanes].phi = f[3];
    for (int c = 0; c < 3; ++c) F[srt::kPlanes].b[c] = f[c];
    F[srt::kFourTaps] = F[srt::kFourPlanes] = F[srt::kPlanes];
    F[srt::kFourPairs] = F[srt::kPairs];
  }
};

template <int L>
void maps_of(const Layouts& Y, long long nside, long long count, int n_steps, float* maps, int* flagged) {
  for (long long r = 0; r < count; ++r) {
    float m[2];
    flagged[r] = srt::trace_ray_mixed<L>(Y.F[L], Y.G, srt::ray_dir_pix(nside, r), n_steps, maps + 6 * r, m);
  }
}

// One evaluation's vjp with the tap cotangents by cells (and, hot, in the copy
// of the region around the observer) or by rows of taps.
struct AccRows {
  float* g;
  SRT_HD bool active() const { return true; }
  SRT_HD void add_row(int64_t row, float a, float b, float c, float d) const {
    g[row] += a;
    g[row + 1] += b;
    g[row + 2] += c;
    g[row + 3] += d;
  }
};

}  // namespace

extern "C" {

void layout_maps(const float* const* f, int n0, int n1, int n2, long long nside, long long count, int n_steps,
                 float* maps, int* flagged) {
  const Layouts Y(f, n0, n1, n2);
  maps_of<srt::kPlanes>(Y, nside, count, n_steps, maps, flagged);
  maps_of<srt::kPairs>(Y, nside, count, n_steps, maps + 6 * count, flagged + count);
  maps_of<srt::kCells>(Y, nside, count, n_steps, maps + 12 * count, flagged + 2 * count);
  maps_of<srt::kFourTaps>(Y, nside, count, n_steps, maps + 18 * count, flagged + 3 * count);
  maps_of<srt::kFourPlanes>(Y, nside, count, n_steps, maps + 24 * count, flagged + 4 * count);
  maps_of<srt::kFourPairs>(Y, nside, count, n_steps, maps + 30 * count, flagged + 5 * count);
}

// Cotangents of `count` rays' right-hand side at affine parameter s[r] and
// perturbation state d[19 r ..] for the output cotangent fb: yb[layout][r][19],
// and the fields' cotangents rows[4][padded] (rows of taps, planes layout) and
// cells[4][padded x 4 floats] (cells layout) with copies[4][kHotSide^3 x 4] for
// the footprints in the region around the observer (hot != 0).
void layout_vjp(const float* const* f, int n0, int n1, int n2, int count, const double* theta, const double* phi,
                const float* s, const float* d, const float* fb, float* yb, float* rows, float* cells, float* copies,
                int hot) {
  const Layouts Y(f, n0, n1, n2);
  const int64_t pvox = Y.G.pxy * (n2 + 3);
  const int64_t region = (int64_t)srt::kHotSide * srt::kHotSide * srt::kHotSide;
  AccRows ar[4];
  srt::AccF32 ac[4];
  std::vector<std::vector<float4>> grid(4, std::vector<float4>((size_t)(pvox + region), make_float4(0, 0, 0, 0)));
  for (int c = 0; c < 4; ++c) {
    ar[c].g = rows + c * pvox;
    ac[c].g = grid[c].data();
    ac[c].hot = hot ? pvox : 0;
  }
  float x0[3];
  srt::mixed_observer(Y.G, x0);
  for (int r = 0; r < count; ++r) {
    srt::MixedRay R;
    float y[srt::kMixedState];
    srt::init_mixed(srt::ray_dir(theta[r], phi[r]), R, y);
    srt::StageView<float> V;
    srt::stage_view_mixed(d + 19 * r, s[r], R, Y.G, x0, V);
    srt::rhs_vjp<float, AccRows, AccRows, srt::kPlanes>(V, Y.F[srt::kPlanes], Y.G, fb, yb + 19 * r, ar, ar[3]);
    float* y1 = yb + 19 * (count + r);
    srt::rhs_vjp<float, srt::AccF32, srt::AccF32, srt::kCells>(V, Y.F[srt::kCells], Y.G, fb, y1, ac, ac[3]);
    float* y2 = yb + 19 * (2 * count + r);
    srt::AccNone none[3];
    srt::AccF32 off{nullptr};
    srt::rhs_vjp<float, srt::AccNone, srt::AccF32, srt::kPairs>(V, Y.F[srt::kPairs], Y.G, fb, y2, none, off);
  }
  for (int c = 0; c < 4; ++c)
    for (int64_t q = 0; q < pvox + region; ++q) {
      float* o = q < pvox ? cells + 4 * (c * pvox + q) : copies + 4 * (c * region + q - pvox);
      o[0] = grid[c][q].x, o[1] = grid[c][q].y, o[2] = grid[c][q].z, o[3] = grid[c][q].w;
    }
}

// The scatter of two stages in one cell (padded index base) at offsets ta, tb with
// cotangents qa, qb, into cells[padded x 4]; and the same by the two stages' own
// passes over field f, into apart[padded x 4].
void scatter_pair(const float* f, int n0, int n1, int n2, long long base, const float* ta, const float* qa,
                  const float* tb, const float* qb, float* cells, float* apart) {
  const float* const four[4] = {f, f, f, f};
  const Layouts Y(four, n0, n1, n2);
  srt::AccF32 two{(float4*)cells}, one{(float4*)apart};
  srt::scatter_two(two, base, -1, Y.G, ta, qa, tb, qb);
  for (int k = 0; k < 2; ++k) {
    srt::Tri<float> Q;
    float xb[3] = {0, 0, 0};
    srt::tricubic_vjp_mixed<1, srt::AccF32>(srt::cell_source<srt::kPlanes>(Y.F[srt::kPlanes], Y.G, 0, base, 0), base, -1,
                                            Y.G, k ? tb : ta, k ? qb : qa, Q, xb, one);
  }
}

int hot_side() { return srt::kHotSide; }
}
