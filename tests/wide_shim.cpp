// Host build of the warp-per-ray right-hand side (snapshot-raytracer_gb300/csrc/
// srt_wide.cuh), its lanes run one after another phase by phase, beside the
// one-lane FP64 form (srt_scheme.cuh), for tests/test_wide_host.py.
#include <vector>
#include "srt_wide.cuh"

namespace {

// n_steps RK4 steps of the state y (19 components) by one emulated warp.
template <typename R>
void wide_trace(double* y, const srt::FieldPtrs& F, const srt::Geom& G, int n_steps) {
  const srt::WideTables tables = srt::make_wide_tables();
  std::vector<R> scratch(srt::kWsSize);
  R* S = scratch.data();
  int cell[6];
  srt::WideLane<R> L[32];
  for (int l = 0; l < 32; ++l) {
    L[l].start(l, tables);
    L[l].constants(S);
    if (l < 19) L[l].y = R(y[l]);
  }
  for (int step = 0; step < n_steps; ++step)
    for (int st = 0; st < 4; ++st) {
      for (auto& l : L) l.stage(S, st);
      for (auto& l : L) l.position(S, cell, G);
      for (auto& l : L) l.load_taps(cell, F, G);
      for (auto& l : L) l.weights(S);
      for (auto& l : L) l.frame(S);
      for (auto& l : L) l.x_pass(S);
      for (auto& l : L) l.y_pass(S);
      for (auto& l : L) l.z_pass(S);
      for (auto& l : L) l.round1(S);
      for (auto& l : L) l.round2(S);
      for (auto& l : L) l.round3(S);
      for (auto& l : L) l.round4(S);
      for (auto& l : L) l.round5(S);
      for (auto& l : L) l.round6(S, st);
    }
  for (int l = 0; l < 19; ++l) y[l] = (double)L[l].y;
}

// The same by an emulated block of five warps (FP64).
void block_trace(double* y, const srt::FieldPtrs& F, const srt::Geom& G, int n_steps) {
  const srt::WideTables tables = srt::make_wide_tables();
  std::vector<double> scratch(srt::kWsBlockSize);
  double* S = scratch.data();
  int cell[12];
  srt::WideLane<double> L[32];
  srt::FieldLane<double> I[4][32];
  for (int l = 0; l < 32; ++l) {
    L[l].start(l, tables);
    L[l].constants(S);
    if (l < 19) L[l].y = y[l];
    for (int f = 0; f < 4; ++f) I[f][l].start(l, f);
  }
  for (int step = 0; step < n_steps; ++step)
    for (int st = 0; st < 4; ++st) {
      for (auto& l : L) l.stage(S, st);
      for (auto& w : I) {
        for (auto& l : w) l.position(S, cell, G);
        for (auto& l : w) l.load_taps(cell, F, G);
        for (auto& l : w) l.weights(S);
        for (auto& l : w) l.x_pass(S);
        for (auto& l : w) l.y_pass(S);
        for (auto& l : w) l.z_pass(S);
      }
      for (auto& l : L) l.frame(S);
      for (auto& l : L) l.round1(S);
      for (auto& l : L) l.round2(S);
      for (auto& l : L) l.round3(S);
      for (auto& l : L) l.round4(S);
      for (auto& l : L) l.round5(S);
      for (auto& l : L) l.round6(S, st);
    }
  for (int l = 0; l < 19; ++l) y[l] = L[l].y;
}

}  // namespace

// The state of RING pixels [begin, begin + count) after n_steps: one[19 r ..]
// by the one-lane FP64 form, wide and dd by the emulated warp in FP64 and in
// double-float, block by the emulated block of five warps.
extern "C" void trace_states(const float* phi, const float* bx, const float* by, const float* bz, int n0, int n1, int n2,
                             long long nside, long long begin, long long count, int n_steps, double* one, double* wide,
                             double* ddf, double* block) {
  srt::Geom G;
  const int n[3] = {n0, n1, n2};
  for (int i = 0; i < 3; ++i) {
    G.n[i] = n[i];
    G.invn[i] = 1.0f / (float)n[i];
  }
  G.px = n0 + 3;
  G.pxy = (int64_t)(n0 + 3) * (n1 + 3);
  G.pxy2 = (int64_t)(n0 + 3) * (n1 + 2);
  srt::FieldPtrs F = {};
  F.phi = phi;
  F.b[0] = bx;
  F.b[1] = by;
  F.b[2] = bz;
  for (long long r = 0; r < count; ++r) {
    double* y[4] = {one + 19 * r, wide + 19 * r, ddf + 19 * r, block + 19 * r};
    const srt::RayDir d = srt::ray_dir_pix(nside, begin + r);
    for (double* v : y) srt::init_std(d, G, v);
    for (int s = 0; s < n_steps; ++s) srt::step_std<srt::kFP64>(F, G, y[0], nullptr);
    wide_trace<double>(y[1], F, G, n_steps);
    wide_trace<srt::dd>(y[2], F, G, n_steps);
    block_trace(y[3], F, G, n_steps);
  }
}
