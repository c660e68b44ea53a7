// The lattice passes' launchers on the stand-in CUDA runtime of runtime.cpp, on two devices.
// Prints one line per launch: device, pass, status.
#include <stdio.h>
#include <stdlib.h>

#include <vector>

#include "mb_ensemble_kernel.cuh"

extern int device;

namespace mb {
int mx_launch_step(const EnsParams &P, const MxStencil &S, int lat, int energy, cudaStream_t s, cudaEvent_t *ev,
                   double *out);
int ens_launch(const EnsParams &P, int grid, cudaStream_t s);
int ens_max_grid(int nsm);
} // namespace mb
using namespace mb;

// Both passes of a lattice of n^3 cells: planned (shell windows or split items by `items`) or by rows.
static void fp64(const char *name, int n_types, const char *items, bool planned) {
  setenv("MB_SPLIT_RHO_ITEMS", items, 1);
  setenv("MB_SPLIT_FORCE_ITEMS", items, 1);
  const double a0 = 2.855, cutoff = 5.6;
  Geom g{};
  g.bcx = g.by = g.bz = 8;
  g.gcx = g.gy = g.gz = 2;
  g.ecx = g.ey = g.ez = 12;
  g.E = 12 * 12 * 12;
  DevPot P{};
  P.n_types = n_types;
  P.nr = n_types == 1 ? 5000 : 2000;
  P.rdr = (P.nr - 1) / cutoff;
  P.cutoff = cutoff;
  std::vector<int64_t> even(512), odd(512);
  int n = 0, rx, ry, rz, near = 0;
  double dist[512];
  int rc = stencil_generate(a0, 6.3, 2 * g.ecx, g.ey, even.data(), odd.data(), 512, &n, &rx, &ry, &rz);
  if (rc == 0) rc = stencil_sort_by_distance(a0, cutoff, 2 * g.ecx, g.ey, even.data(), odd.data(), n, &near, dist);
  StencilSet st{};
  const int par[2] = {0, 1};
  if (rc == 0) rc = stencil_from_linear(even.data(), n, odd.data(), n, 2 * g.ecx, g.ey, g, par, &st);
  st.n_near = near;
  Plan64 plan{};
  if (rc == 0) plan.ok = plan64_shells(P, g, a0, cutoff, dist, st, plan.sh);
  if (rc || !plan.ok) exit(2);
  Lattice64 L{};
  double some = 0.0;
  L.rho = L.fx = L.fy = L.fz = &some;
  StepParams sp{};
  sp.rc2 = cutoff * cutoff;
  for (int energy = 0; energy < 2; energy++) {
    printf("%d %s%d_rho %d\n", device, name, n_types,
           launch_rho64(g, st, P, L, sp.rc2, &some, energy, 0, nullptr, 0, -1, nullptr, planned ? &plan : nullptr));
    printf("%d %s%d_force %d\n", device, name, n_types,
           launch_force64(g, st, P, L, sp, &some, energy, 0, nullptr, 0, -1, nullptr, planned ? &plan : nullptr));
  }
}

static void mixed(int fixed, bool linear) {
  EnsParams P{};
  static MxStencil S{};
  S.fixed = fixed;
  S.n_rs = 24000;
  S.n_fs = 24000;
  S.walk.linear = linear;
  S.walk.n_lats = 1;
  S.walk.n_items = 1 << 20;
  for (int energy = 0; energy < 2; energy++)
    printf("%d mixed%d_%d %d\n", device, fixed, (int)linear, mx_launch_step(P, S, 0, energy, nullptr, nullptr, nullptr));
}

// The persistent kernel with few knots in shared memory and with many, an ensemble of each.
static void persistent() {
  const int knots[2] = {100, 3000};
  for (int k : knots) printf("%d persistent_grid%d %d\n", device, k, ens_max_grid(k) == 148 ? 0 : 1);
  for (int first = 0; first < 2; first++) // either of them made last
    for (int k = 0; k < 2; k++) {
      ens_max_grid(knots[first]);
      EnsParams P{};
      P.nsm = knots[k];
      P.energy = first;
      printf("%d persistent%d_%d %d\n", device, knots[k], first, ens_launch(P, 148, nullptr));
    }
}

// Hooks split items only where a site's index leaves two bits free; a small box inside a wide
// frame of ghosts reaches beyond that.
static void wide_ghosts(int width, bool splits) {
  Geom g{};
  g.bcx = g.by = g.bz = 8;
  g.gcx = g.gy = g.gz = width;
  g.ecx = g.ey = g.ez = 8 + 2 * width;
  g.E = (long long)g.ecx * g.ey * g.ez;
  StencilSet st{};
  st.n = 88;
  Shells64 S;
  printf("%d ghosts%d %d\n", device, width, plan64_entries(g, st, S) == splits ? 0 : 1);
}

int main() {
  for (device = 0; device < 2; device++) {
    for (int n_types : {1, 3}) {
      fp64("shell", n_types, "0", true);
      fp64("split", n_types, "1000000", true);
      fp64("rows", n_types, "0", false);
    }
    for (int fixed : {0, 7, 8})
      for (bool linear : {false, true})
        if (fixed || !linear) mixed(fixed, linear);
    persistent();
    wide_ghosts(400, true);
    wide_ghosts(402, true);
    wide_ghosts(403, false); // 2 x 814^3 sites
    wide_ghosts(500, false);
  }
  return 0;
}
