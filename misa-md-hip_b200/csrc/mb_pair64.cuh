// FP64 pair terms of the lattice passes, shared by the shell-window kernels
// (mb_shell64.cu, large launches) and the entry-split kernels (mb_split64.cu, small ones).
//
// Both sum a site's stencil in the same fixed order, so a lattice gives the same bits
// whichever of them runs (a z-slab of a large lattice may be a small launch):
//   * near entries (inside the cutoff at the ideal lattice, by distance) in runs of up to
//     MB_RUN entries of one shell; then runs of MB_OUT_RUN outer entries;
//   * within a near run first the pairs inside the shell's table window, in entry order,
//     then the others (strongly displaced atoms) that are inside the cutoff, in entry order;
//   * the site's total takes the run sums in order.
// Every rounding is spelled out (__fma_rn and friends), so that the two kernels cannot
// differ in what the compiler contracts.
#pragma once

#include "mb_device.cuh"
#include "mb_ensemble_shells.cuh"

namespace mb {

// Work items: 32 consecutive sites of one (z, sublattice) plane; a lane's entry of the site
// list (Plan64::sites) is its ext index, with MB_SITE_FACE where the site has periodic
// images, or negative (no site).  Items of box layers [z0, z1) are a contiguous range.
#define MB_SITE_FACE 0x40000000
#define MB_SITE_INDEX 0x3fffffff

// Everything the two kinds of kernel need.
struct LatticeArgs {
  Geom g;
  DevPot P;
  Lattice64 L;
  Shells64 sh;
  const int *sites;
  int w0, n_items;       // items [w0, n_items)
  double rc2, rc2m;      // squared cutoff; a hair above it for the outer-entry masks
  int rc2_hi;            // high word of rc2
  int copies;            // table copies of a shell window (several types)
  bool chain;            // see launch_chained
  int flag;              // code bit of the sites an interstitial pass finishes (0: none)
  uint2 *outer;          // per item: the outer entries some lane has inside rc2m (or null)
  double *e0, *e1;       // CTA partials: density pass F(rho); force pass pair and kinetic energy
  StepParams sp;
};

// ------------------------------------------------------------- pair terms
// sqrt(d2) and 1 / sqrt(d2): the hardware's seed y and one step of Householder's iteration
// of order 3, y (1 + e (1/2 + 3/8 e)) with e = 1 - d2 y^2.
__device__ __forceinline__ void root64(double d2, double &r, double &rinv) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d2));
  const double t = __dmul_rn(d2, y), e = __fma_rn(-t, y, 1.0), h = __dmul_rn(e, __fma_rn(0.375, e, 0.5));
  r = __fma_rn(t, h, t);
  rinv = __fma_rn(y, h, y);
}

// Interval of r in a table window that starts at knot lo, given base = MB_FLOOR - lo:
// rounding base + r / dr down to a whole number leaves it in the low word.  True inside
// the window (n intervals, all inside the cutoff): then k is the interval's place in it
// and p the local coordinate.
#define MB_FLOOR 6755399441055744.0 // 1.5 * 2^52
#define MB_FLOOR_HI 0x43380000      // its high word
__device__ __forceinline__ bool window_locate(double r, double rdr, double base, unsigned n, unsigned &k, double &p) {
  const double s = __fma_rd(r, rdr, base);
  k = (unsigned)__double2loint(s);
  p = __fma_rn(r, rdr, __dsub_rn(base, s));
  return __double2hiint(s) == MB_FLOOR_HI && k < n;
}

// The same in the whole table, for the pairs outside their window (r < cutoff).  Coincident
// atoms have no r (0 times an infinite root), and a NaN converts to the most negative integer:
// the clamp compares unsigned, so that m is an interval for any r.  p is then undefined as
// in the row walk's spl_locate_in (one type), or the interval's end as in its spl_locate.
// (The interval's end for one type too, by the compare below or by fmin, costs every outer
// pair: steps at 6^3, 20^3 and 37 x 52 x 45 cells 1% slower.)
__device__ __forceinline__ void table_locate(double r, const DevPot &P, int &m, double &p) {
  m = (int)min((unsigned)(int)__dmul_rd(r, P.rdr), (unsigned)(P.nr - 2));
  p = __fma_rn(r, P.rdr, -(double)m);
  if (P.n_types > 1 && r != r) p = 1.0;
}

// Squared length of d, summed as x, y, z.
__device__ __forceinline__ double len2(double dx, double dy, double dz) {
  return __fma_rn(dz, dz, __fma_rn(dy, dy, __dmul_rn(dx, dx)));
}

// Spline value between the knots k0 = {y, s} and k1: cubic Hermite piece.
__device__ __forceinline__ double hermite64(double2 k0, double2 k1, double p) {
  const double dy = __dsub_rn(k1.x, k0.x), u = __dsub_rn(dy, k0.y), c3 = __dsub_rn(__dsub_rn(k1.y, dy), u);
  return __fma_rn(__fma_rn(__fma_rn(c3, p, __dsub_rn(u, c3)), p, k0.y), p, k0.x);
}

// Spline derivative on an interval from its end values d0, d1 and quadratic coefficient c.
__device__ __forceinline__ double slope64(double d0, double c, double d1, double p) {
  return __fma_rn(__fma_rn(c, p, __dsub_rn(__dsub_rn(d1, d0), c)), p, d0);
}

// Table window in shared memory: `words` 16-byte words per knot, interleaved copies of every
// word, lane l reading copy l % copies; w is the window's first knot.  With 8 copies the 8
// lanes that a wavefront of 16-byte loads serves read 8 different bank groups, whatever
// their knots.
// One type (COPIES > 0): one word {y, s} (density) or two, {f', phi'} at the knot and their
// quadratic coefficients (force).  Several (COPIES == 0, copies at run time): per type
// {y, s}, or {f', coefficient}, then per pair of types {phi', coefficient}.
template <int COPIES>
struct Window64 {
  const double2 *w; // this lane's copy of the window's first knot
  double base;      // MB_FLOOR - first knot
  unsigned n;       // intervals
  int words, copies; // COPIES == 0 only
};

// Word of a pair of types among `nt` (the packed upper triangle, after the nt types).
__device__ __forceinline__ int pair_word(int a, int b, int nt) {
  const int lo = min(a, b), hi = max(a, b);
  return nt + lo * nt - lo * (lo + 1) / 2 + hi;
}

// Whether a pair outside its window may be inside the cutoff (vacant sites are far away).
__device__ __forceinline__ bool maybe_in(const LatticeArgs &a, double d2) { return __double2hiint(d2) <= a.rc2_hi; }

// Density term of a pair with an atom of type tj; false outside the window.
template <int COPIES>
__device__ __forceinline__ bool rho_pair64(const Window64<COPIES> &W, const DevPot &P, double d2, int tj, double &v) {
  double r, rinv, p;
  unsigned k;
  root64(d2, r, rinv);
  const bool ok = window_locate(r, P.rdr, W.base, W.n, k, p);
  k = min(k, W.n - 1);
  if constexpr (COPIES > 0) {
    const double2 *q = W.w + k * COPIES;
    v = hermite64(q[0], q[COPIES], p);
  } else {
    const double2 *q = W.w + (k * W.words + tj) * W.copies;
    v = hermite64(q[0], q[W.words * W.copies], p);
  }
  return ok;
}
__device__ __forceinline__ double rho_table64(const DevPot &P, double d2, int tj) {
  double r, rinv, p;
  int m;
  root64(d2, r, rinv);
  table_locate(r, P, m, p);
  const double2 *q = P.f_ys + (size_t)m * P.n_types + tj;
  return hermite64(__ldg(q), __ldg(q + P.n_types), p);
}

// fpair = -(df_i f'_tj + df_j f'_ti + phi'_titj) / r of a pair; false outside the window.
// With ENERGY e is half its pair energy (inside the window).
__device__ __forceinline__ double half_phi64(const DevPot &P, int ti, int tj, int m, double p) {
  const double4 v = ldg4(P.phi_val + (size_t)pair_idx(ti, tj, P.n_types) * P.nr + m);
  return __dmul_rn(0.5, __fma_rn(__fma_rn(__fma_rn(v.w, p, v.z), p, v.y), p, v.x));
}
// ... from the words of the pair's interval at q (several types), `step` to the next word and
// `knot` to the next knot.
template <class Load>
__device__ __forceinline__ double force_words64(const double2 *q, int step, int knot, int nt, int ti, int tj,
                                                double dfi, double dfj, double p, Load load) {
  auto slope = [&](int word) {
    const double2 a = load(q + word * step), b = load(q + word * step + knot);
    return slope64(a.x, a.y, b.x, p);
  };
  const double fj = slope(tj), fi = slope(ti), ph = slope(pair_word(ti, tj, nt));
  return __fma_rn(dfi, fj, __fma_rn(dfj, fi, ph));
}
template <int COPIES, bool ENERGY>
__device__ __forceinline__ bool force_pair64(const Window64<COPIES> &W, const DevPot &P, double d2, int ti, int tj,
                                             double dfi, double dfj, double &f, double &e) {
  double r, rinv, p;
  unsigned k;
  root64(d2, r, rinv);
  const bool ok = window_locate(r, P.rdr, W.base, W.n, k, p);
  const unsigned kk = min(k, W.n - 1);
  double g;
  if constexpr (COPIES > 0) {
    const double2 *q = W.w + kk * (2 * COPIES);
    const double2 d0 = q[0], c = q[COPIES], d1 = q[2 * COPIES];
    g = __fma_rn(__dadd_rn(dfi, dfj), slope64(d0.x, c.x, d1.x, p), slope64(d0.y, c.y, d1.y, p));
  } else {
    g = force_words64(W.w + kk * (W.words * W.copies), W.copies, W.words * W.copies, P.n_types, ti, tj, dfi, dfj, p,
                      [](const double2 *x) { return *x; });
  }
  f = __dmul_rn(-g, rinv);
  if (ENERGY && ok) e = half_phi64(P, ti, tj, (int)k + (int)(MB_FLOOR - W.base), p);
  return ok;
}
template <bool ENERGY>
__device__ __forceinline__ double force_table64(const DevPot &P, double d2, int ti, int tj, double dfi, double dfj,
                                                double &e) {
  double r, rinv, p, g;
  int m;
  root64(d2, r, rinv);
  table_locate(r, P, m, p);
  if (P.n_types == 1) {
    const double2 *t = P.force2 + 2 * (size_t)m;
    const double2 d0 = __ldg(t), c = __ldg(t + 1), d1 = __ldg(t + 2);
    g = __fma_rn(__dadd_rn(dfi, dfj), slope64(d0.x, c.x, d1.x, p), slope64(d0.y, c.y, d1.y, p));
  } else {
    const int words = P.n_types + P.n_types * (P.n_types + 1) / 2;
    g = force_words64(P.force2 + (size_t)m * words, 1, words, P.n_types, ti, tj, dfi, dfj, p,
                      [](const double2 *x) { return __ldg(x); });
  }
  if (ENERGY) e = half_phi64(P, ti, tj, m, p);
  return __dmul_rn(-g, rinv);
}

// Lane `lane`'s site of item w: index and MB_SITE_FACE, -1 past the end of the plane.
__device__ __forceinline__ int site_ref64(const Geom &g, int w, int lane) {
  const int cpp = (g.bcx * g.by + 31) / 32, p = w / cpp, b = (w - p * cpp) * 32 + lane;
  const int y = b / g.bcx, cx = b - y * g.bcx, s = p & 1, z = p >> 1;
  if (y >= g.by) return -1;
  int ref = (int)ext_index(g, s, cx, y, z);
  if (cx < g.gcx || cx >= g.bcx - g.gcx || y < g.gy || y >= g.by - g.gy || z < g.gz || z >= g.bz - g.gz)
    ref |= MB_SITE_FACE;
  return ref;
}

// A site at work: its record and code, F' and stencil offsets.
struct Site64 {
  const double4 *p;  // its record
  const int8_t *c;   // its code
  const int *off;    // the stencil of its sublattice
  double x, y, z, w; // position and F'
  int type;
};
// Type of the site whose code is *c, of nt (vacant sites: any; the distance rejects them).
__device__ __forceinline__ int type_at(const int8_t *c, int nt) { return min(*c & MB_TYPE_MASK, nt - 1); }
__device__ __forceinline__ int far_type(const LatticeArgs &a, const Site64 &c, int k) {
  return a.P.n_types == 1 ? 0 : type_at(c.c + c.off[k], a.P.n_types);
}

// ------------------------------------------------------------------ runs
// The pairs of a run that fell outside their window: entries k0 + b for the bits b of `far`.
__device__ __forceinline__ void rho_far(const LatticeArgs &a, const Site64 &c, int k0, unsigned far, double &t) {
  while (far) {
    const int k = k0 + __ffs(far) - 1;
    far &= far - 1;
    const double4 q = ld_site(c.p + c.off[k]);
    const double d2 = len2(c.x - q.x, c.y - q.y, c.z - q.z);
    if (d2 < a.rc2) t = __dadd_rn(t, rho_table64(a.P, d2, far_type(a, c, k)));
  }
}
template <bool ENERGY>
__device__ __forceinline__ void force_far(const LatticeArgs &a, const Site64 &c, int k0, unsigned far, double &fx,
                                          double &fy, double &fz, double &ep) {
  while (far) {
    const int k = k0 + __ffs(far) - 1;
    far &= far - 1;
    const double4 q = ld_site(c.p + c.off[k]);
    const double dx = c.x - q.x, dy = c.y - q.y, dz = c.z - q.z, d2 = len2(dx, dy, dz);
    if (d2 < a.rc2) {
      double e;
      const double f = force_table64<ENERGY>(a.P, d2, c.type, far_type(a, c, k), c.w, q.w, e);
      fx = __fma_rn(dx, f, fx);
      fy = __fma_rn(dy, f, fy);
      fz = __fma_rn(dz, f, fz);
      if (ENERGY) ep += e;
    }
  }
}

// One near entry of a run (bit: its place in the run), q the neighbour's record, tj its type.
template <int COPIES>
__device__ __forceinline__ void rho_near(const LatticeArgs &a, const Window64<COPIES> &W, const Site64 &c,
                                         const double4 &q, int tj, int bit, double &t, unsigned &far) {
  const double d2 = len2(c.x - q.x, c.y - q.y, c.z - q.z);
  double v;
  const bool ok = rho_pair64(W, a.P, d2, tj, v);
  if (ok) t = __dadd_rn(t, v);
  if (!ok && maybe_in(a, d2)) far |= 1u << bit;
}
template <int COPIES, bool ENERGY>
__device__ __forceinline__ void force_near(const LatticeArgs &a, const Window64<COPIES> &W, const Site64 &c,
                                           const double4 &q, int tj, int bit, double &fx, double &fy, double &fz,
                                           double &ep, unsigned &far) {
  const double dx = c.x - q.x, dy = c.y - q.y, dz = c.z - q.z, d2 = len2(dx, dy, dz);
  double f, e;
  const bool ok = force_pair64<COPIES, ENERGY>(W, a.P, d2, c.type, tj, c.w, q.w, f, e);
  if (ok) {
    fx = __fma_rn(dx, f, fx);
    fy = __fma_rn(dy, f, fy);
    fz = __fma_rn(dz, f, fz);
    if (ENERGY) ep += e;
  }
  if (!ok && maybe_in(a, d2)) far |= 1u << bit;
}

// The outer entries [k0, k1) of a density sum; near: bit k - k0 set when entry k lies
// inside the margin of the masks.
__device__ __forceinline__ double rho_outer(const LatticeArgs &a, const Site64 &c, int k0, int k1, unsigned &near) {
  double t = 0.0;
#pragma unroll 4
  for (int k = k0; k < k1; k++) {
    const double4 q = ld_site(c.p + c.off[k]);
    const double d2 = len2(c.x - q.x, c.y - q.y, c.z - q.z);
    near |= (unsigned)(d2 < a.rc2m) << (k - k0);
  }
  // inside the margin: nearly always inside the cutoff too
  rho_far(a, c, k0, near, t);
  return t;
}

// The outer entries [k0, k1) of a force: those whose bit k - k0 of `bits` is set (the others
// are beyond the cutoff for every lane of the item), or all (`all`).
template <bool ENERGY>
__device__ __forceinline__ void force_outer(const LatticeArgs &a, const Site64 &c, int k0, int k1, bool all,
                                            unsigned bits, double &fx, double &fy, double &fz, double &ep) {
  fx = fy = fz = 0.0;
  unsigned in = 0;
  if (all) {
#pragma unroll 4
    for (int k = k0; k < k1; k++) {
      const double4 q = ld_site(c.p + c.off[k]);
      in |= (unsigned)(len2(c.x - q.x, c.y - q.y, c.z - q.z) < a.rc2) << (k - k0);
    }
  } else {
    bits &= (1u << (k1 - k0)) - 1u;
    while (bits) {
      const int b = __ffs(bits) - 1;
      bits &= bits - 1;
      const double4 q = ld_site(c.p + c.off[k0 + b]);
      in |= (unsigned)(len2(c.x - q.x, c.y - q.y, c.z - q.z) < a.rc2) << b;
    }
  }
  force_far<ENERGY>(a, c, k0, in, fx, fy, fz, ep);
}

// --------------------------------------------------------- ends of a site
__device__ __forceinline__ void decode_site(const Geom &g, int i, int &s, int &cx, int &y, int &z) {
  const unsigned E = (unsigned)g.E, u = (unsigned)i;
  s = u >= E;
  const unsigned r = u - (s ? E : 0u), row = r / (unsigned)g.ecx;
  cx = (int)(r - row * (unsigned)g.ecx) - g.gcx;
  const unsigned ez = row / (unsigned)g.ey;
  z = (int)ez - g.gz;
  y = (int)(row - ez * (unsigned)g.ey) - g.gy;
}

// df = F'(rho), its ghost images; returns F(rho) with ENERGY.
template <bool ENERGY>
__device__ __forceinline__ double rho_finish64(const Geom &g, const DevPot &P, const Lattice64 &L, int code, int flag,
                                               int ref, double rho) {
  const int i = ref & MB_SITE_INDEX, ti = code & MB_TYPE_MASK;
  if (code & flag) { // the interstitial pass adds its pairs to this sum
    L.rho[i] = rho;
    return 0.0;
  }
  const double df = dF64(P, ti, rho);
  L.p[i].w = df;
  L.rho[i] = rho;
  if (g.images && (ref & MB_SITE_FACE)) {
    int s, cx, y, z;
    decode_site(g, i, s, cx, y, z);
    for_images(g, s, cx, y, z, [&](long long idx, double, double, double) { L.p[idx].w = df; });
  }
  return ENERGY ? F64(P, ti, rho) : 0.0;
}

// Lists the box site of a drifted lattice atom that left its site (conversion on).
__device__ __forceinline__ void conv_check(const Geom &g, const StepParams &sp, int s, int cx, int y, int z, double nx,
                                           double ny, double nz) {
  if (!(sp.conv2 > 0.0)) return;
  double X, Y, Z;
  site_ideal(s, cx, y, z, sp.a0, X, Y, Z);
  const double ux = nx - X, uy = ny - Y, uz = nz - Z;
  if (ux * ux + uy * uy + uz * uz <= sp.conv2) return;
  const int slot = atomicAdd(sp.cand_n, 1);
  if (slot < MB_CAND_CAP) sp.cand[slot] = ((long long)z * g.by + y) * (2LL * g.bcx) + 2LL * cx + s;
}

// Force of a site: stores it, closes the previous step, drifts to the next positions (and
// their ghost images); returns the kinetic energy with ENERGY.
template <bool ENERGY>
__device__ __forceinline__ double force_finish64(const Geom &g, const Lattice64 &L, const StepParams &sp, bool flagged,
                                                 int ref, const Site64 &c, double fx, double fy, double fz) {
  double ek = 0.0;
  const int i = ref & MB_SITE_INDEX;
  L.fx[i] = fx;
  L.fy[i] = fy;
  L.fz[i] = fz;
  if (flagged || !L.vx) return ek; // flagged: the interstitial pass adds its pairs and integrates
  double vx = L.vx[i], vy = L.vy[i], vz = L.vz[i];
  if (sp.kick_pre) {
    vx = __fma_rn(sp.h, fx, vx);
    vy = __fma_rn(sp.h, fy, vy);
    vz = __fma_rn(sp.h, fz, vz);
  }
  if (ENERGY) ek = 0.5 * sp.mass * (vx * vx + vy * vy + vz * vz) * MB_MVV2E;
  if (sp.drift) {
    vx = __fma_rn(sp.h, fx, vx);
    vy = __fma_rn(sp.h, fy, vy);
    vz = __fma_rn(sp.h, fz, vz);
    const double nx = __fma_rn(sp.dt, vx, c.x), ny = __fma_rn(sp.dt, vy, c.y), nz = __fma_rn(sp.dt, vz, c.z);
    st_site(L.n + i, nx, ny, nz, 0.0);
    const bool face = g.images && (ref & MB_SITE_FACE);
    if (face || sp.conv2 > 0.0) {
      int s, cx, y, z;
      decode_site(g, i, s, cx, y, z);
      conv_check(g, sp, s, cx, y, z, nx, ny, nz);
      if (face)
        for_images(g, s, cx, y, z, [&](long long idx, double ox, double oy, double oz) {
          st_site(L.n + idx, nx + ox, ny + oy, nz + oz, 0.0);
        });
    }
  }
  L.vx[i] = vx;
  L.vy[i] = vy;
  L.vz[i] = vz;
  return ek;
}

} // namespace mb
