// Per-pair FP32 arithmetic and interstitial items of the mixed-precision step,
// shared by the persistent tile kernel (mb_ensemble.cu) and the split kernels
// (mb_ensemble_split.cu, one lattice or many).
#pragma once

#include "mb_ensemble_kernel.cuh"

namespace mb {

// Spline knot and local coordinate of a pair from its deviation eps = r - R_k.
__device__ __forceinline__ void knot_of(const EnsParams &P, int s, int k, float eps, int &m, float &q) {
  const float2 kf = P.kf[s][k];
  const float t = kf.x + eps * P.rdr;
  const float fl = floorf(t);
  q = t - fl;
  m = min(max((int)(kf.y + fl), 0), P.P.nr - 2);
}

// Pair geometry shared by both passes (x and y in f32x2 lanes): returns false
// beyond the cutoff; on success r2 and the spline deviation numerator are set.
struct PairGeo {
  float2 dxy;
  float dz, r2, num;
};

// ALWAYS: also compute the numerator beyond the cutoff (branch-free walking).
template <bool ALWAYS>
__device__ __forceinline__ bool pair_geo(const EnsParams &P, const float4 &u, const float4 &nb, const float4 &C,
                                         PairGeo &g) {
  const float2 m1 = make_float2(-1.f, -1.f);
  const float2 exy = __ffma2_rn(make_float2(nb.x, nb.y), m1, make_float2(u.x, u.y)); // u - nb
  const float ez = u.z - nb.z;
  g.dxy = __fadd2_rn(make_float2(C.x, C.y), exy);
  g.dz = C.z + ez;
  const float2 sq = __fmul2_rn(g.dxy, g.dxy);
  g.r2 = sq.x + sq.y + g.dz * g.dz;
  const bool in = g.r2 < P.rc2f;
  if (!ALWAYS && !in) return false;
  const float2 pe = __fmul2_rn(__ffma2_rn(make_float2(2.f, 2.f), make_float2(C.x, C.y), exy), exy); // (2C + e) e
  g.num = pe.x + pe.y + (2.f * C.z + ez) * ez;
  return in;
}

// One density pair.  BF (branch-free): entries inside the cutoff for nearly every
// lane; the value is masked instead of branched around so iterations overlap.
template <bool BF>
__device__ __forceinline__ void rho_pair(const EnsParams &P, const float4 &u, const float4 &nb, const float4 &C, int s,
                                         int k, const float4 *s_fv, float &rs, float &rc) {
  PairGeo g;
  const bool in = pair_geo<BF>(P, u, nb, C, g);
  if (!BF && !in) return;
  const float r = g.r2 * rsqrtf(g.r2);
  int m;
  float q;
  knot_of(P, s, k, __fdividef(g.num, r + C.w), m, q);
  const float4 c = (m >= P.m_lo) ? s_fv[m - P.m_lo] : __ldg(&P.P.f_val32[m]);
  float v = ((c.w * q + c.z) * q + c.y) * q + c.x;
  if (BF) v = in ? v : 0.f;
  two_sum(rs, rc, v);
}

// Knuth two-sum on packed pairs of lanes (f32x2 instructions).
__device__ __forceinline__ void two_sum2(float2 &s, float2 &c, float2 x) {
  const float2 m1 = make_float2(-1.f, -1.f);
  const float2 t = __fadd2_rn(s, x);
  const float2 bp = __ffma2_rn(s, m1, t);                  // t - s
  const float2 sa = __ffma2_rn(__ffma2_rn(bp, m1, t), m1, s); // s - (t - bp)
  const float2 xb = __ffma2_rn(bp, m1, x);                  // x - bp
  c = __fadd2_rn(c, __fadd2_rn(sa, xb));
  s = t;
}

// One pair of the force pass: x and y components ride together in f32x2 lanes, and
// the derivative pieces of f and phi (stored as {f', phi'} pairs per knot) are
// evaluated by one packed Horner chain.
template <bool ENERGY, bool BF>
__device__ __forceinline__ void force_pair(const EnsParams &P, const float4 &u, const float4 &nb, const float4 &C,
                                           int s, int k, const float2 *s_fd, float2 &fxy_s, float2 &fxy_c, float &zs,
                                           float &zc, float &ps, float &pc) {
  PairGeo g;
  const bool in = pair_geo<BF>(P, u, nb, C, g);
  if (!BF && !in) return;
  const float r2 = g.r2, num = g.num, dz = g.dz;
  const float2 dxy = g.dxy;
  float rinv = rsqrtf(r2);
  rinv = rinv * (1.5f - 0.5f * r2 * rinv * rinv);
  const float r = r2 * rinv;
  int m;
  float q;
  knot_of(P, s, k, __fdividef(num, r + C.w), m, q);
  float2 c0, c1, c2;
  if (m >= P.m_lo) {
    const float2 *cp = s_fd + 3 * (m - P.m_lo);
    c0 = cp[0];
    c1 = cp[1];
    c2 = cp[2];
  } else {
    const float2 *cp = P.P.force32 + 3 * m;
    c0 = __ldg(cp);
    c1 = __ldg(cp + 1);
    c2 = __ldg(cp + 2);
  }
  const float2 qq = make_float2(q, q);
  const float2 dd = __ffma2_rn(__ffma2_rn(c2, qq, c1), qq, c0); // {f'(r), phi'(r)}
  float fpair = -((u.w + nb.w) * dd.x + dd.y) * rinv;
  if (BF) fpair = in ? fpair : 0.f;
  two_sum2(fxy_s, fxy_c, __fmul2_rn(dxy, make_float2(fpair, fpair)));
  two_sum(zs, zc, dz * fpair);
  if (ENERGY) {
    const float4 pv = __ldg(&P.P.phi_val32[m]);
    float e = 0.5f * (((pv.w * q + pv.z) * q + pv.y) * q + pv.x);
    if (BF) e = in ? e : 0.f;
    two_sum(ps, pc, e);
  }
}

// ------------------------------------------------------- interstitial items
// Sites marked at the previous step of lattice d lose their mark (threads t, t + n, ...).
// Lists, counts and mark bits alternate with the buffer parity: list cur holds this step's
// sites, list cur ^ 1 last step's.  The bookkeeping at the end of a step empties the latter.
__device__ __forceinline__ int *flag_list_of(const LatDesc &d, int parity) {
  return d.flag_list + (size_t)parity * d.cap_flag;
}
__device__ __forceinline__ void itl_clear_flags(const LatDesc &d, int t, int n) {
  const int old = d.cur ^ 1;
  const int nold = min(d.flag_count[old], d.cap_flag);
  const int *list = flag_list_of(d, old);
  for (int k = t; k < nold; k += n) code_bit_off(d.code + list[k], MB_FLAG_ITL(old));
}

// `n` threads (whole warps; this one is number t) mark the lattice sites within reach of
// interstitial `it`.
__device__ __forceinline__ void itl_mark_one(const EnsParams &P, const LatDesc &d, int it, int t, int n) {
  const Geom g = lat_geom(d);
  const int cur = d.cur;
  int *list = flag_list_of(d, cur);
  const double qx = d.ipx[cur][it], qy = d.ipy[cur][it], qz = d.ipz[cur][it];
  const Window w = make_window(qx, qy, qz, P.a0, P.reach);
  const int ncand = w.nx * w.ny * w.nz;
  for (int base = 0; base < ncand; base += n) { // whole warps per round (warp_append)
    const int k = base + t;
    long long idx = 0;
    double sx, sy, sz;
    const bool fresh = k < ncand && window_site(g, w, k, qx, qy, qz, P.a0, P.reach, idx, sx, sy, sz) &&
                       d.code[idx] >= 0 && code_bit_on(d.code + idx, MB_FLAG_ITL(cur));
    // flag_count[2]: overflow, reported by the host
    warp_append(fresh, (int)idx, &d.flag_count[cur], list, d.cap_flag, &d.flag_count[2]);
  }
}

// Coarse cell of a point of lattice d (wrapped into the box).
__device__ __forceinline__ void itl_cell3(const LatDesc &d, double x, double y, double z, int &cx, int &cy, int &cz) {
  const double fx = x / d.Lx - floor(x / d.Lx), fy = y / d.Ly - floor(y / d.Ly), fz = z / d.Lz - floor(z / d.Lz);
  cx = max(0, min((int)(fx * d.icn[0]), d.icn[0] - 1));
  cy = max(0, min((int)(fy * d.icn[1]), d.icn[1] - 1));
  cz = max(0, min((int)(fz * d.icn[2]), d.icn[2] - 1));
}

// Interstitial-pair part of an item: every interstitial within the 27 cells around the
// query point (the cells are at least cutoff + skin wide, so nothing in reach is left
// out), lane c walking cell c in list order; or the whole list when there is no cell
// list this step.  Each lane sums its own pairs in a fixed order.
template <bool CELLS, class Pair>
__device__ __forceinline__ void itl_pairs(const LatDesc &d, const Geom &g, int cur, double xi, double yi, double zi,
                                          int skip, int lane, Pair pair, bool with_df) {
  if (CELLS && d.icount && d.iflag[0]) {
    if (lane >= 27) return;
    int qx, qy, qz;
    itl_cell3(d, xi, yi, zi, qx, qy, qz);
    const int ox = lane % 3 - 1, oy = (lane / 3) % 3 - 1, oz = lane / 9 - 1;
    const int cx = (qx + ox + d.icn[0]) % d.icn[0], cy = (qy + oy + d.icn[1]) % d.icn[1],
              cz = (qz + oz + d.icn[2]) % d.icn[2];
    const int c = (cz * d.icn[1] + cy) * d.icn[0] + cx;
    const int n = d.icount[c], s0 = d.istart[c];
    for (int j = s0; j < s0 + n; j++) {
      const int K = d.iitem[j];
      if (K == skip) continue;
      pair(min_image(xi - d.ipx[cur][K], g.Lx, g.iLx), min_image(yi - d.ipy[cur][K], g.Ly, g.iLy),
           min_image(zi - d.ipz[cur][K], g.Lz, g.iLz), d.itype[K], with_df ? d.idf[K] : 0.0);
    }
    return;
  }
  for (int K = lane; K < d.n_itl; K += 32) {
    if (K == skip) continue;
    pair(min_image(xi - d.ipx[cur][K], g.Lx, g.iLx), min_image(yi - d.ipy[cur][K], g.Ly, g.iLy),
         min_image(zi - d.ipz[cur][K], g.Lz, g.iLz), d.itype[K], with_df ? d.idf[K] : 0.0);
  }
}

// One FP64 pair of an interstitial item (atom of type ti, df dfi; partner of type tj, df
// dfj at pair vector d = own - partner): its density term into rho, or its force and pair
// energy into f and ep.  Pairs at or beyond the cutoff add nothing.
template <bool FORCE, bool ENERGY>
__device__ __forceinline__ void itl_pair(const EnsParams &P, int ti, double dfi, double dx, double dy, double dz,
                                         int tj, double dfj, double &rho, double &fx, double &fy, double &fz,
                                         double &ep) {
  const double d2 = dx * dx + dy * dy + dz * dz;
  if (d2 >= P.rc2) return;
  const double rinv = rsqrt(d2);
  const double r = d2 * rinv;
  if (!FORCE) {
    rho += rho_of_r(P.P, tj, r);
  } else {
    double ph = 0.0;
    const double psip = pair_psip(P.P, ti, tj, r, dfi, dfj, ENERGY ? &ph : nullptr);
    const double fpair = -psip * rinv;
    fx += dx * fpair;
    fy += dy * fpair;
    fz += dz * fpair;
    if (ENERGY) ep += 0.5 * ph;
  }
}

// Last part of an item, on one lane, from its summed pairs: df (density pass), or force,
// velocity-Verlet, drift and ghost images (force pass), of a flagged site (i at s, cx, y,
// z) or of interstitial it.
template <bool FORCE, bool ENERGY>
__device__ __forceinline__ void itl_finish(const EnsParams &P, const LatDesc &d, const Geom &g, bool is_site,
                                           long long i, int s, int cx, int y, int z, int it, int ti, double xi,
                                           double yi, double zi, double rho, double fx, double fy, double fz,
                                           double ep) {
  const int cur = d.cur;
  if (!FORCE) {
    const double df = dF64(P.P, ti, rho);
    if (is_site) {
      float4 *uw = d.u4[cur];
      reinterpret_cast<float *>(uw + i)[3] = (float)df;
      d.rho[i] = (float)rho;
      for_images(g, s, cx, y, z,
                 [&](long long idx, double, double, double) { reinterpret_cast<float *>(uw + idx)[3] = (float)df; });
    } else {
      d.irho[it] = rho;
      d.idf[it] = df;
    }
    if (ENERGY) atomicAdd(&d.e_itl[0], F64(P.P, ti, rho));
    return;
  }
  double vx, vy, vz;
  if (is_site) {
    d.fx[i] = (float)fx;
    d.fy[i] = (float)fy;
    d.fz[i] = (float)fz;
    vx = d.vx[i];
    vy = d.vy[i];
    vz = d.vz[i];
  } else {
    d.ifx[it] = fx;
    d.ify[it] = fy;
    d.ifz[it] = fz;
    vx = d.ivx[it];
    vy = d.ivy[it];
    vz = d.ivz[it];
  }
  if (d.primed) {
    vx += P.h * fx;
    vy += P.h * fy;
    vz += P.h * fz;
  }
  if (ENERGY) {
    atomicAdd(&d.e_itl[0], ep);
    atomicAdd(&d.e_itl[1], 0.5 * P.mass * (vx * vx + vy * vy + vz * vz) * MB_MVV2E);
  }
  vx += P.h * fx;
  vy += P.h * fy;
  vz += P.h * fz;
  if (is_site) {
    d.vx[i] = vx;
    d.vy[i] = vy;
    d.vz[i] = vz;
    const double nx = d.ux[i] + P.dt * vx, ny = d.uy[i] + P.dt * vy, nz = d.uz[i] + P.dt * vz;
    d.ux[i] = nx;
    d.uy[i] = ny;
    d.uz[i] = nz;
    const float4 nu = make_float4((float)nx, (float)ny, (float)nz, 0.f);
    float4 *un = d.u4[cur ^ 1];
    un[i] = nu;
    ens_conv_check(P, d, s, cx, y, z, nx, ny, nz);
    for_images(g, s, cx, y, z, [&](long long idx, double, double, double) { un[idx] = nu; });
  } else {
    d.ivx[it] = vx;
    d.ivy[it] = vy;
    d.ivz[it] = vz;
    d.ipx[cur ^ 1][it] = xi + P.dt * vx;
    d.ipy[cur ^ 1][it] = yi + P.dt * vy;
    d.ipz[cur ^ 1][it] = zi + P.dt * vz;
  }
}

// Pairs of an interstitial at (xi, yi, zi) with the lattice sites of its window: candidates
// t, t + n, ..., handed to pair (which sums them per thread).
template <class Pair>
__device__ __forceinline__ void itl_window_pairs(const EnsParams &P, const LatDesc &d, const Geom &g,
                                                 const float4 *u4, double xi, double yi, double zi, int t, int n,
                                                 bool with_df, Pair pair) {
  const Window win = make_window(xi, yi, zi, P.a0, P.reach);
  const int ncand = win.nx * win.ny * win.nz;
  for (int c = t; c < ncand; c += n) {
    long long j;
    double ox, oy, oz;
    if (!window_site_rel(g, win, c, xi, yi, zi, P.a0, P.reach, j, ox, oy, oz)) continue;
    const int cj = d.code[j];
    const float4 uj = u4[j];
    if (cj >= 0)
      pair(-(ox + (double)uj.x), -(oy + (double)uj.y), -(oz + (double)uj.z), cj & MB_TYPE_MASK,
           with_df ? (double)uj.w : 0.0);
  }
}

// Work of one warp on item w of lattice d: a flagged site (w < nflag) or an
// interstitial.  FORCE = false: density pass; true: force + integration pass.  A
// flagged site's lattice-pair part comes from the lattice kernels (rho / f of the site);
// its interstitial pairs, df, integration and ghost images are done here.  An
// interstitial's pairs (lattice window and other interstitials) are all done here, FP64.
template <bool FORCE, bool ENERGY>
__device__ void itl_item(const EnsParams &P, const LatDesc &d, int w, int nflag) {
  const int lane = threadIdx.x & 31;
  const Geom g = lat_geom(d);
  const int cur = d.cur;
  const float4 *u4 = d.u4[cur];
  const bool is_site = w < nflag;
  long long i = 0;
  int s = 0, cx = 0, y = 0, z = 0, it = 0, ti;
  double xi, yi, zi, dfi = 0.0;
  if (is_site) {
    i = flag_list_of(d, cur)[w];
    decode_ext(g, i, s, cx, y, z);
    ti = d.code[i] & MB_TYPE_MASK;
    double X, Y, Z;
    ideal_pos(s, cx, y, z, P.a0, X, Y, Z);
    xi = X + d.ux[i];
    yi = Y + d.uy[i];
    zi = Z + d.uz[i];
    if (FORCE) dfi = (double)u4[i].w;
  } else {
    it = w - nflag;
    ti = d.itype[it];
    xi = d.ipx[cur][it];
    yi = d.ipy[cur][it];
    zi = d.ipz[cur][it];
    if (FORCE) dfi = d.idf[it];
  }
  double acc0 = 0.0, fx = 0.0, fy = 0.0, fz = 0.0, ep = 0.0;
  auto pair = [&](double dx, double dy, double dz, int tj, double dfj) {
    itl_pair<FORCE, ENERGY>(P, ti, dfi, dx, dy, dz, tj, dfj, acc0, fx, fy, fz, ep);
  };
  if (is_site) {
    // the lattice kernels summed this site's lattice pairs (FP32, compensated) into
    // rho / f; only the interstitial pairs are added here
    if (lane == 0) {
      if (FORCE) {
        fx = (double)d.fx[i];
        fy = (double)d.fy[i];
        fz = (double)d.fz[i];
      } else {
        acc0 = (double)d.rho[i];
      }
    }
  } else {
    itl_window_pairs(P, d, g, u4, xi, yi, zi, lane, 32, FORCE, pair);
  }
  itl_pairs<false>(d, g, cur, xi, yi, zi, is_site ? -1 : it, lane, pair, FORCE);
  if (!FORCE) {
    acc0 = warp_sum(acc0);
  } else {
    fx = warp_sum(fx);
    fy = warp_sum(fy);
    fz = warp_sum(fz);
    if (ENERGY) ep = warp_sum(ep);
  }
  if (lane == 0) itl_finish<FORCE, ENERGY>(P, d, g, is_site, i, s, cx, y, z, it, ti, xi, yi, zi, acc0, fx, fy, fz, ep);
}

// Flagged lattice site w of lattice d, worked by the 8-lane group of this lane (a warp
// works four sites at once; every lane of the warp takes part in the group sums, with a
// site or not): the lattice kernels summed its lattice pairs (FP32, compensated) into
// rho / f, the group adds its interstitial pairs in FP64 (lane l of the group walks cells
// l, l + 8, l + 16, l + 24 of the 27 around the site in the split kernels' cell list, or
// list entries l, l + 8, ... without one) and its first lane finishes the site.  A
// flagged site's item is a chain of dependent loads with little work, so four of them
// per warp keep four chains in flight.
template <bool FORCE, bool ENERGY>
__device__ void itl_site_group(const EnsParams &P, const LatDesc &d, int w, bool valid) {
  const int l8 = threadIdx.x & 7;
  const Geom g = lat_geom(d);
  const int cur = d.cur;
  long long i = 0;
  int s = 0, cx = 0, y = 0, z = 0, ti = 0;
  double xi = 0.0, yi = 0.0, zi = 0.0, dfi = 0.0;
  double acc0 = 0.0, fx = 0.0, fy = 0.0, fz = 0.0, ep = 0.0;
  auto pair = [&](double dx, double dy, double dz, int tj, double dfj) {
    itl_pair<FORCE, ENERGY>(P, ti, dfi, dx, dy, dz, tj, dfj, acc0, fx, fy, fz, ep);
  };
  if (valid) {
    i = flag_list_of(d, cur)[w];
    decode_ext(g, i, s, cx, y, z);
    ti = d.code[i] & MB_TYPE_MASK;
    double X, Y, Z;
    ideal_pos(s, cx, y, z, P.a0, X, Y, Z);
    xi = X + d.ux[i];
    yi = Y + d.uy[i];
    zi = Z + d.uz[i];
    if (FORCE) dfi = (double)d.u4[cur][i].w;
    if (l8 == 0) {
      if (FORCE) {
        fx = (double)d.fx[i];
        fy = (double)d.fy[i];
        fz = (double)d.fz[i];
      } else {
        acc0 = (double)d.rho[i];
      }
    }
    if (d.icount && d.iflag[0]) {
      int qx, qy, qz;
      itl_cell3(d, xi, yi, zi, qx, qy, qz);
      for (int cc = l8; cc < 27; cc += 8) {
        const int ox = cc % 3 - 1, oy = (cc / 3) % 3 - 1, oz = cc / 9 - 1;
        const int ccx = (qx + ox + d.icn[0]) % d.icn[0], ccy = (qy + oy + d.icn[1]) % d.icn[1],
                  ccz = (qz + oz + d.icn[2]) % d.icn[2];
        const int c = (ccz * d.icn[1] + ccy) * d.icn[0] + ccx;
        const int n = d.icount[c], s0 = d.istart[c];
        for (int jj = s0; jj < s0 + n; jj++) {
          const int K = d.iitem[jj];
          pair(min_image(xi - d.ipx[cur][K], g.Lx, g.iLx), min_image(yi - d.ipy[cur][K], g.Ly, g.iLy),
               min_image(zi - d.ipz[cur][K], g.Lz, g.iLz), d.itype[K], FORCE ? d.idf[K] : 0.0);
        }
      }
    } else {
      for (int K = l8; K < d.n_itl; K += 8)
        pair(min_image(xi - d.ipx[cur][K], g.Lx, g.iLx), min_image(yi - d.ipy[cur][K], g.Ly, g.iLy),
             min_image(zi - d.ipz[cur][K], g.Lz, g.iLz), d.itype[K], FORCE ? d.idf[K] : 0.0);
    }
  }
  if (!FORCE) {
    acc0 = group8_sum(acc0);
  } else {
    fx = group8_sum(fx);
    fy = group8_sum(fy);
    fz = group8_sum(fz);
    if (ENERGY) ep = group8_sum(ep);
  }
  if (valid && l8 == 0)
    itl_finish<FORCE, ENERGY>(P, d, g, true, i, s, cx, y, z, 0, ti, xi, yi, zi, acc0, fx, fy, fz, ep);
}

// Interstitial `it` of lattice d, worked by a whole block: its window's candidates are spread
// over the threads (3 or 4 each instead of 22 rounds of one warp), the first warp adds the
// other interstitials, and thread 0 sums in a fixed order and finishes.  red: 4 x 32 doubles
// of shared memory.
template <bool FORCE, bool ENERGY>
__device__ void itl_block_item(const EnsParams &P, const LatDesc &d, int it, double (*red)[32]) {
  const Geom g = lat_geom(d);
  const int cur = d.cur, ti = d.itype[it], warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const double xi = d.ipx[cur][it], yi = d.ipy[cur][it], zi = d.ipz[cur][it], dfi = FORCE ? d.idf[it] : 0.0;
  double acc0 = 0.0, fx = 0.0, fy = 0.0, fz = 0.0, ep = 0.0;
  auto pair = [&](double dx, double dy, double dz, int tj, double dfj) {
    itl_pair<FORCE, ENERGY>(P, ti, dfi, dx, dy, dz, tj, dfj, acc0, fx, fy, fz, ep);
  };
  itl_window_pairs(P, d, g, d.u4[cur], xi, yi, zi, threadIdx.x, blockDim.x, FORCE, pair);
  if (warp == 0) itl_pairs<true>(d, g, cur, xi, yi, zi, it, lane, pair, FORCE);
  double *vals[4] = {FORCE ? &fx : &acc0, &fy, &fz, &ep};
  const int n = FORCE ? (ENERGY ? 4 : 3) : 1;
  __syncthreads(); // the sums of the block's last item are read
#pragma unroll
  for (int q = 0; q < 4; q++) {
    if (q >= n) break;
    const double v = warp_sum(*vals[q]);
    if (lane == 0) red[q][warp] = v;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int q = 0; q < 4; q++) {
      if (q >= n) break;
      double v = 0.0;
      for (int k = 0; k < (int)(blockDim.x >> 5); k++) v += red[q][k];
      *vals[q] = v;
    }
    itl_finish<FORCE, ENERGY>(P, d, g, false, 0, 0, 0, 0, 0, it, ti, xi, yi, zi, acc0, fx, fy, fz, ep);
  }
}

// Items of every lattice that holds interstitials, split kernels: a block takes one
// interstitial or blockDim / 8 marked sites (8 lanes each), the interstitials first; the
// blocks start at another place of each lattice's items.
template <bool FORCE, bool ENERGY>
__device__ void itl_block_items(const EnsParams &P, double (*red)[32]) {
  const int per = blockDim.x >> 3;
  for (int q = 0; q < P.n_itl_lats; q++) {
    const LatDesc &d = P.lats[P.itl_lats[q]];
    if (!lat_active(d)) continue;
    const int nflag = min(d.flag_count[d.cur], d.cap_flag), n_itl = d.n_itl;
    const int jobs = n_itl + (nflag + per - 1) / per;
    for (int job = (blockIdx.x + 61u * (unsigned)q) % gridDim.x; job < jobs; job += gridDim.x) {
      if (job < n_itl) {
        itl_block_item<FORCE, ENERGY>(P, d, job, red);
      } else {
        const int f = (job - n_itl) * per + (int)(threadIdx.x >> 3);
        itl_site_group<FORCE, ENERGY>(P, d, f, f < nflag);
      }
    }
  }
}

// The same in the persistent kernel: one item per warp, whole interstitial lists.
template <bool FORCE, bool ENERGY>
__device__ void itl_items(const EnsParams &P) {
  const int warps = gridDim.x * (blockDim.x >> 5);
  const int gw = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  for (int q = 0; q < P.n_itl_lats; q++) {
    const LatDesc &d = P.lats[P.itl_lats[q]];
    if (!lat_active(d)) continue;
    const int nflag = min(d.flag_count[d.cur], d.cap_flag);
    const int n = nflag + d.n_itl;
    for (int w = gw; w < n; w += warps) itl_item<FORCE, ENERGY>(P, d, w, nflag);
  }
}

} // namespace mb
