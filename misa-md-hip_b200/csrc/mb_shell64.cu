// FP64 lattice passes for large launches: shell by shell, each with
// its own replicated table window in shared memory.
//
// What bounds a pass with one copy of the table is the SM's 128-byte/clock data stage: in
// a thermally disordered lattice the 32 lanes of a stencil entry look up random knots, and
// a 16-byte shared load, served 8 lanes at a time, waits for the most-used of 8 bank
// groups (2.6 lanes on average).  Here the stencil is walked shell by shell: the knots of
// one shell's distances are few enough for 8 copies, one per bank group, so that a lookup
// always takes the least number of wavefronts.  A CTA runs a batch of its items through
// one shell after the other; the partial sums of the sites rest in their rho / force
// arrays (L2) in between.  The shells are built into the code (mb_ensemble_shells.cuh), so
// that a neighbour costs one 32-byte load with an immediate column offset.
// With several types a window holds the words of every type and pair of types.
// Measured on one B200, 96^3 cells at 300 K: step 1.04 -> 0.79 ms; bank conflicts 0.15 M of
// 27.5 M shared wavefronts (density) and 0.47 M of 42.6 M (force), with one table copy over
// half; instructions per 32-site item 6,250 -> 3,820 and 5,460 -> 4,840.  The density pass is
// now at 83% of the L1TEX data stage, the force pass (63%) waits on neighbour loads (24 warps
// per SM, 80 registers).
#include <math.h>

#include "mb_pair64.cuh"

namespace mb {

#ifndef MB_SHELL_RHO_THREADS
#define MB_SHELL_RHO_THREADS 1024 // 896: step at 96^3 cells 2% slower
#endif
#ifndef MB_SHELL_FORCE_THREADS
#define MB_SHELL_FORCE_THREADS 768 // 896 and 1024 (spills): step at 96^3 cells 1% and 4% slower
#endif
#define MB_MULTI_FORCE_THREADS 640 // several types (768: spills, 512: step 2% and 6% slower)
#ifndef MB_SHELL_ROUNDS
#define MB_SHELL_ROUNDS 12 // items per warp in a batch (6: 3%, 24: 1% slower)
#endif
#define MB_AHEAD 4 // neighbour loads issued ahead (1, 2, 8: the same within 1%)
#define MB_COPIES 8
// Intervals of a window.  Density: 8 copies of 16 bytes per knot, 131 KB (860: 1% slower at
// 300 K, 2.5% at 900 K).  Force: 8 copies of 32 bytes, 162 KB, +-0.36 A with 5,000 knots
// (520: 2% slower at 300 K; 720 and more leave too little L1).
#ifndef MB_RHO_WINDOW
#define MB_RHO_WINDOW 1024
#endif
#ifndef MB_FORCE_WINDOW
#define MB_FORCE_WINDOW 648
#endif
// Several types: windows of as many intervals, in as many copies (8, 4, 2, 1) as take at most
// these bytes; the rest is L1.  Step at 48x40x44 cells, 3 types, 2,000 knots, 600 K: 171 us;
// two copies of the force window (187 KB) 196 us, of a narrower one (133 KB) 191 us; windows
// of +-0.57 and +-0.36 A in more copies 186 us.
#define MB_COPIES_BYTES (130 * 1024 + 512)

// The density pass visits neighbouring shells that share a window together: first shell of
// each visit (the force pass, with twice the bytes per knot, visits them one by one).
template <int NEAR>
struct RhoVisits {
  static constexpr int n = NEAR == 5 ? 3 : 4;
  static constexpr int first[5] = {0, 2, 3, 5, 6};
};

// Fills the window with `words` 16-byte words from src, every word `copies` times: a thread
// reads a word once and lane l starts with copy l % copies, so that the stores of 8 lanes
// fall into 8 bank groups.
__device__ __forceinline__ void fill_window(double2 *w, const double2 *src, int words, int copies) {
#pragma unroll 2
  for (int k = threadIdx.x; k < words; k += blockDim.x) {
    const double2 v = __ldg(src + k);
#pragma unroll
    for (int c = 0; c < MB_COPIES; c++)
      if (c < copies) w[k * copies + ((c + threadIdx.x) & (copies - 1))] = v;
  }
}
// The window of knots [lo, lo + cnt] of a table of `words` words per knot; the first one (SH
// == 0) is filled while the kernel before drains.
template <int COPIES, int SH>
__device__ __forceinline__ Window64<COPIES> take_window(double2 *s_w, const double2 *tab, int words, int copies, int lo,
                                                        int cnt, int &first) {
  if (COPIES > 0) copies = COPIES;
  __syncthreads();
  fill_window(s_w, tab + (size_t)words * lo, (cnt + 1) * words, copies);
  if (SH == 0) chain_wait(first);
  __syncthreads();
  return Window64<COPIES>{s_w + (threadIdx.x & (copies - 1)), MB_FLOOR - lo, (unsigned)cnt, words, copies};
}

// Bases of a site's neighbours: even vectors, and odd ones (on the other sublattice).
struct Bases64 {
  const double4 *be, *bo;
  const int8_t *ce, *co; // codes (several types)
};
__device__ __forceinline__ Bases64 site_bases(const Geom &g, const Lattice64 &L, int i) {
  const int odd = i < (int)g.E ? (int)g.E : -(int)g.E + g.ey * g.ecx + g.ecx + 1;
  return Bases64{L.p + i, L.p + i + odd, L.code + i, L.code + i + odd};
}
template <int K>
__device__ __forceinline__ double4 ld_neighbour(const Bases64 &b, int pl, int rw) {
  using T = HStore<K>;
  return ld_site((T::odd ? b.bo : b.be) + (T::dz * pl + T::dy * rw) + T::dx);
}
template <int K, int COPIES>
__device__ __forceinline__ int neighbour_type(const Bases64 &b, int pl, int rw, int nt) {
  using T = HStore<K>;
  return COPIES > 0 ? 0 : type_at((T::odd ? b.co : b.ce) + (T::dz * pl + T::dy * rw) + T::dx, nt);
}

// Items of a launch in rounds: of the CTA's warps as many take an item in each round as
// spread the items evenly over the least number of rounds.  A batch is a range of rounds; a
// warp's items of it are lo, lo + stride, ... below hi.
struct Rounds64 {
  int rounds, warps, batches;
};
__device__ __forceinline__ Rounds64 launch_rounds(const LatticeArgs &a) {
  Rounds64 r;
  const int n = a.n_items - a.w0, cap = gridDim.x * (blockDim.x >> 5);
  r.rounds = (n + cap - 1) / cap;
  const int share = gridDim.x * r.rounds;
  r.warps = (n + share - 1) / share; // 37 x 52 x 45 cells: step 156 -> 136 us, 64^3 303 -> 281
  r.batches = (r.rounds + MB_SHELL_ROUNDS - 1) / MB_SHELL_ROUNDS;
  return r;
}
struct BatchItems {
  int lo, hi, stride;
};
__device__ __forceinline__ BatchItems batch_items(const LatticeArgs &a, int b, const Rounds64 &r) {
  const int stride = gridDim.x * r.warps, warp = threadIdx.x >> 5;
  const int lo = a.w0 + r.rounds * b / r.batches * stride + (int)blockIdx.x * r.warps + warp;
  const int hi = min(a.n_items, a.w0 + r.rounds * (b + 1) / r.batches * stride);
  return BatchItems{lo, warp < r.warps ? hi : lo, stride};
}

// This lane's entry of item w in the site list (none past the end of the batch).
__device__ __forceinline__ int item_ref(const LatticeArgs &a, int w, int hi) {
  return w < hi ? __ldg(a.sites + 32 * (size_t)w + (threadIdx.x & 31)) : -1;
}

// Density sums of shell SH's runs.
template <int SH, int COPIES>
__device__ __forceinline__ void rho_shell(const LatticeArgs &a, const Window64<COPIES> &W, const Site64 &c,
                                          const Bases64 &b, int pl, int rw, double &rho) {
  constexpr int first = kBcc.start[SH], end = kBcc.start[SH + 1];
  static_for<0, (end - first + MB_RUN - 1) / MB_RUN>([&](auto rc) {
    constexpr int k0 = first + decltype(rc)::value * MB_RUN, k1 = k0 + MB_RUN < end ? k0 + MB_RUN : end;
    double t = 0.0;
    unsigned far = 0;
    static_for<0, (k1 - k0 + MB_AHEAD - 1) / MB_AHEAD>([&](auto cc) {
      constexpr int c0 = k0 + decltype(cc)::value * MB_AHEAD, c1 = c0 + MB_AHEAD < k1 ? c0 + MB_AHEAD : k1;
      double4 q[MB_AHEAD];
      int tj[MB_AHEAD];
      static_for<c0, c1>([&](auto kc) {
        constexpr int k = decltype(kc)::value;
        q[k - c0] = ld_neighbour<k>(b, pl, rw);
        tj[k - c0] = neighbour_type<k, COPIES>(b, pl, rw, a.P.n_types);
      });
      static_for<c0, c1>([&](auto kc) {
        constexpr int k = decltype(kc)::value;
        rho_near(a, W, c, q[k - c0], tj[k - c0], k - k0, t, far);
      });
    });
    rho_far(a, c, k0, far, t);
    rho = __dadd_rn(rho, t);
  });
}

template <int SH, int COPIES, bool ENERGY>
__device__ __forceinline__ void force_shell(const LatticeArgs &a, const Window64<COPIES> &W, const Site64 &c,
                                            const Bases64 &b, int pl, int rw, double &fx, double &fy, double &fz,
                                            double &ep) {
  constexpr int first = kBcc.start[SH], end = kBcc.start[SH + 1];
  static_for<0, (end - first + MB_RUN - 1) / MB_RUN>([&](auto rc) {
    constexpr int k0 = first + decltype(rc)::value * MB_RUN, k1 = k0 + MB_RUN < end ? k0 + MB_RUN : end;
    double tx = 0.0, ty = 0.0, tz = 0.0;
    unsigned far = 0;
    static_for<0, (k1 - k0 + MB_AHEAD - 1) / MB_AHEAD>([&](auto cc) {
      constexpr int c0 = k0 + decltype(cc)::value * MB_AHEAD, c1 = c0 + MB_AHEAD < k1 ? c0 + MB_AHEAD : k1;
      double4 q[MB_AHEAD];
      int tj[MB_AHEAD];
      static_for<c0, c1>([&](auto kc) {
        constexpr int k = decltype(kc)::value;
        q[k - c0] = ld_neighbour<k>(b, pl, rw);
        tj[k - c0] = neighbour_type<k, COPIES>(b, pl, rw, a.P.n_types);
      });
      static_for<c0, c1>([&](auto kc) {
        constexpr int k = decltype(kc)::value;
        force_near<COPIES, ENERGY>(a, W, c, q[k - c0], tj[k - c0], k - k0, tx, ty, tz, ep, far);
      });
    });
    force_far<ENERGY>(a, c, k0, far, tx, ty, tz, ep);
    fx = __dadd_rn(fx, tx);
    fy = __dadd_rn(fy, ty);
    fz = __dadd_rn(fz, tz);
  });
}

// NEAR: shells inside the cutoff at the ideal lattice.  COPIES: table copies; 0 with several types.
template <bool ENERGY, int NEAR, int COPIES>
__global__ void __launch_bounds__(MB_SHELL_RHO_THREADS, 1)
    k_shell_rho64(const __grid_constant__ StencilSet st, const __grid_constant__ LatticeArgs a) {
  extern __shared__ double2 s_w[];
  const Lattice64 &L = a.L;
  constexpr int n_near = kBcc.start[NEAR];
  const int lane = threadIdx.x & 31, pl = a.g.ey * a.g.ecx, rw = a.g.ecx;
  chain_next();
  const Rounds64 rd = launch_rounds(a);
  double e_acc = 0.0;
  for (int b = 0; b < rd.batches; b++) {
    BatchItems it = batch_items(a, b, rd);
    static_for<0, RhoVisits<NEAR>::n>([&](auto vc) {
      constexpr int V = decltype(vc)::value, SH = RhoVisits<NEAR>::first[V], END = RhoVisits<NEAR>::first[V + 1];
      const int lo = a.sh.rho.lo[SH], cnt = a.sh.rho.cnt[SH];
      const Window64<COPIES> W =
          take_window<COPIES, SH>(s_w, a.P.f_ys, COPIES > 0 ? 1 : a.P.n_types, a.copies, lo, cnt, it.lo);
      int next = item_ref(a, it.lo, it.hi);
      for (int w = it.lo; w < it.hi; w += it.stride) {
        const int ref = next, i = ref & MB_SITE_INDEX;
        next = item_ref(a, w + it.stride, it.hi); // under way while this item is worked on
        int code = -1;
        double4 own;
        double rho = 0.0;
        if (ref >= 0) { // three loads at once, before the code is looked at
          code = L.code[i];
          own = ld_site(L.p + i);
          if (SH) rho = L.rho[i];
        }
        unsigned long long near = 0;
        if (code >= 0) {
          const Site64 c{L.p + i, L.code + i, st.off[i >= (int)a.g.E], own.x, own.y, own.z, 0.0, 0};
          const Bases64 bs = site_bases(a.g, L, i);
          static_for<SH, END>([&](auto hc) { rho_shell<decltype(hc)::value, COPIES>(a, W, c, bs, pl, rw, rho); });
          if (END < NEAR) {
            L.rho[i] = rho;
          } else {
            for (int k0 = n_near; k0 < st.n; k0 += MB_OUT_RUN) {
              unsigned m = 0;
              rho = __dadd_rn(rho, rho_outer(a, c, k0, min(k0 + MB_OUT_RUN, st.n), m));
              near |= (unsigned long long)m << (k0 - n_near);
            }
            const double e = rho_finish64<ENERGY>(a.g, a.P, L, code, a.flag, ref, rho);
            if (ENERGY) e_acc += e;
          }
        }
        if (END == NEAR && a.outer) {
          const unsigned lo = __reduce_or_sync(0xffffffffu, (unsigned)near);
          const unsigned hi = __reduce_or_sync(0xffffffffu, (unsigned)(near >> 32));
          if (lane == 0) a.outer[w] = make_uint2(lo, hi);
        }
      }
    });
  }
  if (ENERGY) {
    const double t = block_sum(e_acc);
    if (threadIdx.x == 0) a.e0[blockIdx.x] = t;
  }
}

template <bool ENERGY, int NEAR, int COPIES>
__global__ void __launch_bounds__(COPIES > 0 ? MB_SHELL_FORCE_THREADS : MB_MULTI_FORCE_THREADS, 1)
    k_shell_force64(const __grid_constant__ StencilSet st, const __grid_constant__ LatticeArgs a) {
  extern __shared__ double2 s_w[];
  const Lattice64 &L = a.L;
  constexpr int n_near = kBcc.start[NEAR];
  const int lane = threadIdx.x & 31, pl = a.g.ey * a.g.ecx, rw = a.g.ecx;
  chain_next();
  const Rounds64 rd = launch_rounds(a);
  double e_pair = 0.0, e_kin = 0.0;
  for (int b = 0; b < rd.batches; b++) {
    BatchItems it = batch_items(a, b, rd);
    static_for<0, NEAR>([&](auto shc) {
      constexpr int SH = decltype(shc)::value;
      const int lo = a.sh.force.lo[SH], cnt = a.sh.force.cnt[SH];
      const Window64<COPIES> W =
          take_window<COPIES, SH>(s_w, a.P.force2, COPIES > 0 ? 2 : force_words(a.P.n_types), a.copies, lo, cnt, it.lo);
      int next = item_ref(a, it.lo, it.hi);
      for (int w = it.lo; w < it.hi; w += it.stride) {
        const int ref = next, i = ref & MB_SITE_INDEX;
        next = item_ref(a, w + it.stride, it.hi);
        if (ref < 0) continue;
        const int code = L.code[i];
        const double4 own = ld_site(L.p + i);
        double fx = 0.0, fy = 0.0, fz = 0.0;
        if (SH) {
          fx = L.fx[i];
          fy = L.fy[i];
          fz = L.fz[i];
        }
        if (code < 0) continue;
        const Site64 c{L.p + i, L.code + i, st.off[i >= (int)a.g.E], own.x, own.y, own.z, own.w,
                       COPIES > 0 ? 0 : code & MB_TYPE_MASK};
        force_shell<SH, COPIES, ENERGY>(a, W, c, site_bases(a.g, L, i), pl, rw, fx, fy, fz, e_pair);
        if (SH + 1 < NEAR) {
          L.fx[i] = fx;
          L.fy[i] = fy;
          L.fz[i] = fz;
        } else {
          unsigned long long mask = ~0ull;
          if (a.outer) {
            const uint2 m2 = a.outer[w];
            mask = (unsigned long long)m2.x | ((unsigned long long)m2.y << 32);
          }
          for (int k0 = n_near; k0 < st.n; k0 += MB_OUT_RUN) {
            const unsigned bits = (unsigned)(mask >> (k0 - n_near)) & ((1u << MB_OUT_RUN) - 1u);
            if (!bits) continue;
            double tx, ty, tz;
            force_outer<ENERGY>(a, c, k0, min(k0 + MB_OUT_RUN, st.n), false, bits, tx, ty, tz, e_pair);
            fx = __dadd_rn(fx, tx);
            fy = __dadd_rn(fy, ty);
            fz = __dadd_rn(fz, tz);
          }
          const double ek = force_finish64<ENERGY>(a.g, L, a.sp, code & a.flag, ref, c, fx, fy, fz);
          if (ENERGY) e_kin += ek;
        }
      }
    });
  }
  if (ENERGY) {
    const double t1 = block_sum(e_pair);
    if (threadIdx.x == 0) a.e0[blockIdx.x] = t1;
    const double t2 = block_sum(e_kin);
    if (threadIdx.x == 0) a.e1[blockIdx.x] = t2;
  }
}

static size_t window_bytes(const Windows64 &w, int n, int words, int copies) {
  int knots = 0;
  for (int h = 0; h < n; h++) knots = w.cnt[h] + 1 > knots ? w.cnt[h] + 1 : knots;
  return (size_t)knots * words * copies * sizeof(double2);
}

template <int NEAR, int COPIES>
static int shell_rho(const StencilSet &st, LatticeArgs a, int energy, cudaStream_t s) {
  MB_SMEM_ATTR((k_shell_rho64<false, NEAR, COPIES>), (k_shell_rho64<true, NEAR, COPIES>), MB_SMEM_MAX - 1024);
  a.copies = a.sh.rho.copies;
  const size_t smem = window_bytes(a.sh.rho, a.sh.n, a.P.n_types, a.copies);
  return launch_chained(a.chain, energy ? k_shell_rho64<true, NEAR, COPIES> : k_shell_rho64<false, NEAR, COPIES>,
                        device_sm_count(), MB_SHELL_RHO_THREADS, smem, s, st, a);
}
template <int NEAR, int COPIES>
static int shell_force(const StencilSet &st, LatticeArgs a, int energy, cudaStream_t s) {
  MB_SMEM_ATTR((k_shell_force64<false, NEAR, COPIES>), (k_shell_force64<true, NEAR, COPIES>), MB_SMEM_MAX - 1024);
  a.copies = a.sh.force.copies;
  const size_t smem = window_bytes(a.sh.force, a.sh.n, force_words(a.P.n_types), a.copies);
  const int threads = COPIES > 0 ? MB_SHELL_FORCE_THREADS : MB_MULTI_FORCE_THREADS;
  return launch_chained(a.chain, energy ? k_shell_force64<true, NEAR, COPIES> : k_shell_force64<false, NEAR, COPIES>,
                        device_sm_count(), threads, smem, s, st, a);
}

int launch_shell_rho64(const StencilSet &st, const LatticeArgs &a, int energy, cudaStream_t s) {
  if (a.P.n_types == 1)
    return a.sh.n == 5 ? shell_rho<5, MB_COPIES>(st, a, energy, s) : shell_rho<6, MB_COPIES>(st, a, energy, s);
  return a.sh.n == 5 ? shell_rho<5, 0>(st, a, energy, s) : shell_rho<6, 0>(st, a, energy, s);
}
int launch_shell_force64(const StencilSet &st, const LatticeArgs &a, int energy, cudaStream_t s) {
  if (a.P.n_types == 1)
    return a.sh.n == 5 ? shell_force<5, MB_COPIES>(st, a, energy, s) : shell_force<6, MB_COPIES>(st, a, energy, s);
  return a.sh.n == 5 ? shell_force<5, 0>(st, a, energy, s) : shell_force<6, 0>(st, a, energy, s);
}

// ------------------------------------------------------------------ plan
// Least margin of a window around its shells' ideal distances: atoms displaced by 0.07 A
// per component (300 K) put a pair 0.1 A (rms) off its ideal distance.
#define MB_WINDOW_MARGIN 0.25 // A

// Window of `cap` intervals around the distances r0 .. r1; false when it cannot hold the
// least margin.  It ends inside the cutoff, so that a pair in the window is inside it too.
static bool shell_window(const DevPot &P, double cutoff, double r0, double r1, int cap, int &lo, int &cnt) {
  const int inside = (int)floor(cutoff * P.rdr) - 1; // knots inside the cutoff
  const int mid = (int)(0.5 * (r0 + r1) * P.rdr);
  int hi = mid + cap / 2;
  lo = mid - cap / 2;
  if (lo < 0) lo = 0;
  if (hi > inside) hi = inside;
  if (hi > P.nr - 1) hi = P.nr - 1;
  cnt = hi - lo;
  return cnt > 0 && 0.5 * cap >= (0.5 * (r1 - r0) + MB_WINDOW_MARGIN) * P.rdr;
}

__global__ void k_site_list(const Geom g, int cpp, int *sites) {
  const long long n = 64LL * g.bz * cpp;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < n; t += (long long)gridDim.x * blockDim.x)
    sites[t] = site_ref64(g, (int)(t >> 5), (int)(t & 31));
}

int plan64_items(const Geom &g) { return 2 * g.bz * plan64_plane_items(g); }
int plan64_plane_items(const Geom &g) { return (g.bcx * g.by + 31) / 32; }

// R: the ideal distances of the (sorted) entries.  The plan applies when the near entries
// are exactly BCC shells 1-5 or 1-6 in the order of mb_ensemble_shells.cuh, the ghost
// frame is 2 cells wide, and the knots are coarse enough for windows of at least the least
// margin (finer tables would read global memory too often).
bool plan64_shells(const DevPot &P, const Geom &g, double a0, double cutoff, const double *R, const StencilSet &st,
                   Shells64 &S) {
  S = Shells64{};
  S.n = st.n_near == kBcc.start[5] ? 5 : st.n_near == kBcc.start[6] ? 6 : 0;
  if (!S.n || st.n - st.n_near > 64 || g.E > 0x1fffffffLL) return false;
  double r[MB_NEAR_SHELLS];
  for (int h = 0; h < S.n; h++) {
    r[h] = 0.5 * a0 * sqrt((double)kBcc.n2[h]);
    for (int k = kBcc.start[h]; k < kBcc.start[h + 1]; k++) {
      const HVec v = kBcc.v[k];
      if (fabs(R[k] - r[h]) > 1e-9 * r[h]) return false;
      for (int s = 0; s < 2; s++) { // the offsets are those built into the code
        const int s2 = (s + v.hx) & 1;
        const int dx = (v.hx + s - s2) / 2, dy = (v.hy + s - s2) / 2, dz = (v.hz + s - s2) / 2;
        if (st.off[s][k] != (s2 - s) * (int)g.E + (dz * g.ey + dy) * g.ecx + dx) return false;
      }
    }
    for (int k = kBcc.start[h]; k < kBcc.start[h + 1]; k += MB_RUN) {
      S.shell[S.runs] = (short)h;
      S.kb[S.runs++] = (short)k;
    }
  }
  // windows: one type as measured; several in the most copies that leave the least margin
  const int *first = RhoVisits<5>::first; // the visits of NEAR = 6 begin with the same shells
  auto windows = [&](Windows64 &w, int words, int most, auto fit) {
    const int knot = words * (int)sizeof(double2);
    w.copies = MB_COPIES; // built into the one-type kernels
    if (P.n_types > 1)
      while (w.copies > 1 && (most + 1) * knot * w.copies > MB_COPIES_BYTES) w.copies /= 2;
    const int room = (MB_SMEM_MAX - 2048) / (knot * w.copies) - 1;
    return fit(room < most ? room : most);
  };
  const bool rho = windows(S.rho, P.n_types, MB_RHO_WINDOW, [&](int cap) {
    for (int v = 0; first[v] < S.n; v++)
      for (int h = first[v]; h < first[v + 1]; h++)
        if (!shell_window(P, cutoff, r[first[v]], r[first[v + 1] - 1], cap, S.rho.lo[h], S.rho.cnt[h])) return false;
    return true;
  });
  const bool force = windows(S.force, force_words(P.n_types), MB_FORCE_WINDOW, [&](int cap) {
    for (int h = 0; h < S.n; h++)
      if (!shell_window(P, cutoff, r[h], r[h], cap, S.force.lo[h], S.force.cnt[h])) return false;
    return true;
  });
  if (!rho || !force) return false;
  S.near_runs = S.runs;
  for (int k = st.n_near; k < st.n; k += MB_OUT_RUN) S.kb[S.runs++] = (short)k;
  S.kb[S.runs] = (short)st.n;
  return split64_fits(P, S);
}

int plan64_sites(const Geom &g, int *sites, cudaStream_t s) {
  k_site_list<<<8 * device_sm_count(), 256, 0, s>>>(g, plan64_plane_items(g), sites);
  MB_CUDA(cudaGetLastError());
  return MB_OK;
}

} // namespace mb
