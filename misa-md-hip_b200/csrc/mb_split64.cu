// FP64 lattice passes for small launches: one item's stencil split
// over the warps of a group.
//
// A launch of a few items per SM leaves most warps idle, and its time is the latency of
// one warp walking ~90 entries, each a chain of neighbour load, root, table load and sum.
// Here MB_SPLIT_WARPS warps share an item: each takes whole runs of the site's sum
// (mb_pair64.cuh), leaves the run sums in shared memory and one warp, another for each item,
// adds them in order and finishes the sites while the others go on to the next item.  The
// run sums and their order are those of the shell-window kernels, so both give the same bits.
// One copy of the table serves: the warps in flight are too few for bank conflicts to count.
// The tables of several types that are too wide for shared memory are read where they lie.
// Measured on one B200, 20^3 cells: step 73 -> 27 us (one type), 81 -> 36 us (three).
#include "mb_pair64.cuh"

namespace mb {

#define MB_SPLIT_WARPS 8 // warps per item: the 58 near entries of shells 1-5 make 8 runs
#ifndef MB_SPLIT_GROUPS
#define MB_SPLIT_GROUPS 4 // items a CTA works on at once
#endif
#define MB_SPLIT_THREADS (32 * MB_SPLIT_WARPS * MB_SPLIT_GROUPS)

__device__ __forceinline__ void group_sync(int group) {
  asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "r"(32 * MB_SPLIT_WARPS) : "memory");
}

// The knots of every shell window, one copy.
__device__ __forceinline__ void fill_table(double2 *w, const double2 *tab, int words) {
  for (int k = threadIdx.x; k < words; k += blockDim.x) w[k] = __ldg(tab + k);
}

// A lane's site in item w.
struct SplitSite {
  int ref, code;
  Site64 c;
};
__device__ __forceinline__ SplitSite split_site(const StencilSet &st, const LatticeArgs &a, int w) {
  SplitSite t;
  t.ref = a.sites ? __ldg(a.sites + 32 * (size_t)w + (threadIdx.x & 31)) : site_ref64(a.g, w, threadIdx.x & 31);
  const int i = t.ref & MB_SITE_INDEX;
  const int code = t.ref < 0 ? -1 : a.L.code[i];
  t.code = code;
  if (code < 0) {
    t.ref = -1;
    t.c = Site64{a.L.p, a.L.code, st.off[0], 0.0, 0.0, 0.0, 0.0, 0};
  } else {
    const double4 own = ld_site(a.L.p + i);
    t.c = Site64{a.L.p + i, a.L.code + i,  st.off[i >= (int)a.g.E],          own.x, own.y, own.z,
                 own.w,     a.P.n_types == 1 ? 0 : code & MB_TYPE_MASK};
  }
  return t;
}

template <int COPIES>
__device__ __forceinline__ int split_type(const Site64 &c, int k, int nt) {
  return COPIES > 0 ? 0 : type_at(c.c + c.off[k], nt);
}

// COPIES: 1, or 0 with several types; knots == 0: the table is read where it lies (several
// types, too wide for shared memory).
template <bool ENERGY, int COPIES>
__global__ void __launch_bounds__(MB_SPLIT_THREADS, 1)
    k_split_rho64(const __grid_constant__ StencilSet st, const __grid_constant__ LatticeArgs a, int lo, int knots) {
  extern __shared__ double2 s_w[];
  __shared__ double s_sum[MB_SPLIT_GROUPS][2][MB_RUNS_MAX][32]; // two items' sums, in turn
  __shared__ unsigned s_near[MB_SPLIT_GROUPS][2][MB_RUNS_MAX];
  chain_next();
  const int words = COPIES > 0 ? 1 : a.P.n_types;
  const double2 *tab = a.P.f_ys + (size_t)words * lo;
  if (COPIES > 0 || knots > 0) {
    fill_table(s_w, tab, words * knots);
    tab = s_w;
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = (threadIdx.x >> 5) % MB_SPLIT_WARPS,
            group = threadIdx.x / (32 * MB_SPLIT_WARPS);
  double e_acc = 0.0;
  int turn = 0, w0 = a.w0 + blockIdx.x * MB_SPLIT_GROUPS + group;
  chain_wait(w0);
  for (int w = w0; w < a.n_items; w += gridDim.x * MB_SPLIT_GROUPS, turn++) {
    double(*sums)[32] = s_sum[group][turn & 1];
    unsigned *nears = s_near[group][turn & 1];
    const SplitSite t = split_site(st, a, w);
    for (int r = warp; r < a.sh.runs; r += MB_SPLIT_WARPS) {
      const int k0 = a.sh.kb[r], k1 = a.sh.kb[r + 1];
      double sum = 0.0;
      unsigned near = 0;
      if (t.ref >= 0) {
        if (r < a.sh.near_runs) {
          const int h = a.sh.shell[r];
          const int wl = a.sh.rho.lo[h];
          const Window64<COPIES> W{tab + words * (wl - lo), MB_FLOOR - wl, (unsigned)a.sh.rho.cnt[h], words, 1};
          unsigned far = 0;
#pragma unroll 4
          for (int k = k0; k < k1; k++)
            rho_near(a, W, t.c, ld_site(t.c.p + t.c.off[k]), split_type<COPIES>(t.c, k, a.P.n_types), k - k0, sum, far);
          rho_far(a, t.c, k0, far, sum);
        } else {
          sum = rho_outer(a, t.c, k0, k1, near);
        }
      }
      sums[r][lane] = sum;
      if (r >= a.sh.near_runs && a.outer) {
        near = __reduce_or_sync(0xffffffffu, near);
        if (lane == 0) nears[r] = near;
      }
    }
    // one barrier an item: the sums of the item before last were read before the last one
    group_sync(group);
    if (warp == turn % MB_SPLIT_WARPS) {
      if (t.ref >= 0) {
        double rho = 0.0;
        for (int r = 0; r < a.sh.runs; r++) rho = __dadd_rn(rho, sums[r][lane]);
        const double e = rho_finish64<ENERGY>(a.g, a.P, a.L, t.code, a.flag, t.ref, rho);
        if (ENERGY) e_acc += e;
      }
      if (a.outer && lane == 0) {
        unsigned long long m = 0;
        for (int r = a.sh.near_runs; r < a.sh.runs; r++)
          m |= (unsigned long long)nears[r] << (a.sh.kb[r] - a.sh.kb[a.sh.near_runs]);
        a.outer[w] = make_uint2((unsigned)m, (unsigned)(m >> 32));
      }
    }
  }
  if (ENERGY) {
    const double t = block_sum(e_acc);
    if (threadIdx.x == 0) a.e0[blockIdx.x] = t;
  }
}

template <bool ENERGY, int COPIES>
__global__ void __launch_bounds__(MB_SPLIT_THREADS, 1)
    k_split_force64(const __grid_constant__ StencilSet st, const __grid_constant__ LatticeArgs a, int lo, int knots) {
  extern __shared__ double2 s_w[]; // table, then the run sums
  chain_next();
  const int words = COPIES > 0 ? 2 : force_words(a.P.n_types);
  const double2 *tab = a.P.force2 + (size_t)words * lo;
  if (COPIES > 0 || knots > 0) {
    fill_table(s_w, tab, words * knots);
    tab = s_w;
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = (threadIdx.x >> 5) % MB_SPLIT_WARPS,
            group = threadIdx.x / (32 * MB_SPLIT_WARPS);
  double *sums = reinterpret_cast<double *>(s_w + words * knots) + (size_t)group * 2 * a.sh.runs * 96 + lane;
  double e_pair = 0.0, e_kin = 0.0;
  int turn = 0, w0 = a.w0 + blockIdx.x * MB_SPLIT_GROUPS + group;
  chain_wait(w0);
  for (int w = w0; w < a.n_items; w += gridDim.x * MB_SPLIT_GROUPS, turn++) {
    double *sum = sums + (turn & 1) * a.sh.runs * 96;
    const SplitSite t = split_site(st, a, w);
    unsigned long long mask = 0;
    if (a.outer) {
      const uint2 m2 = a.outer[w];
      mask = (unsigned long long)m2.x | ((unsigned long long)m2.y << 32);
    }
    for (int r = warp; r < a.sh.runs; r += MB_SPLIT_WARPS) {
      const int k0 = a.sh.kb[r], k1 = a.sh.kb[r + 1];
      double fx = 0.0, fy = 0.0, fz = 0.0;
      if (t.ref >= 0) {
        if (r < a.sh.near_runs) {
          const int h = a.sh.shell[r];
          const int wl = a.sh.force.lo[h];
          const Window64<COPIES> W{tab + words * (wl - lo), MB_FLOOR - wl, (unsigned)a.sh.force.cnt[h], words, 1};
          unsigned far = 0;
#pragma unroll 4
          for (int k = k0; k < k1; k++)
            force_near<COPIES, ENERGY>(a, W, t.c, ld_site(t.c.p + t.c.off[k]),
                                       split_type<COPIES>(t.c, k, a.P.n_types), k - k0, fx, fy, fz, e_pair, far);
          force_far<ENERGY>(a, t.c, k0, far, fx, fy, fz, e_pair);
        } else {
          const unsigned bits = a.outer ? (unsigned)(mask >> (k0 - a.sh.kb[a.sh.near_runs])) : 0u;
          force_outer<ENERGY>(a, t.c, k0, k1, !a.outer, bits, fx, fy, fz, e_pair);
        }
      }
      sum[r * 96] = fx;
      sum[r * 96 + 32] = fy;
      sum[r * 96 + 64] = fz;
    }
    group_sync(group);
    if (warp == turn % MB_SPLIT_WARPS && t.ref >= 0) {
      double fx = 0.0, fy = 0.0, fz = 0.0;
      for (int r = 0; r < a.sh.runs; r++) {
        fx = __dadd_rn(fx, sum[r * 96]);
        fy = __dadd_rn(fy, sum[r * 96 + 32]);
        fz = __dadd_rn(fz, sum[r * 96 + 64]);
      }
      const double ek = force_finish64<ENERGY>(a.g, a.L, a.sp, t.code & a.flag, t.ref, t.c, fx, fy, fz);
      if (ENERGY) e_kin += ek;
    }
  }
  if (ENERGY) {
    const double t1 = block_sum(e_pair);
    if (threadIdx.x == 0) a.e0[blockIdx.x] = t1;
    const double t2 = block_sum(e_kin);
    if (threadIdx.x == 0) a.e1[blockIdx.x] = t2;
  }
}

static void table_range(const Windows64 &w, int n, int &lo, int &knots) {
  int hi = 0;
  if (n == 0) { // an entry plan: no windows
    lo = knots = 0;
    return;
  }
  lo = 1 << 30;
  for (int h = 0; h < n; h++) {
    lo = w.lo[h] < lo ? w.lo[h] : lo;
    hi = w.lo[h] + w.cnt[h] > hi ? w.lo[h] + w.cnt[h] : hi;
  }
  knots = hi - lo + 1;
}

static size_t run_sum_bytes(const Shells64 &sh) { return sizeof(double) * 2 * 96 * MB_SPLIT_GROUPS * sh.runs; }
static const int kRhoSmem = MB_SMEM_MAX - 40 * 1024; // beside its static run sums
static const int kForceSmem = MB_SMEM_MAX - 2 * 1024;

// Knots of the union of the windows that shared memory takes with `used` bytes taken; 0: too
// many.
static int smem_knots(int knots, int words, size_t used, int most) {
  return used + (size_t)knots * words * sizeof(double2) <= (size_t)most ? knots : 0;
}
static int split_grid(const LatticeArgs &a) {
  const int grid = (a.n_items - a.w0 + MB_SPLIT_GROUPS - 1) / MB_SPLIT_GROUPS;
  return grid < device_sm_count() ? grid : device_sm_count();
}

// Plan of a stencil in no order and of no known lattice (the hooks): every entry is tested,
// MB_OUT_RUN to a run, and the tables are read where they lie.  A site's index leaves the top
// two bits free (MB_SITE_FACE, no site), which the hooks' own limit does not ask for.
bool plan64_entries(const Geom &g, const StencilSet &st, Shells64 &S) {
  if (st.n < 1 || st.n > MB_OUT_RUN * MB_RUNS_MAX || 2 * g.E > MB_SITE_INDEX) return false;
  S = Shells64{};
  for (int k = 0; k < st.n; k += MB_OUT_RUN) S.kb[S.runs++] = (short)k;
  S.kb[S.runs] = (short)st.n;
  return true;
}

// Whether the entry-split kernels take the plan's tables.
bool split64_fits(const DevPot &P, const Shells64 &sh) {
  int lo, rho, force;
  table_range(sh.rho, sh.n, lo, rho);
  table_range(sh.force, sh.n, lo, force);
  return run_sum_bytes(sh) <= (size_t)kForceSmem &&
         (P.n_types > 1 || (smem_knots(rho, 1, 0, kRhoSmem) && smem_knots(force, 2, run_sum_bytes(sh), kForceSmem)));
}

template <int COPIES>
static int split_rho(const StencilSet &st, const LatticeArgs &a, int energy, cudaStream_t s) {
  int lo, knots;
  table_range(a.sh.rho, a.sh.n, lo, knots);
  knots = smem_knots(knots, a.P.n_types, 0, kRhoSmem);
  const size_t smem = (size_t)knots * a.P.n_types * sizeof(double2);
  MB_SMEM_ATTR((k_split_rho64<false, COPIES>), (k_split_rho64<true, COPIES>), kRhoSmem);
  return launch_chained(a.chain, energy ? k_split_rho64<true, COPIES> : k_split_rho64<false, COPIES>, split_grid(a),
                        MB_SPLIT_THREADS, smem, s, st, a, lo, knots);
}

template <int COPIES>
static int split_force(const StencilSet &st, const LatticeArgs &a, int energy, cudaStream_t s) {
  int lo, knots;
  table_range(a.sh.force, a.sh.n, lo, knots);
  knots = smem_knots(knots, force_words(a.P.n_types), run_sum_bytes(a.sh), kForceSmem);
  const size_t smem = (size_t)knots * force_words(a.P.n_types) * sizeof(double2) + run_sum_bytes(a.sh);
  MB_SMEM_ATTR((k_split_force64<false, COPIES>), (k_split_force64<true, COPIES>), kForceSmem);
  return launch_chained(a.chain, energy ? k_split_force64<true, COPIES> : k_split_force64<false, COPIES>, split_grid(a),
                        MB_SPLIT_THREADS, smem, s, st, a, lo, knots);
}

int launch_split_rho64(const StencilSet &st, const LatticeArgs &a, int energy, cudaStream_t s) {
  return a.P.n_types == 1 ? split_rho<1>(st, a, energy, s) : split_rho<0>(st, a, energy, s);
}
int launch_split_force64(const StencilSet &st, const LatticeArgs &a, int energy, cudaStream_t s) {
  return a.P.n_types == 1 ? split_force<1>(st, a, energy, s) : split_force<0>(st, a, energy, s);
}

} // namespace mb
