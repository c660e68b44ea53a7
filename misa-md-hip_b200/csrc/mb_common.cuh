// Shared declarations of the misa_b200 library (host + device).
//
// Device layout (split by sublattice): the reference indexes a BCC lattice
// with x doubled, so neighbouring memory cells alternate between the two
// simple-cubic sublattices and every warp mixes two stencils
// (src/kernels/kernel_itl.hpp:82,86).  Here each sublattice s in {0,1} is its own
// ghost-extended (ecx, ey, ez) array, x fastest, so a warp always walks one
// stencil and every neighbour fetch is a contiguous 32-site row.  The site at
// doubled ext index ex lives in sublattice ex & 1, column ex >> 1.
#pragma once

#include <cuda_runtime.h>
#include <nvtx3/nvToolsExt.h>
#include <stdint.h>
#include <stdlib.h>

#include <atomic>
#include <string>
#include <vector>

#include "../../include/misa_b200.h"

#define MB_MAX_STENCIL 320       // per parity; the reference's full stencil is about 228
#define MB_FTM2V 9.64853321233e-3 // (eV/A)/amu -> A/fs^2
#define MB_MVV2E (1.0 / MB_FTM2V) // amu A^2/fs^2 -> eV
#define MB_VACANT_POS 1.0e30      // position given to vacant sites: every r^2 test rejects them
// Site code: type, or negative for a vacancy; two bits mark a site that has an interstitial
// within reach, one for the steps at either position buffer (a step's marks can be set while
// the last step's come off).
#define MB_TYPE_MASK 0x1F
#define MB_FLAG_ITL(cur) ((cur) ? 0x20 : 0x40)

namespace mb {

// Read-only 32-byte load through the non-coherent path (two 16-byte halves).
__device__ __forceinline__ double4 ldg4(const double4 *p) {
  const double2 a = __ldg(reinterpret_cast<const double2 *>(p));
  const double2 b = __ldg(reinterpret_cast<const double2 *>(p) + 1);
  return make_double4(a.x, a.y, b.x, b.y);
}

// 32-byte record of a site in one load / store (32-byte aligned).  The load may be moved
// across stores: only for positions that the kernel does not write (and F' only where the
// kernel does not write it).
__device__ __forceinline__ double4 ld_site(const double4 *p) {
  double4 v;
  asm("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(v.x), "=d"(v.y), "=d"(v.z), "=d"(v.w) : "l"(p));
  return v;
}
// The same for a site's float4 {u, F'} of the mixed path.
__device__ __forceinline__ float4 ld_u4(const float4 *p) {
  float4 v;
  asm("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ void st_site(double4 *p, double x, double y, double z, double w) {
  asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(x), "d"(y), "d"(z), "d"(w) : "memory");
}

// ------------------------------------------- kernels of a step, one after another
// A chained kernel starts while the kernel before it in the stream drains: it announces
// itself to its successor (chain_next), does what needs no earlier result (tables into
// shared memory) and waits (chain_wait) until all earlier kernels are done and their results
// visible.  Every thread waits before its first access to the state, so that a kernel's end
// implies the ends of all before it.  State is read with plain loads only: the non-coherent
// path is for data that no kernel of the chain writes.  `first` is an index from which the
// caller's addresses follow: it ties loads that the compiler may move to the wait.
// Measured on one B200, steps: 6^3 cells 23.9 -> 22.0 us (two kernels), 20^3 cells of the
// mixed path 43 -> 39 us (three), 48 lattices of 1.33 M sites 437 -> 425 us.
__device__ __forceinline__ void chain_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
template <class Int>
__device__ __forceinline__ void chain_wait(Int &first) {
  static_assert(sizeof(Int) == 4, "a 32-bit index");
  asm volatile("griddepcontrol.wait;" : "+r"(first)::"memory");
}
__device__ __forceinline__ void chain_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// ----------------------------------------------------------------- tracing
// NVTX range around an entry point's work (shows in Nsight timelines; costs nothing
// when no tool is attached).
struct NvtxRange {
  explicit NvtxRange(const char *name) { nvtxRangePushA(name); }
  ~NvtxRange() { nvtxRangePop(); }
  NvtxRange(const NvtxRange &) = delete;
  NvtxRange &operator=(const NvtxRange &) = delete;
};
#define MB_RANGE(name) ::mb::NvtxRange mb_nvtx_range_(name)

// ---------------------------------------------------------------- errors
void set_error(const std::string &msg);
int fail(int code, const std::string &msg);
int cuda_fail(cudaError_t e, const char *what);

#define MB_CUDA(call)                                                                                          \
  do {                                                                                                         \
    cudaError_t e_ = (call);                                                                                   \
    if (e_ != cudaSuccess) return ::mb::cuda_fail(e_, #call);                                                  \
  } while (0)

// Whether steps chain their kernels (the environment variable MB_CHAIN=0: one by one).
inline bool chain_on() {
  const char *v = getenv("MB_CHAIN");
  return !v || atoi(v) != 0;
}
// Launch of a kernel that calls chain_wait; chained: it may start early (the operation
// before it in the stream is a kernel of the same step, or anything that completes first).
template <class... P, class... A>
int launch_chained(bool chained, void (*kernel)(P...), int grid, int block, size_t smem, cudaStream_t s, A &&...args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c{};
  c.gridDim = dim3((unsigned)grid);
  c.blockDim = dim3((unsigned)block);
  c.dynamicSmemBytes = smem;
  c.stream = s;
  c.attrs = &attr;
  c.numAttrs = chained ? 1 : 0;
  MB_CUDA(cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...));
  return MB_OK;
}

#define MB_TRY(call)                                                                                           \
  do {                                                                                                         \
    int rc_ = (call);                                                                                          \
    if (rc_ != MB_OK) return rc_;                                                                              \
  } while (0)

// ------------------------------------------------------------ potential
// Per-knot cubic pieces.  value(p) = ((c3 p + c2) p + s) p + y on [m, m+1];
// d/dx value = (d2 p + d1) p + d0 with d = (s, 2 c2, 3 c3) / dx.
struct DevPot {
  int n_types, nr, nrho;
  double rdr, rdrho, rho_max, cutoff;
  const double4 *f_val;   // [nt][nr]   {y, s, c2, c3}
  const double4 *f_der;   // [nt][nr]   {d0, d1, d2, 0}
  const double4 *F_val;   // [nt][nrho]
  const double4 *F_der;   // [nt][nrho]
  const double4 *phi_val; // [np][nr]
  const double4 *phi_der; // [np][nr]
  const double2 *force1;  // single type: [nr][3] {f d0, phi d0}, {f d1, phi d1}, {f d2, phi d2}
  // knot form: an interval takes its own knot and the next one
  const double2 *f_ys;    // [nr][nt] {y, s} of f (a cubic Hermite piece)
  const double2 *force2;  // one type: [nr][2] {f d0, phi d0}, {f d2, phi d2}; several:
                          // [nr][nt + np] {f d0, f d2} per type, {phi d0, phi d2} per pair
  // single precision copies for the mixed path
  const float4 *f_val32;   // [nt][nr]  {y, s, c2, c3}
  const float2 *force32;   // single type: [nr][3] {f d0, phi d0}, {f d1, phi d1}, {f d2, phi d2}
  const float4 *phi_val32; // single type: [nr]
  // single type, squared-distance form for the mixed split kernels, on uniform grids in
  // s = r^2, built from the FP64 r-spline and interpolated linearly.  Density: per
  // interval {value at s_j, rise over the interval}.
  // Force: per knot {A, B} = {f'(r) / r, phi'(r) / r} (knot pairs are read, which
  // halves the table against per-interval storage and allows a finer grid).
  // n_rs = n_fs = 0 when not built (several types).
  int n_rs;            // density intervals
  double ds_r;
  const float2 *fs32;  // [n_rs]
  int n_fs;            // force intervals
  double ds_f;
  const float2 *ab32;  // [n_fs + 1] knots
  const float4 *ps32;  // [n_fs] per interval cubic of phi in p (energy steps)
};

struct PotHost;
int pot_build(const mb_eam_tables *t, PotHost **out);
void pot_free(PotHost *p);
const DevPot &pot_dev(const PotHost *p);

// ------------------------------------------------------------- geometry
struct Geom {
  int ecx, ey, ez; // ext size per sublattice
  int gcx, gy, gz; // ghost widths (cells along x)
  int bcx, by, bz; // box size per sublattice
  int images;      // 1: sites write their periodic ghost images (device-resident mode)
  int zimg;        // with images: 1 also along z; 0 for a z-slab of a larger lattice, whose
                   // z ghost layers come from the neighbouring slabs
  long long E;     // sites per sublattice array
  double Lx, Ly, Lz;
  double iLx, iLy, iLz; // 1 / L (0 when there is no periodic box)
};

struct StencilSet {
  int n;                          // entries per parity (equal for both)
  int n_near;                     // leading entries inside the cutoff at the ideal lattice (0: unknown)
  int off[2][MB_MAX_STENCIL];     // [sublattice] split-layout linear offsets
};

// Convert reference-style doubled-x linear offsets to split-layout offsets.
// parity_of_sublattice[s] selects which reference stencil (0 even, 1 odd) the sites
// of sublattice s walk.
int stencil_from_linear(const int64_t *even, size_t n_even, const int64_t *odd, size_t n_odd, int ext_x, int ext_y,
                        const Geom &g, const int parity_of_sublattice[2], StencilSet *out);
// BCC stencil of every site with ideal distance < reach (doubled-x linear form,
// ordered dz, dy, dx ascending), for an ext array of ext_x x ext_y.
int stencil_generate(double a0, double reach, int ext_x, int ext_y, int64_t *even, int64_t *odd, int cap, int *n,
                     int *reach_x, int *reach_y, int *reach_z);
int stencil_sort_by_distance(double a0, double cutoff, int ext_x, int ext_y, int64_t *even, int64_t *odd, int n,
                             int *n_near, double *dist = nullptr);

// Shell windows and summation runs of a stencil whose near entries are BCC shells
// (mb_pair64.cuh, mb_shell64.cu): near shell h looks up the table intervals lo[h] ..
// lo[h] + cnt[h] - 1 of the density window and of the force window; run r holds the
// entries [kb[r], kb[r + 1]), the first near_runs of them near ones of shell[r].
#define MB_NEAR_SHELLS 6
#define MB_RUNS_MAX 16
#define MB_RUN 8      // near entries per run
#define MB_OUT_RUN 16 // outer entries per run
struct Windows64 {
  int lo[MB_NEAR_SHELLS], cnt[MB_NEAR_SHELLS];
  int copies; // of every word in shared memory
};
struct Shells64 {
  int n, runs, near_runs;
  Windows64 rho, force;
  short kb[MB_RUNS_MAX + 1], shell[MB_RUNS_MAX];
};
struct Plan64 {
  bool ok; // the stencil and tables suit the shell-window and entry-split kernels
  bool entries; // every entry is tested, items are always split (plan64_entries); no site list
  bool chain; // launches join the chain of a resident step (launch_chained)
  Shells64 sh;
  int *sites; // site list of the work items
};
// R: ideal distance of the entries of `st` (sorted).  False when the kernels do not apply.
struct StencilSet;
bool plan64_shells(const DevPot &P, const Geom &g, double a0, double cutoff, const double *R, const StencilSet &st,
                   Shells64 &S);
bool plan64_entries(const Geom &g, const StencilSet &st, Shells64 &S);
int plan64_plane_items(const Geom &g); // work items of one (z, sublattice) plane
int plan64_items(const Geom &g);       // ... of the box
int plan64_sites(const Geom &g, int *sites, cudaStream_t s);
bool split64_fits(const DevPot &P, const Shells64 &sh);
// 16-byte words per knot of the force tables (DevPot::force2).
__host__ __device__ __forceinline__ int force_words(int n_types) {
  return n_types == 1 ? 2 : n_types + n_types * (n_types + 1) / 2;
}

// ------------------------------------------------------ kernel arguments
struct Lattice64 {
  double4 *p;           // {x, y, z, F'(rho)} of every site (ext), 32-byte aligned
  int8_t *code;         // type, < 0 vacant, MB_FLAG_ITL bits
  double *rho;          // optional rho output (ext) or nullptr
  double *vx, *vy, *vz; // velocities (box sites used)
  double *fx, *fy, *fz; // forces (box sites used)
  double4 *n;           // records whose positions the drift writes (ext) or nullptr
};

struct Itl64 {
  int n;                   // count, when nd is null (lists fixed by the host)
  const int *nd;           // device-resident count (lists that change on the device), or null
  int cap;                 // capacity of the list
  int cap_flag;
  double *px, *py, *pz;    // current positions
  double *nx, *ny, *nz;    // next positions
  double *vx, *vy, *vz, *fx, *fy, *fz, *rho, *df;
  int8_t *type;
  int64_t *id;
  int flag;                // this step's mark in the site codes
  int *flag_list, *flag_count; // sites marked this step (ext index)
  int *old_list, *old_count;   // ... and last step, whose marks are the other bit
  int *overflow;               // set when a list is too short
  double a0, reach;        // window radius in A (cutoff + skin)
};

struct StepParams {
  double rc2;
  double h;      // 0.5 * dt * ftm2v / mass
  double dt;
  double mass;
  int kick_pre;  // 1: v += h f before the energy sample (closes the previous step)
  int drift;     // 1: v += h f ; x_next = x + dt v
  // lattice -> interstitial conversion (conv2 > 0): sites whose drifted atom lies
  // farther than sqrt(conv2) from the ideal site are listed in cand (box index)
  double a0, conv2;
  long long *cand;
  int *cand_n;
};
#define MB_CAND_CAP 2048     // conversion candidates handled per step
#define MB_CONV_ITL_MAX 65536 // interstitial capacity with conversion on

// Ideal position of box site (s, cx, y, z): x doubled = 2 cx + s.
__host__ __device__ __forceinline__ void site_ideal(int s, int cx, int y, int z, double a0, double &X, double &Y,
                                                    double &Z) {
  const double h = 0.5 * s;
  X = 0.5 * a0 * (double)(2 * cx + s);
  Y = a0 * ((double)y + h);
  Z = a0 * ((double)z + h);
}

// kernels (mb_kernels64.cu)
// flag: the code bit of sites near an interstitial (0: none): a lattice pass leaves the sums
// over lattice atoms in rho / force of such a site and the interstitial pass finishes it.
// [z0, z1): the box layers a launch covers (z1 < 0: up to the last layer).  The
// interstitial passes then take the flagged sites in those layers and the
// interstitials whose wrapped z lies in them.
// outer: per-item masks of the outer stencil entries (beyond the cutoff at the ideal
// lattice) that some site of the item has inside the cutoff, one uint2 per item of the
// box (items_per_box).  The density pass writes them; a force pass given them walks only
// those entries, so it must run on the positions of the density pass that wrote them
// (null: the force pass walks every entry).
// pass_kind64: the kernels that a pass takes (MB_PASS_*).
int pass_kind64(const Geom &g, const DevPot &pot, const Plan64 *plan, double rc2, bool force, int z0 = 0, int z1 = -1);
int launch_rho64(const Geom &g, const StencilSet &st, const DevPot &pot, const Lattice64 &L, double rc2,
                 double *e_partial, int energy, int flag, cudaStream_t s, int z0 = 0, int z1 = -1,
                 uint2 *outer = nullptr, const Plan64 *plan = nullptr);
int launch_force64(const Geom &g, const StencilSet &st, const DevPot &pot, const Lattice64 &L, const StepParams &sp,
                   double *e_partial, int energy, int flag, cudaStream_t s, int z0 = 0, int z1 = -1,
                   const uint2 *outer = nullptr, const Plan64 *plan = nullptr);
// Work items (32-site row chunks) of the whole box: the length of the outer masks.
inline long long items_per_box(const Geom &g) { return (long long)((g.bcx + 31) / 32) * g.by * 2 * g.bz; }
// Outer-entry masks on (default), or off when MB_OUTER_MASKS=0 (the force passes then walk
// every outer entry: the same results, kept for checking that); read when a sim is
// created or an ensemble's walk is rebuilt.
inline bool outer_masks_on() {
  const char *v = getenv("MB_OUTER_MASKS");
  return !(v && v[0] == '0');
}
// Marks the sites of layers [z0, z1) near an interstitial; with clear set, last step's marks
// come off.  This step's list must be empty: a force pass empties the other one.
int launch_itl_mark64(const Geom &g, const Lattice64 &L, const Itl64 &I, int clear, cudaStream_t s, int z0 = 0,
                      int z1 = -1, bool chain = false);
// Takes off the marks of both lists and empties them.
int launch_itl_reset64(const Lattice64 &L, const Itl64 &I, cudaStream_t s);
int launch_itl_rho64(const Geom &g, const DevPot &pot, const Lattice64 &L, const Itl64 &I, double rc2,
                     double *e_partial, int energy, cudaStream_t s, int z0 = 0, int z1 = -1, bool chain = false);
int launch_itl_force64(const Geom &g, const DevPot &pot, const Lattice64 &L, const Itl64 &I, const StepParams &sp,
                       double *e_partial, int energy, cudaStream_t s, int z0 = 0, int z1 = -1, bool chain = false);
int launch_images64(const Geom &g, const Lattice64 &L, int what, cudaStream_t s, int z0 = 0,
                    int z1 = -1); // what: 1 pos+code, 2 df
// Lattice <-> interstitial bookkeeping after a drift (one CTA): candidates of
// sp.cand become interstitials (box order), then interstitials within sqrt(rec2) of a
// vacant site take it (list order, first claim wins).  counters: [0] conversions,
// [1] recombinations, [2] refused conversions (list full), [3] dropped candidates.
int launch_convert64(const Geom &g, const Lattice64 &L, const Itl64 &I, const StepParams &sp, double rec2,
                     int64_t *site_id, int *nd, long long *counters, cudaStream_t s);
int launch_itl_kick_drift64(const Itl64 &I, const StepParams &sp, cudaStream_t s);
int launch_reduce(const double *partials, int n, double *out, cudaStream_t s);
int energy_partials_needed();

// AoS conversion (mb_layout.cu)
// Records whose type has no potential table (type >= n_types) raise *bad_type and
// are kept out of the passes as vacant sites.
// [t0, t1): ext records (t1 < 0: to the end); [z0, z1): box layers (z1 < 0: to the last).
int launch_unpack_ext(const Geom &g, const mb_atom_element *aos, int ext_x, int ext_y, int ext_z, Lattice64 L,
                      int with_df, int *bad_type, int n_types, cudaStream_t s, long long t0 = 0, long long t1 = -1);
int launch_pack_ext(const Geom &g, mb_atom_element *aos, int ext_x, int ext_y, const Lattice64 &L, int what,
                    cudaStream_t s, int z0 = 0, int z1 = -1); // what: 1 rho+df, 2 force, 3 df only
// Records of a host step as they arrive: unpacked, kicked and drifted, ghost images written.
int launch_arrive64(const Geom &g, const mb_atom_element *aos, const Lattice64 &L, const StepParams &sp, int *bad_type,
                    int64_t *ids, int n_types, cudaStream_t s, int z0 = 0, int z1 = -1);
// Interstitial records in (setting the device count) and out.
int launch_unpack_itl(const Itl64 &I, const mb_atom_element *aos, int n, int *nd, cudaStream_t s);
int launch_pack_itl(const Itl64 &I, mb_atom_element *aos, int n, double h, int unkick, cudaStream_t s);
int launch_unpack_box_ids(const Geom &g, const mb_atom_element *aos, Lattice64 L, int with_f, int *bad_type,
                          int64_t *ids, int n_types, cudaStream_t s, int z0 = 0, int z1 = -1);
int launch_pack_box_ids(const Geom &g, mb_atom_element *aos, const Lattice64 &L, const double4 *pos, double h,
                        int unkick, const int64_t *ids, cudaStream_t s, int z0 = 0, int z1 = -1);
int launch_df_from_rho(const Geom &g, const DevPot &pot, const Lattice64 &L, cudaStream_t s);
// z-slab halo layers (mb_layout.cu): sites of one message, and the pack (box layers ->
// buf) / unpack (buf -> ghost layers, z positions + z_shift) of one field: what 1 positions,
// 2 df (both of the records p), 3 site codes.
long long halo_sites(const Geom &g);
int launch_halo(const Geom &g, int what, int pack, int side, double4 *p, int8_t *code, void *buf, double z_shift,
                cudaStream_t s);

// Half-neighbour hook passes (mb_half.cu): a decoded half-stencil offset.
struct HalfOff {
  long long off; // linear offset in the host's ext array
  int dx, dy, dz, pad_;
};
int half_stencil_build(const mb_device_domain &d, const int64_t *even, size_t n_even, const int64_t *odd, size_t n_odd,
                       std::vector<HalfOff> &out, int &cap);
int launch_half64(bool force, mb_atom_element *aos, const mb_device_domain &d, const HalfOff *st, int cap,
                  const int n[2], const DevPot &P, double rc2, int *bad, cudaStream_t s);

// ------------------------------------------------------------ utilities
int device_sm_count();
#define MB_SMEM_MAX (227 * 1024)
// Something done once for each device that the process uses (kernel attributes belong to a
// device).  Two threads may do it at once.
class DeviceOnce {
  std::atomic<unsigned long long> devices{0};

 public:
  // The current device's bit while it is still to be done, else 0.
  unsigned long long todo() const {
    int d = 0;
    if (cudaGetDevice(&d) != cudaSuccess) cudaGetLastError();
    const unsigned long long bit = 1ull << (d & 63);
    return devices.load() & bit ? 0 : bit;
  }
  void done(unsigned long long bit) { devices |= bit; }
};
// Lets two kernels use `bytes` of dynamic shared memory.
#define MB_SMEM_ATTR(k0, k1, bytes)                                                                            \
  do {                                                                                                         \
    static ::mb::DeviceOnce once_;                                                                             \
    if (const unsigned long long bit_ = once_.todo()) {                                                        \
      MB_CUDA(cudaFuncSetAttribute(k0, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(bytes)));            \
      MB_CUDA(cudaFuncSetAttribute(k1, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(bytes)));            \
      once_.done(bit_);                                                                                        \
    }                                                                                                          \
  } while (0)

} // namespace mb
