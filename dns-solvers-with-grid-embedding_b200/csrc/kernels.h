// Host-side launchers of the device kernels (internal to libdnsembed).
#pragma once

#include <cstddef>
#include <cstdint>
#include <string>

#include <cuda_runtime.h>

#include "../../include/dns_embed.h"

namespace dns {

// Running statistics of one composite-profile plane, kStatRow doubles.  Each
// sample's plane moments are exact two-pass quantities: every block keeps a
// running (count, means, sums of squared deviations) per thread (Welford) and
// merges them pairwise (Chan, Golub and LeVeque's parallel update), so a
// plane's variance is never formed as E[x^2] - E[x]^2.  The row holds:
//   0..3   sums over samples of (m - c) for the plane means m of u, v, w, rho;
//   4..8   sums over samples of (mu - cu)^2, (mv - cv)^2, (mw - cw)^2,
//          (mu - cu)(mw - cw), (mr - cr)^2 (the plane means' time variation);
//   9..13  sums over samples of the per-sample plane variances of u, v, w, the
//          covariance uw and the variance of rho;
//   14     nodes per plane; 15 samples;
//   16..19 c = (cu, cv, cw, cr): the plane means of the first sample after a
//          reset, about which the plane means are summed.
// Per-block partials of one sample: kStatPart doubles, (n, 4 means, 5 sums of
// squared deviations).
constexpr int kStatPart = 10;
constexpr int kStatRow = 20;

// Device-side scalar state carried between steps (one instance per handle).
struct DevState {
  double force;     // force[0] of the next step
  double momentum;  // encalc2 momentum of the current state
  double denst;     // encalc2 mass of the current state
  double pad;
};

// One row of the per-step log, filled on the device (time is added on the host).
struct DevLog {
  double force, momentum, denst, flowrate, stup, stdown, stress, pgrad;
};

struct Dims {
  int nx, ny, nzc;        // coarse
  int nxf, nyf, zdf, zds; // fine block; zds planes stored per block
  int gr, nzs;
};

// Tiles of the kernels that take two fine substeps in one pass (pair_f64.cu):
// ntx tiles along x and nly runs of ly rows along y, per block.
struct PairGrid {
  int ntx = 0, ly = 0, nly = 0;
  int ns = 1;  // warps side by side along x (a tile is at most 32 ns - 2 nodes wide)
  bool on() const { return ntx > 0; }
  long blocks() const { return (long)ntx * nly; }  // per fine block
};

// Launch geometry shared by the kernels and the reductions.
struct LaunchShape {
  int bx;          // threads per block along x
  int jb;          // rows (y) per block
  int cgx, cgy;    // coarse grid x/y blocks (z = nzc planes)
  int fgx, fgy;    // fine grid x/y blocks (z = 2 zds planes)
  int igx, igy;    // interface tile grid
  int jgx, jgy;    // injection / extraction grid (x, y) per wall
  int vgx;         // blocks of the filtered injection along x
  PairGrid pair;   // tiles of the passes that take two fine substeps (of the precision asked for)
  long n_coarse_blocks() const { return (long)cgx * cgy; }  // per plane
  long n_fine_blocks() const { return (long)fgx * fgy; }    // per plane
};

LaunchShape make_shape(const Dims &d, bool f32 = false);

constexpr int kPairMaxZds = 16;  // planes that fit the shared-memory ring
PairGrid make_pair_grid(const Dims &d);      // off where zds > kPairMaxZds
PairGrid make_pair_grid_f32(const Dims &d);  // the FP32 form's tiles
void pair_runs(const Dims &d, int per_sm, PairGrid &g);  // runs along y, per_sm blocks on an SM
// whether they are faster than one substep at a time
bool pairs_pay_f64(const Dims &d, const PairGrid &g);
bool pairs_pay_f32(const Dims &d, const PairGrid &g);
// raise the kernels' shared-memory limit on the current device (0, or -1)
int prepare_pair_f64();
// two substeps from src into dst; mid: the interface planes between them,
// [2 walls][19][nyf][nxf]; part: per-block flow-rate pairs [2 g.blocks()] (last);
// wpart: per-block wall-shear pairs [6][g.blocks()] (first); lost: set, and never
// cleared, where a wait of the kernel ran out (dst is not valid)
int prepare_pair_f32();
void launch_fine_pair_f32(const float *src, float *dst, const float *mid, const int8_t *wflag, const Dims &d,
                          const PairGrid &g, double om, const DevState *st, double *part, double *wpart,
                          unsigned int *lost, bool first, bool last, cudaStream_t stream);
void launch_fine_pair_f64(const double *src, double *dst, const double *mid, const int8_t *wflag, const Dims &d,
                          const PairGrid &g, double om, const DevState *st, double *part, double *wpart,
                          unsigned int *lost, bool first, bool last, cudaStream_t stream);


// record a message for dns_last_error() on the calling thread (dns_api.cu)
void set_last_error(const std::string &msg);

// Reduction scratch sizes (doubles) for a given shape.
struct PartialLayout {
  long coarse, fine, inject, wall, stats_c, stats_f, flow, level2;  // offsets into one buffer
  long total;
};
PartialLayout partial_layout(const Dims &d, const LaunchShape &s);

struct StepParams {
  double omega_c, omega_f;
  double ub;        // bulk velocity (constant flow rate target)
  double gconst;    // constant body force
  int cfr;          // 1: force = ub - momentum
  int fltr;         // the injection is the filtered one
  double den_offset;  // encalc2 weight sum added to the mass partials (FP32 form: they sum deviations)
};

// --- FP64 kernels (kernels_f64.cu) ---
// stats: also the per-block moments of the sampled statistics (kStatPart doubles per block)
void launch_coarse_f64(const double *src, double *dst, const Dims &d, const LaunchShape &s, double om,
                       const DevState *st, double *partials, const PartialLayout &pl, bool stats,
                       cudaStream_t stream);
void launch_extract_f64(const double *fc, double *hist_n, const Dims &d, const LaunchShape &s,
                        cudaStream_t stream);
void launch_fine_f64(const double *src, double *dst, const int8_t *wflag, const Dims &d, const LaunchShape &s,
                     double om, const DevState *st, double *partials, const PartialLayout &pl, bool first,
                     bool last, bool stats, cudaStream_t stream);
// plane statistics of the stored fine state, into the partials of a sampled step (one
// whose first pass takes two substeps; else fine's stats does it), kStatRows rows a block
constexpr int kStatRows = 8;
void launch_fine_stats_f64(const double *src, const Dims &d, const LaunchShape &s, double *partials,
                           const PartialLayout &pl, cudaStream_t stream);
void launch_fine_stats_f32(const float *src, const Dims &d, const LaunchShape &s, double *partials,
                           const PartialLayout &pl, cudaStream_t stream);
// The interface transfers of n substeps (at most 4), two launches: macroscopic
// fields into each one's mac[2 walls][4][nyf][nxf], then one block per (tile,
// substep, wall, population) into the substep's planes
struct IfaceTarget {
  int substep;
  double *mac;    // FP64 form
  void *out[2];   // plane of population 0 of the lower / upper wall
  size_t stride;  // elements from one population's plane to the next
};
void launch_interface_f64(const double *hn, const double *hp, const double *hpp, const IfaceTarget *tg, int n,
                          const Dims &d, const LaunchShape &s, double omega_c, double omega_f,
                          cudaStream_t stream);
// filtered: the FLTR transfer (ftcdtransfer_lesfltr.c) instead of ftcdtransfer.c
// (its kernels' shared-memory limit is raised first, on the current device)
int prepare_filter_f64();
int prepare_filter_f32();
void launch_inject_f64(const double *fsrc, double *cdst, const Dims &d, const LaunchShape &s, double omega_c,
                       double omega_f, double *partials, const PartialLayout &pl, bool filtered,
                       cudaStream_t stream);
// counter: one device unsigned int, zero between launches (the kernel resets it);
// pair_first / pair_last: the step's first / last fine pass took two substeps
// (it left the wall-shear / flow-rate partials by its own tiles)
// log: the rows of a group of steps; counter[1] is the next row, counter[0] the
// kernel's block count (0 between launches); a row's wall stress is NaN where
// counter[2] is set (a two-substep pass gave up)
void launch_finalize(DevState *st, DevLog *log, double *partials, unsigned int *counter,
                     const PartialLayout &pl, const Dims &d, const LaunchShape &s, const StepParams &sp,
                     bool pair_first, bool pair_last, cudaStream_t stream);
// own_pass: the fine partials are launch_fine_stats's
void launch_stats_finalize(double *acc, const double *partials, const PartialLayout &pl, const Dims &d,
                           const LaunchShape &s, bool own_pass, cudaStream_t stream);
// direct encalc2 reduction of the stored state into st (momentum, denst, force)
void launch_flow_sums_f64(const double *fc, const double *ff, DevState *st, double *partials,
                          const PartialLayout &pl, const Dims &d, const LaunchShape &s, const StepParams &sp,
                          cudaStream_t stream);
// the same reduction over a caller-held state, with caller-provided block scratch
// (scratch_pairs = flow_sums_pairs(d, s) pairs of doubles), result into *out
long flow_sums_pairs(const Dims &d, const LaunchShape &s);
void launch_flow_sums_scratch(const double *fc, const double *ff, DevState *out, double *scratch, const Dims &d,
                              const LaunchShape &s, const StepParams &sp, cudaStream_t stream);
// finalize a direct (flow_sums) reduction of npairs block partials into *st
void finalize_flow_sums(DevState *st, const double *pairs, long npairs, const Dims &d, const LaunchShape &s,
                        const StepParams &sp, cudaStream_t stream);
// encalc2 weight of every node summed (the mass of a state with rho = 1)
double encalc2_weight_sum(const Dims &d);
void launch_seed_f64(double *fc, double *ff, double *hist3, const Dims &d, uint64_t seed, double uc, double amp,
                     cudaStream_t stream);
// vel_print field records of np device planes p0.. into vel[i][j][k][3] and
// den[i][j][k] (nz_aos planes, device plane p0 + q at k = k0_aos + q)
void launch_fields_f64(const double *soa, double *vel, double *den, int nx, int ny, int P, int p0, int np, int nz_aos,
                       int k0_aos, cudaStream_t stream);
void launch_fields_f32(const float *soa, double *vel, double *den, int nx, int ny, int P, int p0, int np, int nz_aos,
                       int k0_aos, cudaStream_t stream);
// the same moments as planar fields q[c][k][j][i] (c = u, v, w, den / 3) of a
// level with nz planes, device plane p0 + s at k = k0 + s
void launch_fields_planar_f64(const double *soa, double *q, int nx, int ny, int P, int p0, int np, int nz,
                              int k0, cudaStream_t stream);
void launch_fields_planar_f32(const float *soa, double *q, int nx, int ny, int P, int p0, int np, int nz, int k0,
                              cudaStream_t stream);
// Mode -i start: one level of the embedded grid interpolated from a uniform-grid
// state.  uni is the uniform state in reference AoS order [xu][yu][zd][19]; out
// receives the level in reference AoS order [nxl][nyl][nzl][19] (wall plane of a
// fine block = the rest equilibrium w_a).  *bad is set when a stencil index
// leaves the reference's two-deep halo in x or y, or the grid in z (those
// nodes are not read).  level: 0 coarse, 1 lower fine, 2 upper fine.
struct UniformMap {
  int level, nxl, nyl, nzl;  // output level extents (nzl = zdc or zdf)
  int xu, yu, zd;            // uniform grid: xdu, ydu, zdu + 2
  int gr, zdf, zdc;
  double dxf, dxc, dxr;      // node spacings as the reference's initializer forms them
  double fac;                // (dxr / dx_level) (omega / omega_level), the f^neq rescaling
};
void launch_uniform_interp_f64(const double *uni, const UniformMap &m, double *out, int *bad, cudaStream_t stream);
// Turbulence statistics / kinetic-energy budget of one snapshot (tke.cu) from
// the device field arrays of the three levels in the reference file layout
// (0 coarse vel[i][j][k][3] / den[i][j][k], 1 lower fine, 2 upper fine);
// prof on the host, [DNS_TKE_NPROF][nz_profile]; ufl / vfl optional.
int tke_validate(const dns_params &p);
int tke_budget_device(const dns_params &p, const dns_geometry &g, const double *const vel[3],
                      const double *const den[3], double *prof, double *ufl, double *vfl, cudaStream_t st);
// the same from planar fields q[l] = [4][nz][ny][nx] (u, v, w, den / 3) per level
// work: device space of tke_workspace_bytes(g) (8-byte aligned), or null to
// allocate per call
size_t tke_workspace_bytes(const dns_geometry &g);
int tke_budget_planar(const dns_params &p, const dns_geometry &g, const double *const q[3], double *prof,
                      double *ufl, double *vfl, cudaStream_t st, void *work = nullptr);
// Plane statistics of the state (fc, ff) in the reference's summation order, one
// row of 9 per plane: means of u, v, w, density, mean squares uu, vv, ww, uw, rr
// about them.  fine: the 2 zds stored planes; coarse: planes 2..zdc-3.  qc, qf:
// device scratch, (4 x nodes + 9) doubles a plane of each level.
int plane_record_device(const void *fc, const void *ff, bool f32, double *qc, double *qf, const dns_geometry &g,
                        double *fine, double *coarse, cudaStream_t st);
// wall plane kw of a level in reference AoS order [nodes = nx ny][nz][19] to
// (to_aos) or from the compact wall array [nodes][19]
void launch_wall_plane(double *aos, double *wall, long long nodes, int nz, int kw, bool to_aos, cudaStream_t stream);
// layout transposes between the device SoA state and the reference AoS order
// [i0, i1): the x indices to move (i1 < 0: all); the AoS side is i-major, so
// an x range is one contiguous run of it
void launch_soa_to_aos(const double *soa, double *aos, int nx, int ny, int P, int p0, int np, int nz_aos,
                       int k0_aos, cudaStream_t stream, int i0 = 0, int i1 = -1);
void launch_history(const double *in, void *hist, bool f32, int nx, int ny, cudaStream_t stream);
void launch_aos_to_soa(const double *aos, double *soa, int nx, int ny, int P, int p0, int np, int nz_aos,
                       int k0_aos, cudaStream_t stream, int i0 = 0, int i1 = -1);

// --- FP32 deviation-storage kernels (kernels_f32.cu); same layouts in float ---
void launch_coarse_f32(const float *src, float *dst, const Dims &d, const LaunchShape &s, double om,
                       const DevState *st, double *partials, const PartialLayout &pl, bool stats,
                       cudaStream_t stream);
void launch_extract_f32(const float *fc, float *hist_n, const Dims &d, const LaunchShape &s, cudaStream_t stream);
void launch_fine_f32(const float *src, float *dst, const int8_t *wflag, const Dims &d, const LaunchShape &s,
                     double om, const DevState *st, double *partials, const PartialLayout &pl, bool first, bool last,
                     bool stats, cudaStream_t stream);
// corner: scratch of 2 x 23 x ny x nx float4 (corner values and derivatives)
void launch_interface_f32(const float *hn, const float *hp, const float *hpp, float *corner, const IfaceTarget &tg,
                          const Dims &d, double omega_c, double omega_f, cudaStream_t stream);
void launch_inject_f32(const float *fsrc, float *cdst, const Dims &d, const LaunchShape &s, double omega_c,
                       double omega_f, double *partials, const PartialLayout &pl, bool filtered,
                       cudaStream_t stream);
void launch_flow_sums_f32(const float *fc, const float *ff, DevState *st, double *partials, const PartialLayout &pl,
                          const Dims &d, const LaunchShape &s, const StepParams &sp, cudaStream_t stream);
void launch_seed_f32(float *fc, float *ff, float *hist3, const Dims &d, uint64_t seed, double uc, double amp,
                     cudaStream_t stream);
// device float deviations <-> reference AoS doubles (f = w + d)
void launch_dev_to_aos_f32(const float *soa, double *aos, int nx, int ny, int P, int p0, int np, int nz_aos,
                           int k0_aos, cudaStream_t stream, int i0 = 0, int i1 = -1);
void launch_aos_to_dev_f32(const double *aos, float *soa, int nx, int ny, int P, int p0, int np, int nz_aos,
                           int k0_aos, cudaStream_t stream, int i0 = 0, int i1 = -1);

}  // namespace dns
