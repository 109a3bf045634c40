// FP64 plain form: two fine substeps in one pass over the fine state.
//
// The stream-collide of one substep reads and writes every population once
// (304 bytes a node), so a coarse step with its GR substeps moves the fine
// state GR times through HBM.  This kernel advances both near-wall blocks by
// two substeps with one read and one write: a thread block owns a column of a
// fine block (a tile along x, all zds planes, a run of rows along y) and marches
// along y, keeping the state between the two substeps in shared memory.
//
//   row t:  collide its nodes (substep 1), push into the shared rows t - 1, t, t + 1;
//   then    row t - 1 is complete: collide it (substep 2), push to HBM.
//
// A warp signals that it has pushed its row, and waits for the planes beside it to
// have pushed theirs, before it takes the complete row; it signals that it has
// taken it, and waits for its neighbours' signal two collisions later, before its
// next push.  Planes are held together only through their neighbours: with
// barriers of the whole block the warps moved in step, all collisions and all
// stores together, and a row took 11.0 instead of 8.4 thousand cycles.
//
// A warp holds 32 columns of one plane, a lane one column.  The first and last
// column of a tile are computed in substep 1 only (their pushes complete the
// tile's own columns), and so are the rows above and below the run: the
// redundant work is 2 columns of a tile and 2 rows of a run.  Sixteen warps fill
// the register file at 128 registers a thread.
//
// Shared memory holds for every population as many rows as are live: pushes
// with e_y = -1 complete the row that is taken next (1 row; 2 for populations
// 17 and 18, which half-way bounce-back also writes one row early), e_y = 0 two
// rows, e_y = +1 three (population 0 stays in its lane's registers): 38 rows of
// 32 nodes a plane, and 19 for the next row of src, which bulk copies bring in
// during both substeps of the present one: 224 KB for zds = 16.  The loop loads
// nothing from global memory into registers: with three populations and the wall
// flags loaded that way, the waits for them, at whatever the load shared its
// scoreboard with, took a quarter of the time.  Pushes that leave the tile land in
// a neighbouring row's first or last column, which is never read, so pushes need
// no test along x.
//
// The interface plane of the state between the substeps comes from the
// coarse-to-fine transfer (mid), its rows by bulk copies too.  Pushes into the
// interface plane are dropped in both substeps, as in the one-substep kernel.
//
// 256x128x83 (two blocks of 512 x 256 x 16): 308 us for both substeps, 4.1 TB/s of
// state; as two launches of the one-substep kernel 435 us, 5.9 TB/s.  Bound by
// FP64 issue and latency: a row of 16 planes takes 8 thousand cycles, of which the
// FP64 pipe needs 4.2; HBM at the copy rate would take 195 us.
//
// The arithmetic per node is collide_f64's and the wall rule, in the
// one-substep kernel's order: with a constant force the state is the same bit
// for bit.  Built with -fmad=false.
#include "kernels.h"
#include "lattice.cuh"
#include "pair_sync.cuh"

namespace dns {

namespace {

constexpr int kPairThreads = 32 * kPairMaxZds;

constexpr int kPad = 2;  // before and after the ring: pushes off its first and last row

// ring of zds - 1 planes, 19 rows of the interface plane, the next row of src
size_t pair_smem(int zds, int ns) {
  return ((size_t)ns * 32 * ((zds - 1) * kRing + 19 + zds * 19) + 2 * kPad) * sizeof(double);
}

// Keep the compiler from moving a node's collision into the branches that store
// it: the 19 updates are independent and overlap only while they are together.
__device__ __forceinline__ void pin(double (&f)[19]) {
#pragma unroll
  for (int a = 0; a < 19; a++) asm volatile("" : "+d"(f[a]));
}

// where tile i of n along a row of nx nodes starts: even, sizes at most two apart
__host__ __device__ __forceinline__ int pair_x0(int i, int nx, int n) {
  return 2 * (int)((long long)i * (nx / 2) / n);
}

// MODE bits: 1 flow-rate partials of dst (the step's last pass), 2 wall-shear
// sums of src (the step's first pass).  NS warps side by side take the 32 NS
// columns of a plane.
template <int MODE, int NS>
__global__ void __launch_bounds__(kPairThreads, 1)
    fine_pair_kernel(const double *__restrict__ src, double *__restrict__ dst, const double *__restrict__ mid,
                     const int8_t *__restrict__ wf, Dims d, PairGrid g, double om, const DevState *st,
                     double *__restrict__ part, double *__restrict__ wpart, unsigned int *__restrict__ lost) {
  extern __shared__ __align__(16) double M[];  // bulk copies land in it
  constexpr int kTX = 32 * NS, kPlane = kRing * kTX;
  const int zds = d.zds, zdf = d.zdf, gr = d.gr, nx = d.nxf, ny = d.nyf;
  const int lane = threadIdx.x & 31, warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);  // warp-uniform
  const bool upper = blockIdx.z != 0;
  // column c is node x0 + c (wrapped); tiles start at even nodes
  const int x0 = pair_x0(blockIdx.x, nx, g.ntx), cnt = pair_x0(blockIdx.x + 1, nx, g.ntx) - x0;
  const int y0 = blockIdx.y * g.ly, L = min(g.ly, ny - y0);
  const int qi = upper ? 0 : zds - 1, qw = upper ? zds - 1 : 0;  // interface and wall-adjacent planes
  const int q = warp / NS, col = (warp % NS) * 32 + lane;        // columns 1..cnt are the tile's own
  const bool own = col >= 1 && col <= cnt;
  int x = x0 + min(col, cnt + 1);
  x = x >= nx ? x - nx : x;
  const int xm = x == 0 ? nx - 1 : x - 1, xp = x == nx - 1 ? 0 : x + 1;
  const int p = (upper ? zds : 0) + q, k = upper ? q : q + 1;  // device plane, reference k
  const size_t plane = (size_t)ny * nx, pstride = (size_t)2 * zds * plane;
  const double Gf = (1. / ((double)gr)) * st->force;
  const bool wall = q == qw, iface = q == qi;
  // pushes by e_z that stay in the block and off the interface plane
  const bool z0 = !iface, zup = q + 1 < zds && q + 1 != qi, zdn = q > 0 && q - 1 != qi;
  const bool inner = z0 && zup && zdn;
  // planes in the order away from the wall, the interface plane last
  const int pos = upper ? zds - 1 - q : q;
  double *const Mq = M + kPad + (size_t)pos * kPlane + col;
  // the column this lane collides in substep 2: an own one for every lane (zeros or
  // stale values would send a warp's division down its slow path)
  const double *const Mr = Mq - col + min(max(col, 1), cnt);
  double *const Mup = Mq + (upper ? -kPlane : kPlane), *const Mdn = Mq - (upper ? -kPlane : kPlane);
  double *const Sw = M + 2 * kPad + (size_t)(zds - 1) * kPlane + 19 * kTX + (size_t)warp * 19 * 32, *const Sq = Sw + lane;
  // the warp's columns in memory: n1 nodes from node xs (an even count and start:
  // 16-byte aligned), and the columns of the row's end that continue at its
  // start, which their lanes copy one by one (a second bulk copy a row made the
  // last tile's blocks 25% slower than the others)
  const int cs = (warp % NS) * 32, ncol = max(0, min(32, cnt + 2 - cs));
  const int xs = x0 + cs >= nx ? x0 + cs - nx : x0 + cs, n1 = min(ncol, nx - xs);
  const bool wraps = lane >= n1 && lane < ncol;
  double acc[2] = {0., 0.}, wacc[2] = {0., 0.};
  const bool wall_sum_plane =
      upper ? (k == zdf - 2 || k == zdf - 3 || k == zdf - 4) : (k == 1 || k == 2 || k == 3);
  const bool wall_rho_plane = upper ? (k == zdf - 4) : (k == 1);
  // encalc2 weights of the destination planes k - 1, k, k + 1 (what heads into the
  // wall stays on plane k; dropped pushes head for planes of weight 0)
  double wz[3];
#pragma unroll
  for (int c = 0; c < 3; c++) {
    const int kd = (wall && c == (upper ? 2 : 0)) ? k : k + c - 1;
    wz[c] = !upper ? ((kd >= 1 && kd < zdf - gr) ? 1.0 : 0.0)
                   : ((kd >= gr && kd < zdf - 1) ? (kd == gr ? 0.5 : 1.0) : 0.0);
  }
  // where they are all 1 the partials are the nodes' post-collision moments
  const bool unit = wz[0] == 1. && wz[1] == 1. && wz[2] == 1., none = wz[0] == 0. && wz[1] == 0. && wz[2] == 0.;
  const unsigned rowb = (unsigned)nx * 8u, planeb = (unsigned)plane * 8u;
  const unsigned nodeb = (unsigned)p * planeb + (unsigned)x * 8u;  // byte offset of (plane, x) in a population
  __shared__ unsigned long long pushed[kPairMaxZds], taken[kPairMaxZds], staged[kPairMaxZds], middle[kPairMaxZds];
  __shared__ unsigned long long solid[kMaxRun + 4];
  __shared__ int stop;
  if (threadIdx.x == 0) {
    stop = 0;
    for (int w = 0; w < zds; w++) {
      const int n = (1 + (w > 0) + (w < zds - 1)) * NS;
      mb_init(&pushed[w], n);
      mb_init(&taken[w], n);
    }
  }
  if (lane == 0) {  // one arrival for the bulk copies, one for each lane that copies by itself
    mb_init(&staged[warp], 1 + ncol - n1);
    mb_init(&middle[warp], 1 + ncol - n1);
  }
  // columns past the tile collide ones; what they push is never read
#pragma unroll
  for (int a = 0; a < 19; a++) Sq[a * 32] = 1.;
  // wall flags of rows t = -1 .. L + 2, one mask of the tile's columns a row
  for (int r = warp; r < L + 4; r += zds * NS) {
    int yr = y0 - 2 + r;
    yr = yr < 0 ? yr + ny : (yr >= ny ? yr - ny : yr);
    unsigned long long m = 0;
#pragma unroll
    for (int s = 0; s < NS; s++) {
      int xr = x0 + min(s * 32 + lane, cnt + 1);
      xr = xr >= nx ? xr - nx : xr;
      m |= (unsigned long long)__ballot_sync(0xffffffffu, wf[(size_t)yr * nx + xr] == -1) << (s * 32);
    }
    if (lane == 0) solid[r] = m;
  }
  fence_async_proxy();
  __syncthreads();
  bool ok = true, gone = false;  // a wait of the block ran out
  double f[19], k0 = 0., p0 = 0.;  // population 0 of rows t and t - 1
  // the warp's columns of a row of 19 populations (stride apart) into rows
  // `pitch` apart: lane a copies population a.  (Every lane has collided the rows'
  // old values; the fence puts the reads before the copies, which go by another
  // way to shared memory.  Without it, and issued right behind the reads, copies
  // overtook them.)
  auto copy = [&](double *row, int pitch, const double *from, size_t stride, unsigned long long *b) {
    fence_async_proxy();
    __syncwarp();
    if (lane == 0) mb_expect(b, (unsigned)(19 * n1) * 8u);
    __syncwarp();
    if (lane < 19 && n1 > 0) bulk_copy(row + lane * pitch, from + (size_t)lane * stride + xs, (unsigned)n1 * 8u, b);
    if (wraps) {
#pragma unroll
      for (int a = 0; a < 19; a++) lane_copy(row + a * pitch + lane, from + (size_t)a * stride + (lane - n1));
      lane_copies_arrive(b);
    }
  };
  auto stage = [&](int y) { copy(Sw, 32, src + ((size_t)p * ny + y) * nx, pstride, &staged[warp]); };
  auto next = [&](int y) { return y == ny - 1 ? 0 : y + 1; };
  int y = y0 == 0 ? ny - 1 : y0 - 1;  // row t = 0
  int yd = y;                         // the row that substep 2 takes (t - 1)
  int t = 0, s3 = 0;                  // s3: t mod 3
  // substep 1 of row t1 (the y index of the row after it: ahead), up to the collision
  auto first_half = [&](int t1, int ahead) {
    if (t1 <= L + 1) ok = mb_wait(&staged[warp], t1 & 1, &stop) && ok;
#pragma unroll
    for (int a = 0; a < 19; a++) f[a] = Sq[a * 32];
    double dens, u0, u1, u2;
    collide_pairs_f64(f, om, Gf, dens, u0, u1, u2);
    pin(f);
    gone = !__all_sync(0xffffffffu, ok);
    if (t1 <= L && !gone) stage(ahead);
    if ((MODE & 2) && own && t1 >= 1 && t1 <= L) {
      if (wall_sum_plane) wacc[0] += u0;
      if (wall_rho_plane) wacc[1] += dens;
    }
  };
  stage(y);
  first_half(0, next(y));
  for (; !gone && t <= L + 1; t++) {
    const int yn = next(y);
    // rows t - 1, t, t + 1 in the two- and three-row rings
    const int r2c = (t & 1) * kTX, r2p = kTX - r2c;
    const int r3c = s3 * kTX, r3n = (s3 == 2 ? 0 : s3 + 1) * kTX, r3p = (s3 == 0 ? 2 : s3 - 1) * kTX;
    if (t > 0) ok = mb_wait(&taken[q], (t - 1) & 1, &stop) && ok;
    {
      // where a push of population a from row t lands: row t + e_y, or t itself for a bounce
      auto slot = [&](int a, int row) {
        const int r = ring_depth(a) == 1 ? 0
                      : ring_depth(a) == 2 ? (row == 0 ? r2c : r2p)
                                           : (row == 0 ? r3c : (row > 0 ? r3n : r3p));
        return ring_off(a) * kTX + r;
      };
      p0 = k0;
      k0 = f[0];
      auto to = [&](int a) { return ez_of(a) == 0 ? Mq : (ez_of(a) > 0 ? Mup : Mdn); };
      if (inner) {
#pragma unroll
        for (int a = 1; a < 19; a++) to(a)[slot(a, ey_of(a)) + ex_of(a)] = f[a];
      } else {
#pragma unroll
        for (int c = -1; c <= 1; c++)
          if (c == 0 ? z0 : (c > 0 ? zup : zdn))
#pragma unroll
            for (int a = 1; a < 19; a++)
              if (ez_of(a) == c) to(a)[slot(a, ey_of(a)) + ex_of(a)] = f[a];
        if (wall) {
          const int sb = solid_bits(solid, t, col);
#pragma unroll
          for (int a = 1; a < 19; a++) {
            if (ez_of(a) == 0 || (ez_of(a) > 0) != upper) continue;
            Mq[(sb & 1) && (sb & dest_bit(a)) ? slot(opp_of(a), 0) : slot(mir_of(a), ey_of(a)) + ex_of(a)] = f[a];
          }
        }
      }
    }
    mb_arrive(pushed, lane, q, zds);
    ok = mb_wait(&pushed[q], t & 1, &stop) && ok;
    double h[19];
    // the interface row: row t - 1, the copies' (t - 2)nd phase
    if (iface && t >= 2) ok = mb_wait(&middle[warp], t & 1, &stop) && ok;
#pragma unroll
    for (int a = 1; a < 19; a++)
      h[a] = Mr[iface ? a * kTX : ring_off(a) * kTX + (ring_depth(a) == 1 ? 0 : (ring_depth(a) == 2 ? r2p : r3p))];
    h[0] = iface ? Mr[0] : p0;
    mb_arrive(taken, lane, q, zds);
    double dens, u0, u1, u2;
    collide_pairs_f64(h, om, Gf, dens, u0, u1, u2);
    pin(h);
    // the interface row that substep 2 takes next (row t)
    if (iface && t >= 1 && t <= L && __all_sync(0xffffffffu, ok))
      copy(Mq - lane, kTX, mid + ((size_t)(upper ? 19 : 0) * ny + y) * nx, plane, &middle[warp]);
    if (t >= 2 && own) {
      if ((MODE & 1) && unit) {
        acc[0] += dens * u0 + dens * Gf;
        acc[1] += dens;
      }
      const int ym = yd == 0 ? ny - 1 : yd - 1;  // rows yd - 1, yd, y
      const unsigned o = nodeb + (unsigned)yd * rowb;
      const unsigned dxm = (unsigned)(xm - x) * 8u, dxp = (unsigned)(xp - x) * 8u;
      const unsigned dym = (unsigned)(ym - yd) * rowb, dyp = (unsigned)(y - yd) * rowb;
      auto off = [&](int a) {
        return (ey_of(a) > 0 ? dyp : (ey_of(a) < 0 ? dym : 0u)) + (ex_of(a) > 0 ? dxp : (ex_of(a) < 0 ? dxm : 0u));
      };
      auto offz = [&](int a) { return ez_of(a) > 0 ? planeb : (ez_of(a) < 0 ? 0u - planeb : 0u); };
      if (inner) {
#pragma unroll
        for (int a = 0; a < 19; a++) *at(dst + (size_t)a * pstride, o + off(a) + offz(a)) = h[a];
      } else {
#pragma unroll
        for (int c = -1; c <= 1; c++)
          if (c == 0 ? z0 : (c > 0 ? zup : zdn))
#pragma unroll
            for (int a = 0; a < 19; a++)
              if (ez_of(a) == c) *at(dst + (size_t)a * pstride, o + off(a) + offz(a)) = h[a];
        if (wall) {
          const int sb = solid_bits(solid, t - 1, col);
#pragma unroll
          for (int a = 0; a < 19; a++) {
            if (ez_of(a) == 0 || (ez_of(a) > 0) != upper) continue;
            const bool bounce = (sb & 1) && (sb & dest_bit(a));
            const unsigned to = bounce ? o : o + off(a);
            *at(bounce ? dst + (size_t)opp_of(a) * pstride : dst + (size_t)mir_of(a) * pstride, to) = h[a];
            // a bounce reverses its momentum
            if ((MODE & 1) && ex_of(a) != 0 && bounce) acc[0] -= 2. * ex_of(a) * wz[1] * h[a];
          }
        }
      }
      if ((MODE & 1) && !unit && !none) {
        // mass and momentum by destination plane
        const double m0 = ((h[0] + h[1]) + (h[2] + h[3])) + ((h[4] + h[7]) + (h[8] + h[9])) + h[10];
        const double mp = ((h[5] + h[11]) + (h[14] + h[15])) + h[18];
        const double mm = ((h[6] + h[12]) + (h[13] + h[16])) + h[17];
        const double p0 = ((h[1] - h[2]) + (h[7] - h[8])) + (h[10] - h[9]);
        acc[1] += wz[0] * mm + wz[1] * m0 + wz[2] * mp;
        acc[0] += wz[0] * (h[12] - h[13]) + wz[1] * p0 + wz[2] * (h[11] - h[14]);
      }
    }
    first_half(t + 1, next(yn));
    yd = y;
    y = yn;
    s3 = s3 == 2 ? 0 : s3 + 1;
  }
  if (gone) {
    stop = 1;
    *lost = 1u;
    drain(&staged[warp], min(t, L + 1));
    if (iface) drain(&middle[warp], min(t - 1, L) - 1);
  }
  __syncthreads();
  // partials in a fixed order: lanes by shuffles, then the warps in order
  const int nblk = gridDim.x * gridDim.y, blk = blockIdx.y * gridDim.x + blockIdx.x;
  if (MODE) {
    double v[4] = {acc[0], acc[1], wacc[0], wacc[1]};
#pragma unroll
    for (int c = 0; c < 4; c++) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v[c] += __shfl_down_sync(0xffffffffu, v[c], o);
      if (lane == 0) M[warp * 4 + c] = v[c];
    }
    __syncthreads();
    if ((MODE & 1) && threadIdx.x < 2) {
      double s = 0.;
      for (int w = 0; w < zds * NS; w++) s += M[w * 4 + threadIdx.x];
      part[((size_t)blockIdx.z * nblk + blk) * 2 + threadIdx.x] = s;
    }
    // wall-shear rows: lower k = 1, 2, 3, upper k = zdf - 2, -3, -4
    if ((MODE & 2) && threadIdx.x >= 32 && threadIdx.x < 38) {
      const int r = (threadIdx.x - 32) >> 1, c = threadIdx.x & 1;
      const int w0 = (upper ? zds - 1 - r : r) * NS;
      double s = 0.;
      for (int w = w0; w < w0 + NS; w++) s += M[w * 4 + 2 + c];
      wpart[((size_t)(upper ? 3 + r : r) * nblk + blk) * 2 + c] = s;
    }
  }
}

}  // namespace

// The number of runs along y that gives the shortest schedule: rows of a run, the
// two redundant rows and about two rows' worth of start and end, times the waves.
void pair_runs(const Dims &d, int per_sm, PairGrid &g) {
  constexpr int kSm = 148;
  long best = -1;
  for (int n = 1; n <= d.nyf && n <= 1024; n++) {
    const int ly = (d.nyf + n - 1) / n, nly = (d.nyf + ly - 1) / ly;
    if (ly > kMaxRun) continue;
    const long waves = (2L * g.ntx * nly + kSm * per_sm - 1) / (kSm * per_sm), cost = waves * (ly + 4);
    if (best < 0 || cost < best) {
      best = cost;
      g.ly = ly;
      g.nly = nly;
    }
  }
  if (best < 0) g.ntx = 0;  // more rows than runs can hold
}

// Tiles of a fine block: two warps side by side where two segments of planes
// fit the ring and the row is longer than one.
PairGrid make_pair_grid(const Dims &d) {
  PairGrid g;
  // 32-bit byte offsets in a population; rows of 16-byte multiples
  if (d.zds > kPairMaxZds || 2LL * d.zds * d.nyf * d.nxf >= (1LL << 29) || d.nxf % 2) return g;
  g.ns = (2 * d.zds <= kPairMaxZds && d.nxf > 30) ? 2 : 1;
  const int w = 32 * g.ns - 2;
  g.ntx = (d.nxf + w - 1) / w;
  pair_runs(d, 1, g);
  return g;
}

// Two substeps at a time pay where the substeps are bound by HBM: a fine state of
// 100 MB and more (two of them are past the 126 MB L2) with 16 warps a block,
// more with fewer warps, which hide less latency.  Measured us per step, pairs
// against single substeps: GR 2, zds 16: 80 MB 122 / 116, 120 MB 144 / 165,
// 159 MB 169 / 186, 638 MB 564 / 683; zds 12: 60 MB 113 / 102, 478 MB 522 / 571;
// zds 8: 80 MB 142 / 138, 319 MB 425 / 459; GR 3, zds 9: 222 MB 426 / 409; GR 4,
// zds 10: 149 MB 342 / 347, 398 MB 797 / 840.  (The line does not see the ratio: at
// GR 4, where pairs also save transfers, the first of these lies 1.4% on its wrong side.)
bool pairs_pay_f64(const Dims &d, const PairGrid &g) {
  const double w = 16. / (d.zds * g.ns), mb = 2. * d.zds * d.nyf * d.nxf * 19 * 8 * 1e-6;
  return g.on() && mb >= 100. * w * w;
}

int prepare_pair_f64() {
  const int bytes = (int)pair_smem(kPairMaxZds, 1);
  const void *fn[8] = {(const void *)fine_pair_kernel<0, 1>, (const void *)fine_pair_kernel<1, 1>,
                       (const void *)fine_pair_kernel<2, 1>, (const void *)fine_pair_kernel<3, 1>,
                       (const void *)fine_pair_kernel<0, 2>, (const void *)fine_pair_kernel<1, 2>,
                       (const void *)fine_pair_kernel<2, 2>, (const void *)fine_pair_kernel<3, 2>};
  for (const void *f : fn)
    if (cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess) return -1;
  return 0;
}

void launch_fine_pair_f64(const double *src, double *dst, const double *mid, const int8_t *wflag, const Dims &d,
                          const PairGrid &g, double om, const DevState *st, double *part, double *wpart,
                          unsigned int *lost, bool first, bool last, cudaStream_t stream) {
  const dim3 grid(g.ntx, g.nly, 2), block(32 * d.zds * g.ns);
  const size_t smem = pair_smem(d.zds, g.ns);
#define PAIR_CASE(M, N) \
  case M * 2 + N - 1:   \
    fine_pair_kernel<M, N><<<grid, block, smem, stream>>>(src, dst, mid, wflag, d, g, om, st, part, wpart, lost); break;
  switch (((last ? 1 : 0) | (first ? 2 : 0)) * 2 + g.ns - 1) {
    PAIR_CASE(0, 1) PAIR_CASE(1, 1) PAIR_CASE(2, 1) PAIR_CASE(3, 1)
    PAIR_CASE(0, 2) PAIR_CASE(1, 2) PAIR_CASE(2, 2) PAIR_CASE(3, 2)
  }
#undef PAIR_CASE
}

}  // namespace dns
