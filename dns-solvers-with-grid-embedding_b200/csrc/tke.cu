// Turbulence statistics and kinetic-energy budget of one snapshot, on the
// device: the reference's offline program TKE-budget/computations
// (budget-no-slip-mgrd.c:95-105 loop body: reading.c, budget2D.c:13-1736,
// uv_fluc.c:15-49) applied to the vel-* / den-* fields of the three levels.
//
// Pipeline (all FP64):
//   1. planar copy of each level's fields, q[c][k][j][i] with c = u, v, w and
//      den / 3 (the reference's pressure, budget2D.c:184);
//   2. plane means of the composite profile (budget2D.c:178-241): lower fine
//      planes 0..zdf-1, coarse planes 2..zdc-3, upper fine planes 0..zdf-1,
//      each summed in the reference's order, so they are bit-identical;
//   3. per-plane sums of the 44 products of fluctuations and their gradients
//      (budget2D.c:448-1002): 4th-order central differences in x and y,
//      the reference's plane-dependent rules in z (one-sided at the walls,
//      mixed-spacing at the level joins, reading the neighbouring level);
//   4. on the host, the O(NZ) finalisation of budget2D.c:1004-1550: plane
//      averages, rms, skewness, flatness, vorticity rms, production,
//      turbulent / pressure / viscous transport, pressure strain, dissipation.
// Block partials of the 44 products are summed in a fixed order, so results are
// deterministic; they differ from the reference's sequential plane sums by
// rounding only.
// This unit is built without fused multiply-add, like the reference.
#include <cmath>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

#include <cuda_runtime.h>

#include "host.h"
#include "kernels.h"
#include "lattice.cuh"

namespace dns {

namespace {

constexpr int kT = 128;  // threads per block
constexpr int kNS = 44;  // per-plane sums of the budget pass

// accumulator order (the reference's reduction order, budget2D.c:1070-1244)
enum {
  S_UU, S_UV, S_UW, S_VV, S_VW, S_WW, S_DD,
  S_SKU, S_SKV, S_SKW, S_SKP, S_SKUW, S_SKUV, S_SKVW,
  S_KUU, S_KUV, S_KUW, S_KUP, S_KUUW, S_KUVW, S_KUUV,
  S_WX, S_WY, S_WZ, S_UUW, S_VVW, S_WWW, S_UWW, S_PU, S_PV, S_PW,
  S_PAIUU, S_PAIVV, S_PAIWW, S_PAIUW, S_EPUU, S_EPVV, S_EPWW, S_EPUW,
  S_USUW, S_VSVW, S_WSWW, S_WSUW, S_USWW, S_COUNT
};
static_assert(S_COUNT == kNS, "44 budget sums");

struct TkeArgs {
  const double *q[3];  // planar fields per level (0 coarse, 1 lower fine, 2 upper fine)
  const double *mean;  // [NZ][4] plane means of u, v, w, den/3
  double *part;        // [NZ][nymax][W] partials of kRows rows each
  int nx[3], ny[3], nz[3];
  int gr, zdf, zdc, NZ, nymax;
  double coef;         // 1 / GR
};

// sum c of the block goes to out[to[c]]
template <int N>
__device__ __forceinline__ void block_sum(double (&v)[N], double *out, const unsigned char *to) {
  __shared__ double red[N][kT / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < N; q++) {
    double x = v[q];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if (lane == 0) red[q][warp] = x;
  }
  __syncthreads();
  for (int q = threadIdx.x; q < N; q += blockDim.x) {
    double s = red[q][0];
#pragma unroll
    for (int w = 1; w < kT / 32; w++) s += red[q][w];
    out[to[q]] = s;
  }
}

// reference file layout vel[i][j][k][3], den[i][j][k] -> q[c][k][j][i]
__global__ void __launch_bounds__(kT) tke_planar_kernel(const double *__restrict__ vel,
                                                        const double *__restrict__ den, int nx, int ny, int nz,
                                                        double *__restrict__ q) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y, k = blockIdx.z;
  if (i >= nx) return;
  const size_t node = ((size_t)i * ny + j) * nz + k, plane = (size_t)nz * ny * nx;
  const size_t o = ((size_t)k * ny + j) * nx + i;
  q[o] = vel[node * 3];
  q[plane + o] = vel[node * 3 + 1];
  q[2 * plane + o] = vel[node * 3 + 2];
  q[3 * plane + o] = (1. / 3.) * den[node];
}

// composite-profile plane of (level, k)
__device__ __forceinline__ int profile_of(const TkeArgs &A, int l, int k) {
  return l == 1 ? k : (l == 0 ? A.zdf - 2 + k : A.zdf + A.zdc - 4 + k);
}

// ------------------------------------------------------------ ordered sums
// Sums of NF sequences of n values, each in sequence order (the reference's plane
// loops: the results are its to the last bit).  The chain of n dependent adds
// sets the time (8.3 cycles an add on B200: 0.57 ms for 131,072 nodes); everything
// else is kept off it.  Warps 1.. form the values of a chunk in shared memory
// while lanes 0..NF-1 of warp 0 add the previous one, each lane its own sequence,
// sixteen values ahead in registers: 0.58 ms for 131,072 nodes.  (Staged, waited
// for and added in turn by the same warps: 38 cycles an add, 2.6 ms.)
// value(t, v): the NF values at position t.  Result in out[NF] (shared), visible
// to every thread of the block on return; kSumThreads threads.
constexpr int kSumChunk = 512, kSumThreads = 160;
template <int NF>
struct alignas(16) SumSmem {  // read in 16-byte pairs
  // rows two banks apart: the adding lanes read the same position of NF rows
  double buf[2][NF][kSumChunk + 2];
};

template <int NF, class Value>
__device__ __forceinline__ void ordered_sums(SumSmem<NF> &S, size_t n, Value value, double *out) {
  static_assert(NF <= 32, "one lane a sequence");
  static_assert(alignof(SumSmem<NF>) >= 16 && (kSumChunk + 2) % 2 == 0, "every row starts on 16 bytes");
  constexpr int W = kSumThreads - 32, PER = kSumChunk / W;
  const int t0 = (int)threadIdx.x - 32, lane = threadIdx.x & 31;
  auto produce = [&](size_t base, int b) {
    const int len = (int)(n - base < (size_t)kSumChunk ? n - base : (size_t)kSumChunk);
    double v[PER][NF];
#pragma unroll
    for (int r = 0; r < PER; r++)
      if (t0 + r * W < len) value(base + t0 + r * W, v[r]);
#pragma unroll
    for (int r = 0; r < PER; r++)
      if (t0 + r * W < len)
#pragma unroll
        for (int c = 0; c < NF; c++) S.buf[b][c][t0 + r * W] = v[r][c];
  };
  double s = 0.;
  if (t0 >= 0) produce(0, 0);
  __syncthreads();
  int b = 0;
  for (size_t base = 0; base < n; base += kSumChunk, b ^= 1) {
    if (t0 >= 0) {
      if (base + kSumChunk < n) produce(base + kSumChunk, b ^ 1);
    } else if (lane < NF) {
      const double *v = S.buf[b][lane];
      const int len = (int)(n - base < (size_t)kSumChunk ? n - base : (size_t)kSumChunk);
      if (len == kSumChunk) {
        double2 x[8], y[8];
        const double2 *w = reinterpret_cast<const double2 *>(v);
#pragma unroll
        for (int q = 0; q < 8; q++) x[q] = w[q];
#pragma unroll 1
        for (int t = 0; t < kSumChunk / 2; t += 16) {
#pragma unroll
          for (int q = 0; q < 8; q++) y[q] = w[t + 8 + q];
#pragma unroll
          for (int q = 0; q < 8; q++) {
            s += x[q].x;
            s += x[q].y;
          }
#pragma unroll
          for (int q = 0; q < 8; q++) x[q] = w[(t + 16 + q) % (kSumChunk / 2)];  // the last ones are not used
#pragma unroll
          for (int q = 0; q < 8; q++) {
            s += y[q].x;
            s += y[q].y;
          }
        }
      } else {
        for (int t = 0; t < len; t++) s += v[t];
      }
    }
    __syncthreads();
  }
  if (t0 < 0 && lane < NF) out[lane] = s;
  __syncthreads();
}

// plane means of u, v, w, den / 3, each plane summed in its memory order (j outer,
// i inner: the reference's) and divided by its node count (budget2D.c:178-241);
// one block per profile plane K
__global__ void __launch_bounds__(kSumThreads) tke_mean_seq(TkeArgs A, double *__restrict__ mean) {
  __shared__ SumSmem<4> S;
  __shared__ double sum[4];
  const int K = blockIdx.x;
  const int l = K < A.zdf ? 1 : (K < A.zdf + A.zdc - 4 ? 0 : 2);
  const int k = l == 1 ? K : (l == 0 ? K - A.zdf + 2 : K - (A.zdf + A.zdc - 4));
  const size_t n = (size_t)A.nx[l] * A.ny[l], field = (size_t)A.nz[l] * n;
  const double *q = A.q[l] + (size_t)k * n;
  ordered_sums<4>(S, n, [&](size_t t, double (&v)[4]) {
#pragma unroll
    for (int c = 0; c < 4; c++) v[c] = q[c * field + t];
  }, sum);
  if (threadIdx.x < 4) mean[(size_t)K * 4 + threadIdx.x] = sum[threadIdx.x] / (double)(A.nx[l] * A.ny[l]);
}

// ------------------------------------------------------------ plane-statistics record
// statistics.c:48-300 on the device: per profile plane the means of u, v, w and
// the density, then the mean squares of the deviations from them and of
// u' w', each summed over the plane in the reference's order (i outer, j inner).
// The fields first, per plane [c][plane][i][j], transposed through shared memory.
template <class T>
__device__ __forceinline__ double population(const T *p, int a);
template <>
__device__ __forceinline__ double population<double>(const double *p, int) {
  return *p;
}
template <>
__device__ __forceinline__ double population<float>(const float *p, int a) {  // as the exported state
  const double w = a == 0 ? 1. / 3. : (a <= 6 ? 1. / 18. : 1. / 36.);
  return w + (double)*p;
}

template <class T>
__global__ void __launch_bounds__(256) record_fields(const T *__restrict__ soa, int nx, int ny, int P, int p0, int np,
                                                     double *__restrict__ q) {
  __shared__ double tile[4][32][33];
  const int i0 = blockIdx.x * 32, j0 = blockIdx.y * 32, k = blockIdx.z;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const size_t plane = (size_t)ny * nx, stride = (size_t)P * plane;
  const T *s = soa + (size_t)(p0 + k) * plane;
  for (int r = ty; r < 32; r += 8)
    if (i0 + tx < nx && j0 + r < ny) {
      const T *f = s + (size_t)(j0 + r) * nx + i0 + tx;
      double g[19];
#pragma unroll
      for (int a = 0; a < 19; a++) g[a] = population<T>(f + (size_t)a * stride, a);
      double dens, mx, my, mz;
      moments_f64(g, dens, mx, my, mz);
      if (!isfinite(dens)) {  // 0 f of the definition's sums is not 0 where f is not finite
        mx = my = mz = 0.;
#pragma unroll
        for (int a = 0; a < 19; a++) {
          mx += (double)ex_of(a) * g[a];
          my += (double)ey_of(a) * g[a];
          mz += (double)ez_of(a) * g[a];
        }
      }
      tile[0][r][tx] = mx / dens;
      tile[1][r][tx] = my / dens;
      tile[2][r][tx] = mz / dens;
      tile[3][r][tx] = dens;
    }
  __syncthreads();
  for (int r = ty; r < 32; r += 8)
    if (i0 + r < nx && j0 + tx < ny)
#pragma unroll
      for (int c = 0; c < 4; c++) q[((size_t)c * np + k) * plane + (size_t)(i0 + r) * ny + j0 + tx] = tile[c][tx][r];
}

struct RecordLevel {
  const double *q;  // [4][np][nodes]
  double *out;      // [np][9]: means of u, v, w, density; mean squares uu, vv, ww, uw, rr
  size_t nodes;     // per plane
  int np;
};
// one block per plane, the fine level's first (they take longest)
__global__ void __launch_bounds__(kSumThreads) record_sums(RecordLevel fine, RecordLevel coarse) {
  __shared__ union {
    SumSmem<4> a;
    SumSmem<5> b;
  } S;
  __shared__ double mean[4], sum[5];
  const bool f = (int)blockIdx.x < fine.np;
  const RecordLevel &L = f ? fine : coarse;
  const int k = f ? blockIdx.x : blockIdx.x - fine.np;
  const size_t n = L.nodes, field = (size_t)L.np * n;
  const double *q = L.q + (size_t)k * n;
  const double norm = (double)n;
  ordered_sums<4>(S.a, n, [&](size_t t, double (&v)[4]) {
#pragma unroll
    for (int c = 0; c < 4; c++) v[c] = q[c * field + t];
  }, sum);
  if (threadIdx.x < 4) mean[threadIdx.x] = L.out[(size_t)k * 9 + threadIdx.x] = sum[threadIdx.x] / norm;
  __syncthreads();
  ordered_sums<5>(S.b, n, [&](size_t t, double (&v)[5]) {
    const double u = q[t] - mean[0], w = q[2 * field + t] - mean[2], vv = q[field + t] - mean[1],
                 d = q[3 * field + t] - mean[3];
    v[0] = u * u;
    v[1] = vv * vv;
    v[2] = w * w;
    v[3] = u * w;
    v[4] = d * d;
  }, sum);
  if (threadIdx.x < 5) L.out[(size_t)k * 9 + 4 + threadIdx.x] = sum[threadIdx.x] / norm;
}

// plane totals of W row partials in row order
__global__ void tke_sum_rows(const double *__restrict__ part, int nymax, int W, const int *__restrict__ rows,
                             double *__restrict__ out) {
  const int K = blockIdx.x;
  for (int q = threadIdx.x; q < W; q += blockDim.x) {
    double s = 0.;
    for (int j = 0; j < rows[K]; j++) s += part[((size_t)K * nymax + j) * W + q];
    out[(size_t)K * W + q] = s;
  }
}

// fluctuation of field c at (i, j, k) of level l (budget2D.c:243-291)
__device__ __forceinline__ double fl(const TkeArgs &A, int l, int c, int i, int j, int k) {
  const int nx = A.nx[l], ny = A.ny[l], nz = A.nz[l];
  return A.q[l][(((size_t)c * nz + k) * ny + j) * nx + i] - A.mean[profile_of(A, l, k) * 4 + c];
}

__device__ __forceinline__ int wrapn(int v, int n) { return v < 0 ? v + n : (v >= n ? v - n : v); }

// d/dz of field c at (i, j, k) of level l by the reference's plane rules
// (lower budget2D.c:548-599, coarse :732-761, upper :924-975)
__device__ __forceinline__ double ddz(const TkeArgs &A, int l, int c, int i, int j, int k) {
  const int gr = A.gr, zdf = A.zdf, zdc = A.zdc;
  const double coef = A.coef;
  if (l == 1) {
    if (k == 1) {
      const double q0 = fl(A, 1, c, i, j, k), q1 = fl(A, 1, c, i, j, k + 1), q2 = fl(A, 1, c, i, j, k + 2);
      const double q3 = fl(A, 1, c, i, j, k + 3), q4 = fl(A, 1, c, i, j, k + 4);
      const double tmp = (2. / 3.) * (q3 - q1) - (1. / 12.) * (q4 - q0);
      return -(7. / 3.) * q0 + 6. * q1 - 3. * q2 - (2. / 3.) * q3 + 3. * tmp;
    }
    if (k == zdf - 1) {
      const double qc = fl(A, 0, c, i / gr, j / gr, 2);
      const double q0 = fl(A, 1, c, i, j, k), qm = fl(A, 1, c, i, j, k - 1);
      return (coef * (qc - q0) + gr * (q0 - qm)) * 1. / (1. + gr);
    }
    return 0.5 * (fl(A, 1, c, i, j, k + 1) - fl(A, 1, c, i, j, k - 1));
  }
  if (l == 0) {
    if (k == 2) return 0.5 * coef * (fl(A, 0, c, i, j, k + 1) - fl(A, 1, c, i * gr, j * gr, zdf - 1));
    if (k == 3 || k == zdc - 4) return 0.5 * coef * (fl(A, 0, c, i, j, k + 1) - fl(A, 0, c, i, j, k - 1));
    if (k == zdc - 3) return 0.5 * coef * (fl(A, 2, c, i * gr, j * gr, 0) - fl(A, 0, c, i, j, k - 1));
    return 0.5 * coef * (fl(A, 0, c, i, j, k + 1) - fl(A, 0, c, i, j, k - 1));
  }
  if (k == 0) {
    const double q0 = fl(A, 2, c, i, j, 0), q1 = fl(A, 2, c, i, j, 1);
    const double qc = fl(A, 0, c, i / gr, j / gr, zdc - 3);
    return (gr * (q1 - q0) + coef * (q0 - qc)) * 1. / (1. + gr);
  }
  if (k == zdf - 2) {
    const double q0 = fl(A, 2, c, i, j, k), q1 = fl(A, 2, c, i, j, k - 1), q2 = fl(A, 2, c, i, j, k - 2);
    const double q3 = fl(A, 2, c, i, j, k - 3), q4 = fl(A, 2, c, i, j, k - 4);
    const double tmp = (2. / 3.) * (q1 - q3) - (1. / 12.) * (q0 - q4);
    return (7. / 3.) * q0 - 6. * q1 + 3. * q2 + (2. / 3.) * q3 + 3. * tmp;
  }
  return 0.5 * (fl(A, 2, c, i, j, k + 1) - fl(A, 2, c, i, j, k - 1));
}

// The 44 per-node terms of budget2D.c:448-624 (and the identical coarse and
// upper bodies), summed over kRows rows of plane k of level L (lower fine
// 1..zdf-1, coarse 2..zdc-3, upper fine 0..zdf-2).  FP64 latency bounds it: two
// kinds of block, one for the 28 products of the fluctuations alone, one for the
// 16 with gradients, keep the sums of a thread in fewer registers (255 with
// spills for all 44) and twice the warps on an SM; and as the block sums take as
// many instructions as some five nodes of a thread, a block takes four rows.
// 256x128x83: 633 us with one block a row and all sums, 503 us with four rows,
// 393 / 320 / 304 us with two kinds of block at 3 / 4 / 5 of them on an SM.
constexpr int kRows = 4;
constexpr int kNV = 28, kNG = 16;
__constant__ unsigned char c_val_sum[kNV] = {
    S_UU, S_UV, S_UW, S_VV, S_VW, S_WW, S_DD, S_SKU, S_SKV, S_SKW, S_SKP, S_SKUW, S_SKUV, S_SKVW,
    S_KUU, S_KUV, S_KUW, S_KUP, S_KUUW, S_KUVW, S_KUUV, S_UUW, S_VVW, S_WWW, S_UWW, S_PU, S_PV, S_PW};
__constant__ unsigned char c_grad_sum[kNG] = {S_WX, S_WY, S_WZ, S_PAIUU, S_PAIVV, S_PAIWW, S_PAIUW, S_EPUU,
                                              S_EPVV, S_EPWW, S_EPUW, S_USUW, S_VSVW, S_WSWW, S_WSUW, S_USWW};

__device__ __forceinline__ void value_rows(const TkeArgs &A, int l, int k, int jb) {
  const int K = profile_of(A, l, k), nx = A.nx[l], ny = A.ny[l];
  const size_t n = (size_t)ny * nx, field = (size_t)A.nz[l] * n;
  const double *q = A.q[l] + (size_t)k * n, *m = A.mean + (size_t)K * 4;
  const double um = m[0], vm = m[1], wm = m[2], dm = m[3];
  double s[kNV];
#pragma unroll
  for (int c = 0; c < kNV; c++) s[c] = 0.;
  // the block's rows are one run of memory
  const size_t lo = (size_t)jb * kRows * nx, hi = min(n, lo + (size_t)kRows * nx);
  for (size_t t = lo + threadIdx.x; t < hi; t += blockDim.x) {
    const double u = q[t] - um, v = q[field + t] - vm, w = q[2 * field + t] - wm, d = q[3 * field + t] - dm;
    s[0] += u * u;
    s[1] += u * v;
    s[2] += u * w;
    s[3] += v * v;
    s[4] += v * w;
    s[5] += w * w;
    s[6] += d * d;
    s[7] += u * u * u;
    s[8] += v * v * v;
    s[9] += w * w * w;
    s[10] += d * d * d;
    s[11] += u * u * u * w * w * w;
    s[12] += u * u * u * v * v * v;
    s[13] += v * v * v * w * w * w;
    s[14] += u * u * u * u;
    s[15] += v * v * v * v;
    s[16] += w * w * w * w;
    s[17] += d * d * d * d;
    s[18] += u * u * u * u * w * w * w * w;
    s[19] += v * v * v * v * w * w * w * w;
    s[20] += u * u * u * u * v * v * v * v;
    s[21] += u * u * w;
    s[22] += v * v * w;
    s[23] += w * w * w;
    s[24] += u * w * w;
    s[25] += u * d;
    s[26] += v * d;
    s[27] += w * d;
  }
  block_sum<kNV>(s, A.part + ((size_t)K * A.nymax + jb) * kNS, c_val_sum);
}

template <int L>
__device__ __forceinline__ void gradient_rows(const TkeArgs &A, int k, int jb) {
  constexpr int l = L;
  const int K = profile_of(A, L, k), nx = A.nx[l], ny = A.ny[l];
  const double cx = l == 0 ? A.coef : 1.;
  const double davg = A.mean[K * 4 + 3];
  double s[kNG];
#pragma unroll
  for (int c = 0; c < kNG; c++) s[c] = 0.;
  for (int j = jb * kRows; j < min((jb + 1) * kRows, ny); j++) {
    const int jp = wrapn(j - 1, ny), jpp = wrapn(j - 2, ny), jn = wrapn(j + 1, ny), jnn = wrapn(j + 2, ny);
    for (int i = threadIdx.x; i < nx; i += blockDim.x) {
      const int ip = wrapn(i - 1, nx), ipp = wrapn(i - 2, nx), in = wrapn(i + 1, nx), inn = wrapn(i + 2, nx);
      const double u = fl(A, l, 0, i, j, k), v = fl(A, l, 1, i, j, k), w = fl(A, l, 2, i, j, k);
      const double dfl = A.q[l][(((size_t)3 * A.nz[l] + k) * ny + j) * nx + i] - davg;
      double gx[3], gy[3], gz[3];
#pragma unroll
      for (int c = 0; c < 3; c++) {
        // along x and y the plane mean cancels
        const double *qc = A.q[l] + ((size_t)c * A.nz[l] + k) * ny * nx, *qr = qc + (size_t)j * nx;
        const double dx = (2. / 3.) * (qr[in] - qr[ip]) - (1. / 12.) * (qr[inn] - qr[ipp]);
        const double dy = (2. / 3.) * (qc[(size_t)jn * nx + i] - qc[(size_t)jp * nx + i]) -
                          (1. / 12.) * (qc[(size_t)jnn * nx + i] - qc[(size_t)jpp * nx + i]);
        gx[c] = l == 0 ? cx * dx : dx;
        gy[c] = l == 0 ? cx * dy : dy;
        gz[c] = ddz(A, l, c, i, j, k);
      }
      const double dudx = gx[0], dvdx = gx[1], dwdx = gx[2];
      const double dudy = gy[0], dvdy = gy[1], dwdy = gy[2];
      const double dudz = gz[0], dvdz = gz[1], dwdz = gz[2];
      const double ox = (dwdy - dvdz), oy = (dudz - dwdx), oz = (dvdx - dudy);
      s[0] += ox * ox;
      s[1] += oy * oy;
      s[2] += oz * oz;
      s[3] += dfl * dudx;
      s[4] += dfl * dvdy;
      s[5] += dfl * dwdz;
      s[6] += dfl * (dudz + dwdx);
      s[7] += dudx * (dudx + dudx) + dudy * (dudy + dvdx) + dudz * (dudz + dwdx);
      s[8] += dvdx * (dvdx + dudy) + dvdy * (dvdy + dvdy) + dvdz * (dvdz + dwdy);
      s[9] += dwdx * (dwdx + dudz) + dwdy * (dwdy + dvdz) + dwdz * (dwdz + dwdz);
      s[10] += dudx * (dwdx + dudz) + dudy * (dwdy + dvdz) + dudz * (dwdz + dwdz) + dwdx * (dudx + dudx) +
               dwdy * (dudy + dvdx) + dwdz * (dudz + dwdx);
      s[11] += 0.5 * u * (dudz + dwdx);
      s[12] += 0.5 * v * (dvdz + dwdy);
      s[13] += 0.5 * w * (dwdz + dwdz);
      s[14] += 0.5 * w * (dudz + dwdx);
      s[15] += 0.5 * u * (dwdz + dwdz);
    }
  }
  block_sum<kNG>(s, A.part + ((size_t)K * A.nymax + jb) * kNS, c_grad_sum);
}

// both kinds of block of every level in one launch: the gradients, which take
// longer, first, and of each the fine blocks' planes first
__global__ void __launch_bounds__(kT, 5) tke_budget_rows(TkeArgs A) {
  const int nf = (A.ny[1] + kRows - 1) / kRows, nc = (A.ny[0] + kRows - 1) / kRows, pf = A.zdf - 1, pc = A.zdc - 4;
  const int half = 2 * nf * pf + nc * pc;
  const bool grad = (int)blockIdx.x < half;
  int b = grad ? blockIdx.x : blockIdx.x - half;
  if (b < nf * pf) {
    if (grad) gradient_rows<1>(A, 1 + b / nf, b % nf);
    else value_rows(A, 1, 1 + b / nf, b % nf);
  } else if ((b -= nf * pf) < nf * pf) {
    if (grad) gradient_rows<2>(A, b / nf, b % nf);
    else value_rows(A, 2, b / nf, b % nf);
  } else {
    b -= nf * pf;
    if (grad) gradient_rows<0>(A, 2 + b / nc, b % nc);
    else value_rows(A, 0, 2 + b / nc, b % nc);
  }
}

// ------------------------------------------------------------ finalisation
// budget2D.c:1004-1550 on the plane sums; profile rows in the order of the
// three output files (turb-fld-2d :1555-1579, vort-fluc-2d :1585-1587,
// KE-Budget-2d :1592-1639).
enum {
  P_UAVG, P_VAVG, P_WAVG, P_UTIN, P_VTIN, P_WTIN, P_UW, P_DAVG, P_DTIN, P_SKU, P_SKV, P_SKW, P_SKUW, P_SKP,
  P_KUU, P_KUV, P_KUW, P_KUUW, P_KUP,
  P_WX, P_WY, P_WZ,
  P_PII, P_PUU, P_PVV, P_PWW, P_PUW, P_TIIR, P_TUUR, P_TVVR, P_TWWR, P_TUWR, P_TIIPAI, P_TUUPAI, P_TVVPAI,
  P_TWWPAI, P_TUWPAI, P_PAIUU, P_PAIVV, P_PAIWW, P_PAIUW, P_TIIS, P_TUUS, P_TVVS, P_TWWS, P_TUWS, P_EPII,
  P_EPUU, P_EPVV, P_EPWW, P_EPUW, P_KE, P_COUNT
};
static_assert(P_COUNT == DNS_TKE_NPROF, "profile count");

// the reference's profile-derivative macros (TKE-budget/computations/definitions.h:56-94)
inline double ddz1f(const std::vector<double> &a, int k) { return (a[k + 1]) - (a[k]); }
inline double ddz1b(const std::vector<double> &a, int k) { return (a[k]) - (a[k - 1]); }
inline double ddz2c(const std::vector<double> &a, int k) { return ((a[k + 1]) - (a[k - 1])) * 0.5; }
inline double ddz2cnul(const std::vector<double> &a, int k, double r) {
  return (1. / (1. + r)) * ((1. / r) * ((a[k + 1]) - (a[k])) + r * ((a[k]) - (a[k - 1])));
}
inline double ddz2cnuu(const std::vector<double> &a, int k, double r) {
  return (1. / (1. + r)) * ((1. / r) * ((a[k]) - (a[k - 1])) + r * ((a[k + 1]) - (a[k])));
}

void finalize(const TkeArgs &A, double nu, const double *mean, const double *sums, double *prof) {
  const int NZ = A.NZ, zdf = A.zdf, zdc = A.zdc, GR = A.gr;
  const double coef = A.coef;
  auto col = [&](int q) {
    std::vector<double> v(NZ);
    for (int K = 0; K < NZ; K++) v[K] = sums[(size_t)K * kNS + q];
    return v;
  };
  std::vector<double> U(NZ), V(NZ), W(NZ), D(NZ);
  for (int K = 0; K < NZ; K++) {
    U[K] = mean[K * 4];
    V[K] = mean[K * 4 + 1];
    W[K] = mean[K * 4 + 2];
    D[K] = mean[K * 4 + 3];
  }
  std::vector<double> uu = col(S_UU), uv = col(S_UV), uw = col(S_UW), vv = col(S_VV), vw = col(S_VW),
                      ww = col(S_WW), dd = col(S_DD), SKu = col(S_SKU), SKv = col(S_SKV), SKw = col(S_SKW),
                      SKp = col(S_SKP), SKuw = col(S_SKUW), SKuv = col(S_SKUV), SKvw = col(S_SKVW),
                      KUu = col(S_KUU), KUv = col(S_KUV), KUw = col(S_KUW), KUp = col(S_KUP), KUuw = col(S_KUUW),
                      KUvw = col(S_KUVW), KUuv = col(S_KUUV), wx = col(S_WX), wy = col(S_WY), wz = col(S_WZ),
                      uuw = col(S_UUW), vvw = col(S_VVW), www = col(S_WWW), uww = col(S_UWW), pu = col(S_PU),
                      pv = col(S_PV), pw = col(S_PW), Paiuu = col(S_PAIUU), Paivv = col(S_PAIVV),
                      Paiww = col(S_PAIWW), Paiuw = col(S_PAIUW), Epuu = col(S_EPUU), Epvv = col(S_EPVV),
                      Epww = col(S_EPWW), Epuw = col(S_EPUW), usuw = col(S_USUW), vsvw = col(S_VSVW),
                      wsww = col(S_WSWW), wsuw = col(S_WSUW), usww = col(S_USWW);
  std::vector<double *> all = {uu.data(),   uv.data(),    uw.data(),    vv.data(),    vw.data(),   ww.data(),
                               dd.data(),   SKu.data(),   SKv.data(),   SKw.data(),   SKp.data(),  SKuw.data(),
                               SKuv.data(), SKvw.data(),  KUu.data(),   KUv.data(),   KUw.data(),  KUp.data(),
                               KUuw.data(), KUuv.data(),  KUvw.data(),  wx.data(),    wy.data(),   wz.data(),
                               uuw.data(),  vvw.data(),   www.data(),   uww.data(),   pu.data(),   pv.data(),
                               pw.data(),   Paiuu.data(), Paivv.data(), Paiww.data(), Paiuw.data(), Epuu.data(),
                               Epvv.data(), Epww.data(),  Epuw.data(),  usuw.data(),  vsvw.data(), wsww.data(),
                               wsuw.data(), usww.data()};
  // :1004-1064 plane averages
  for (int K = 0; K < NZ; K++) {
    long num;
    if (K < zdf) num = (long)A.nx[1] * A.ny[1];
    else if (K < zdf + zdc - 4) num = (long)A.nx[0] * A.ny[0];
    else num = (long)A.nx[2] * A.ny[2];
    for (double *a : all) a[K] /= (double)(num);
  }
  // mean shear (:295-444)
  std::vector<double> dUdz(NZ, 0.);
  for (int k = 1; k < zdf; k++) {
    if (k == 1) {
      const double tmp = (2. / 3.) * (U[k + 3] - U[k + 1]) - (1. / 12.) * (U[k + 4] - U[k]);
      dUdz[k] = -(7. / 3.) * U[k] + 6. * U[k + 1] - 3. * U[k + 2] - (2. / 3.) * U[k + 3] + 3. * tmp;
    } else if (k == zdf - 1) {
      dUdz[k] = (coef * (U[k + 1] - U[k]) + GR * (U[k] - U[k - 1])) * 1. / (1. + GR);
    } else if (k == 2 || k == zdf - 2) {
      dUdz[k] = 0.5 * (U[k + 1] - U[k - 1]);
    } else {
      dUdz[k] = (2. / 3.) * (U[k + 1] - U[k - 1]) - (1. / 12.) * (U[k + 2] - U[k - 2]);
    }
  }
  for (int k = 2; k < zdc - 2; k++) {
    const int K = zdf - 2 + k;
    if (k == 2 || k == 3 || k == zdc - 4 || k == zdc - 3)
      dUdz[K] = 0.5 * coef * (U[K + 1] - U[K - 1]);
    else
      dUdz[K] = coef * ((2. / 3.) * (U[K + 1] - U[K - 1]) - (1. / 12.) * (U[K + 2] - U[K - 2]));
  }
  for (int k = 0; k < zdf - 1; k++) {
    const int K = zdf + zdc - 4 + k;
    if (k == 0) {
      dUdz[K] = (GR * (U[K + 1] - U[K]) + coef * (U[K] - U[K - 1])) * 1. / (1. + GR);
    } else if (k == zdf - 2) {
      const double tmp = (2. / 3.) * (U[K - 1] - U[K - 3]) - (1. / 12.) * (U[K] - U[K - 4]);
      dUdz[K] = (7. / 3.) * U[K] - 6. * U[K - 1] + 3. * U[K - 2] + (2. / 3.) * U[K - 3] + 3. * tmp;
    } else if (k == 1 || k == zdf - 3) {
      dUdz[K] = 0.5 * (U[K + 1] - U[K - 1]);
    } else {
      dUdz[K] = (2. / 3.) * (U[K + 1] - U[K - 1]) - (1. / 12.) * (U[K + 2] - U[K - 2]);
    }
  }
  std::vector<double> UTIN(NZ, 0.), VTIN(NZ, 0.), WTIN(NZ, 0.), DTIN(NZ, 0.), KE(NZ, 0.), Epii(NZ, 0.);
  // :1249-1284
  for (int k = 1; k < NZ - 1; k++) {
    const double siu = UTIN[k] = std::sqrt(uu[k]);
    const double siv = VTIN[k] = std::sqrt(vv[k]);
    const double siw = WTIN[k] = std::sqrt(ww[k]);
    const double sip = DTIN[k] = std::sqrt(dd[k]);
    KE[k] += (uu[k] + vv[k] + ww[k]);
    wx[k] = std::sqrt(wx[k]);
    wy[k] = std::sqrt(wy[k]);
    wz[k] = std::sqrt(wz[k]);
    SKu[k] /= (siu * siu * siu);
    SKv[k] /= (siv * siv * siv);
    SKw[k] /= (siw * siw * siw);
    SKp[k] /= (sip * sip * sip);
    SKuw[k] /= (siu * siu * siu * siw * siw * siw);
    SKvw[k] /= (siv * siv * siv * siw * siw * siw);
    SKuv[k] /= (siu * siu * siu * siv * siv * siv);
    KUu[k] /= (siu * siu * siu * siu);
    KUv[k] /= (siv * siv * siv * siv);
    KUw[k] /= (siw * siw * siw * siw);
    KUp[k] /= (sip * sip * sip * sip);
    KUuw[k] /= (siu * siu * siu * siu * siw * siw * siw * siw);
    KUuv[k] /= (siu * siu * siu * siu * siv * siv * siv * siv);
    KUvw[k] /= (siv * siv * siv * siv * siw * siw * siw * siw);
    Epuu[k] *= nu;
    Epvv[k] *= nu;
    Epww[k] *= nu;
    Epuw[k] *= (2. * nu);
    Epii[k] = (Epuu[k]) + (Epvv[k]) + (Epww[k]);
  }
  std::vector<double> Pii(NZ, 0.), Puu(NZ, 0.), Pvv(NZ, 0.), Pww(NZ, 0.), Puw(NZ, 0.), Tiir(NZ, 0.), Tuur(NZ, 0.),
      Tvvr(NZ, 0.), Twwr(NZ, 0.), Tuwr(NZ, 0.), Tiipai(NZ, 0.), Tuupai(NZ, 0.), Tvvpai(NZ, 0.), Twwpai(NZ, 0.),
      Tuwpai(NZ, 0.), Tiis(NZ, 0.), Tuus(NZ, 0.), Tvvs(NZ, 0.), Twws(NZ, 0.), Tuws(NZ, 0.);
  auto production = [&](int K) {
    Pii[K] = -(uw[K]) * (dUdz[K]);
    Puu[K] = 2. * (Pii[K]);
    Pvv[K] = 0.;
    Pww[K] = 0.;
    Puw[K] = -(ww[K]) * (dUdz[K]);
    Tuupai[K] = 0.;
    Tvvpai[K] = 0.;
  };
  // one transport rule: D is the profile derivative, h the factor of the
  // diagonal turbulent-transport terms
  auto fine_rule = [&](int K, auto Dz, double h) {
    Tuur[K] = h * Dz(uuw, K);
    Tvvr[K] = h * Dz(vvw, K);
    Twwr[K] = h * Dz(www, K);
    Tuwr[K] = -Dz(uww, K);
    Tiipai[K] = -Dz(pw, K);
    Twwpai[K] = -2. * Dz(pw, K);
    Tuwpai[K] = -Dz(pu, K);
    Tuus[K] = 2. * nu * Dz(usuw, K);
    Tvvs[K] = 2. * nu * Dz(vsvw, K);
    Twws[K] = 2. * nu * Dz(wsww, K);
    Tuws[K] = 2. * nu * Dz(wsuw, K) + 2. * nu * Dz(wsww, K);
  };
  auto d1f = [](const std::vector<double> &a, int K) { return ddz1f(a, K); };
  auto d1b = [](const std::vector<double> &a, int K) { return ddz1b(a, K); };
  auto d2c = [](const std::vector<double> &a, int K) { return ddz2c(a, K); };
  auto nul = [GR](const std::vector<double> &a, int K) { return ddz2cnul(a, K, GR); };
  auto nuu = [GR](const std::vector<double> &a, int K) { return ddz2cnuu(a, K, GR); };
  // lower fine (:1286-1381)
  for (int k = 1; k < zdf; k++) {
    production(k);
    if (k == 1) fine_rule(k, d1f, -1.);
    else if (k == zdf - 1) fine_rule(k, nul, -1.);
    else if (k == 2 || k == zdf - 2) fine_rule(k, d2c, -1.);
    else fine_rule(k, d2c, -0.5);
    Tiis[k] = 0.5 * (Tuus[k] + Tvvs[k] + Twws[k]);
    Tiir[k] = 0.5 * (Tuur[k] + Tvvr[k] + Twwr[k]);
  }
  // coarse (:1383-1465): the rules at k = 2, 3, zdc-4, zdc-3 coincide
  for (int k = 2; k < zdc - 2; k++) {
    const int K = zdf - 2 + k;
    production(K);
    if (k == 2 || k == 3 || k == zdc - 4 || k == zdc - 3) {
      Tuur[K] = -coef * ddz2c(uuw, K);
      Tvvr[K] = -coef * ddz2c(vvw, K);
      Twwr[K] = -coef * ddz2c(www, K);
      Tuwr[K] = -coef * ddz2c(uww, K);
      Tiipai[K] = -coef * ddz2c(pw, K);
      Twwpai[K] = -2. * coef * ddz2c(pw, K);
      Tuwpai[K] = -coef * ddz2c(pu, K);
      Tuus[K] = 2. * nu * coef * ddz2c(usuw, K);
      Tvvs[K] = 2. * nu * coef * ddz2c(vsvw, K);
      Twws[K] = 2. * nu * coef * ddz2c(wsww, K);
      Tuws[K] = 2. * nu * coef * ddz2c(wsuw, K) + 2. * nu * coef * ddz2c(wsww, K);
    } else {
      Tuur[K] = -coef * 0.5 * ddz2c(uuw, K);
      Tvvr[K] = -coef * 0.5 * ddz2c(vvw, K);
      Twwr[K] = -coef * 0.5 * ddz2c(www, K);
      Tuwr[K] = -coef * ddz2c(uww, K);
      Tiipai[K] = -coef * ddz2c(pw, K);
      Twwpai[K] = -2. * coef * ddz2c(pw, K);
      Tuwpai[K] = -coef * ddz2c(pu, K);
      Tuus[K] = coef * 2. * nu * ddz2c(usuw, K);
      Tvvs[K] = coef * 2. * nu * ddz2c(vsvw, K);
      Twws[K] = coef * 2. * nu * ddz2c(wsww, K);
      Tuws[K] = coef * 2. * nu * ddz2c(wsuw, K) + coef * 2. * nu * ddz2c(wsww, K);
    }
    Tiis[K] = 0.5 * (Tuus[K] + Tvvs[K] + Twws[K]);
    Tiir[K] = 0.5 * (Tuur[K] + Tvvr[K] + Twwr[K]);
  }
  // upper fine (:1467-1548)
  for (int k = 0; k < zdf - 1; k++) {
    const int K = zdf + zdc - 4 + k;
    production(K);
    if (k == 0) fine_rule(K, nuu, -1.);
    else if (k == zdf - 2) fine_rule(K, d1b, -1.);
    else if (k == 2 || k == zdf - 3) fine_rule(K, d2c, -1.);
    else fine_rule(K, d2c, -0.5);
    Tiis[K] = 0.5 * (Tuus[K] + Tvvs[K] + Twws[K]);
    Tiir[K] = 0.5 * (Tuur[K] + Tvvr[K] + Twwr[K]);
  }
  const std::vector<double> *rows[P_COUNT] = {
      &U,    &V,      &W,      &UTIN,   &VTIN,   &WTIN,   &uw,     &D,     &DTIN,  &SKu,  &SKv,  &SKw,  &SKuw,
      &SKp,  &KUu,    &KUv,    &KUw,    &KUuw,   &KUp,    &wx,     &wy,    &wz,    &Pii,  &Puu,  &Pvv,  &Pww,
      &Puw,  &Tiir,   &Tuur,   &Tvvr,   &Twwr,   &Tuwr,   &Tiipai, &Tuupai, &Tvvpai, &Twwpai, &Tuwpai, &Paiuu,
      &Paivv, &Paiww, &Paiuw,  &Tiis,   &Tuus,   &Tvvs,   &Twws,   &Tuws,  &Epii,  &Epuu, &Epvv, &Epww, &Epuw,
      &KE};
  for (int r = 0; r < P_COUNT; r++) std::memcpy(prof + (size_t)r * NZ, rows[r]->data(), (size_t)NZ * 8);
}

}  // namespace

int tke_validate(const dns_params &p) {
  if (p.zds < 5) return fail_with(DNS_EINVAL, "the budget needs zds >= 5 (its wall stencils reach 4 planes)");
  if (p.zdv < 7) return fail_with(DNS_EINVAL, "the budget needs zdv >= 7 (coarse planes 2..zdc-3 with 4-point rules)");
  if (p.ydv < 4 || p.xdv < 4) return fail_with(DNS_EINVAL, "the budget needs xdv, ydv >= 4 (5-point stencils)");
  return DNS_OK;
}

size_t tke_workspace_bytes(const dns_geometry &g) {
  const size_t NZ = g.nz_profile;
  return (NZ * ((g.nyf + kRows - 1) / kRows) * kNS + NZ * 4 + NZ * kNS) * 8 + NZ * sizeof(int);
}

int tke_budget_planar(const dns_params &p, const dns_geometry &g, const double *const q[3], double *prof,
                      double *ufl, double *vfl, cudaStream_t st, void *work) {
  int rc = tke_validate(p);
  if (rc) return rc;
  TkeArgs A{};
  A.nx[0] = g.nx;
  A.ny[0] = g.ny;
  A.nz[0] = g.nzc;
  for (int l = 1; l < 3; l++) {
    A.nx[l] = g.nxf;
    A.ny[l] = g.nyf;
    A.nz[l] = g.zdf;
  }
  for (int l = 0; l < 3; l++) A.q[l] = q[l];
  A.gr = g.gr;
  A.zdf = g.zdf;
  A.zdc = g.nzc;
  A.NZ = g.nz_profile;
  A.nymax = (g.nyf + kRows - 1) / kRows;
  A.coef = (1. / ((double)g.gr));
  const int NZ = A.NZ;
  // budget2D.c:57-60, tauf the fine relaxation time
  const double tauf = (3. / p.Rebs) * p.ub * (g.nzs - 2.) + 0.5;
  const double nu = (1. / 6.) * (2. * tauf - 1.);
  const size_t npart = (size_t)NZ * A.nymax * kNS;
  const size_t nbuf = npart + (size_t)NZ * 4 + (size_t)NZ * kNS;
  void *owned = nullptr;
  if (!work) {
    if (cudaMalloc(&owned, tke_workspace_bytes(g)) != cudaSuccess) return fail_with(DNS_ENOMEM, "budget work space");
    work = owned;
  }
  double *buf = static_cast<double *>(work);
  int *dims = reinterpret_cast<int *>(buf + nbuf);
  double *part = buf, *mean = part + npart, *sums = mean + (size_t)NZ * 4;
  std::vector<int> hdims(NZ);
  const int nyc = (g.ny + kRows - 1) / kRows, nyf = (g.nyf + kRows - 1) / kRows;  // row blocks of a plane
  for (int K = 0; K < NZ; K++) hdims[K] = (K >= g.zdf && K < g.zdf + g.nzc - 4) ? nyc : nyf;
  A.part = part;
  A.mean = mean;
  cudaError_t e = cudaMemcpyAsync(dims, hdims.data(), NZ * sizeof(int), cudaMemcpyHostToDevice, st);
  if (e == cudaSuccess) {
    tke_mean_seq<<<NZ, kSumThreads, 0, st>>>(A, mean);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemsetAsync(part, 0, npart * 8, st);  // profile planes 0, NZ-1: no products
  if (e == cudaSuccess) {
    tke_budget_rows<<<2 * (2 * nyf * (g.zdf - 1) + nyc * (g.nzc - 4)), kT, 0, st>>>(A);
    tke_sum_rows<<<NZ, 64, 0, st>>>(part, A.nymax, kNS, dims, sums);
    e = cudaGetLastError();
  }
  std::vector<double> hmean((size_t)NZ * 4), hsums((size_t)NZ * kNS);
  if (e == cudaSuccess) e = cudaMemcpyAsync(hmean.data(), mean, hmean.size() * 8, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaMemcpyAsync(hsums.data(), sums, hsums.size() * 8, cudaMemcpyDeviceToHost, st);
  // uv_fluc.c:24-33: fluctuations of the lower fine plane k = 4
  const size_t pl = (size_t)g.nyf * g.nxf;
  std::vector<double> plane;
  if (e == cudaSuccess && (ufl || vfl)) {
    plane.resize(2 * pl);
    e = cudaMemcpyAsync(plane.data(), q[1] + 4 * pl, pl * 8, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(plane.data() + pl, q[1] + (size_t)g.zdf * pl + 4 * pl, pl * 8, cudaMemcpyDeviceToHost,
                          st);
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (owned) cudaFree(owned);
  if (e != cudaSuccess) return fail_with(DNS_ECUDA, cudaGetErrorString(e));
  finalize(A, nu, hmean.data(), hsums.data(), prof);
  if (ufl || vfl) {
    for (int i = 0; i < g.nxf; i++)
      for (int j = 0; j < g.nyf; j++) {
        if (ufl) ufl[(size_t)i * g.nyf + j] = plane[(size_t)j * g.nxf + i] - hmean[4 * 4 + 0];
        if (vfl) vfl[(size_t)i * g.nyf + j] = plane[pl + (size_t)j * g.nxf + i] - hmean[4 * 4 + 1];
      }
  }
  return DNS_OK;
}

template <class T>
static cudaError_t plane_record(const T *fc, const T *ff, double *qc, double *qf, const dns_geometry &g, double *fine,
                                double *coarse, cudaStream_t st) {
  const int zds = g.zdf - 1, npf = 2 * zds, npc = g.nzc - 4;
  const size_t nf = (size_t)g.nxf * g.nyf, nc = (size_t)g.nx * g.ny;
  const RecordLevel F{qf, qf + 4 * npf * nf, nf, npf}, C{qc, qc + 4 * npc * nc, nc, npc};
  record_fields<T><<<dim3((g.nxf + 31) / 32, (g.nyf + 31) / 32, npf), 256, 0, st>>>(ff, g.nxf, g.nyf, npf, 0, npf, qf);
  record_fields<T><<<dim3((g.nx + 31) / 32, (g.ny + 31) / 32, npc), 256, 0, st>>>(fc, g.nx, g.ny, g.nzc, 2, npc, qc);
  record_sums<<<npf + npc, kSumThreads, 0, st>>>(F, C);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaMemcpyAsync(fine, F.out, (size_t)npf * 9 * 8, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaMemcpyAsync(coarse, C.out, (size_t)npc * 9 * 8, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  return e;
}

int plane_record_device(const void *fc, const void *ff, bool f32, double *qc, double *qf, const dns_geometry &g,
                        double *fine, double *coarse, cudaStream_t st) {
  const cudaError_t e =
      f32 ? plane_record(static_cast<const float *>(fc), static_cast<const float *>(ff), qc, qf, g, fine, coarse, st)
          : plane_record(static_cast<const double *>(fc), static_cast<const double *>(ff), qc, qf, g, fine, coarse, st);
  return e == cudaSuccess ? DNS_OK : fail_with(DNS_ECUDA, cudaGetErrorString(e));
}

int tke_budget_device(const dns_params &p, const dns_geometry &g, const double *const vel[3],
                      const double *const den[3], double *prof, double *ufl, double *vfl, cudaStream_t st) {
  int rc = tke_validate(p);
  if (rc) return rc;
  const int nx[3] = {g.nx, g.nxf, g.nxf}, ny[3] = {g.ny, g.nyf, g.nyf}, nz[3] = {g.nzc, g.zdf, g.zdf};
  size_t nq = 0;
  for (int l = 0; l < 3; l++) nq += 4ull * nx[l] * ny[l] * nz[l];
  double *buf = nullptr;
  if (cudaMalloc(&buf, nq * 8) != cudaSuccess) return fail_with(DNS_ENOMEM, "budget planar fields");
  const double *q[3];
  double *ql = buf;
  cudaError_t e = cudaSuccess;
  for (int l = 0; l < 3 && e == cudaSuccess; l++) {
    q[l] = ql;
    dim3 grid((nx[l] + kT - 1) / kT, ny[l], nz[l]);
    tke_planar_kernel<<<grid, kT, 0, st>>>(vel[l], den[l], nx[l], ny[l], nz[l], ql);
    ql += 4ull * nx[l] * ny[l] * nz[l];
    e = cudaGetLastError();
  }
  rc = e == cudaSuccess ? tke_budget_planar(p, g, q, prof, ufl, vfl, st) : fail_with(DNS_ECUDA, cudaGetErrorString(e));
  cudaStreamSynchronize(st);
  cudaFree(buf);
  return rc;
}

}  // namespace dns
