// The filtered fine-to-coarse transfer (FLTR, ftcdtransfer_lesfltr.c:163-363,
// GR = 4) of a row segment of coarse vertices: f - feq of each of the 5 x 5 x 5
// fine nodes around a vertex (planes kb-2..kb+2, x and y wrapped), summed as
// (w f^neq) / GR^3 with the trapezoid weights (1/2, 1, 1, 1, 1/2) per axis, x outer,
// z inner; the equilibrium is that of the vertex node's density and momentum sums
// (the reference keeps the momentum where it reads the velocity back, :185-188,
// :222-225).
//
// A block takes kFiltV vertices of a row: its threads form f^neq of the fine nodes
// in shared memory, once for all the vertices that weigh them, then one thread
// per vertex and population sums its 125 terms in the reference's order.  (One
// thread per vertex, 125 nodes of 19 loads and a collision's moments each one
// after another: 321 us for 96 x 48 vertices a wall, 72 blocks; this way 77 us.)
//
// A: the arithmetic of the form.  A::T the stored type, A::R the computing type;
// neq(f, n, mac): non-equilibrium parts and the node's four moments; weight(w):
// the factor of a node of trapezoid weight w; result(a, mac, t, fac).
#pragma once

#include "kernels.h"
#include "lattice.cuh"

namespace dns {

constexpr int kFiltV = 4, kFiltX = 4 * kFiltV + 1, kFiltThreads = 256;
template <class R>
constexpr size_t filter_smem() {
  return sizeof(R) * ((size_t)19 * 25 * kFiltX + kFiltV * 4 + 2 * kFiltV * 19);
}

template <class A>
__device__ __forceinline__ void filtered_row(const typename A::T *__restrict__ fsrc, typename A::T *__restrict__ cdst,
                                             const Dims &d, int i0, int jc, int w, typename A::R fac,
                                             double *__restrict__ part, typename A::R *sm) {
  using R = typename A::R;
  const int gr = d.gr, zds = d.zds, nxf = d.nxf, nyf = d.nyf;
  R *const neq = sm, *const mac = sm + 19 * 25 * kFiltX, *const out = mac + kFiltV * 4;
  const int kb = w == 0 ? d.zdf - 1 - gr : gr;
  const size_t fplane = (size_t)nyf * nxf, fstride = (size_t)2 * zds * fplane;
  for (int q = threadIdx.x; q < 25 * kFiltX; q += blockDim.x) {
    // [jj][kk][x]: consecutive threads take consecutive fine nodes
    const int xx = q % kFiltX, jk = q / kFiltX, jj = jk / 5 - 2, kk = jk % 5 - 2;
    int x = i0 * gr + xx - 2, y = jc * gr + jj;
    x = x < 0 ? x + nxf : (x >= nxf ? (x - nxf) % nxf : x);
    y = y < 0 ? y + nyf : (y >= nyf ? y - nyf : y);
    const int k = kb + kk, p = w == 0 ? k - 1 : zds + k;
    const typename A::T *s = fsrc + (size_t)p * fplane + (size_t)y * nxf + x;
    R f[19], n[19], m[4];
#pragma unroll
    for (int a = 0; a < 19; a++) f[a] = __ldg(s + (size_t)a * fstride);
    A::neq(f, n, m);
#pragma unroll
    for (int a = 0; a < 19; a++) neq[(a * 25 + jk) * kFiltX + xx] = n[a];
    const int v = (xx - 2) / gr;
    if (jj == 0 && kk == 0 && xx >= 2 && (xx - 2) % gr == 0 && v < kFiltV)
#pragma unroll
      for (int c = 0; c < 4; c++) mac[v * 4 + c] = m[c];
  }
  __syncthreads();
  const int v = threadIdx.x / 19, a = threadIdx.x % 19;
  if (v < kFiltV && i0 + v < d.nx) {
    R t = 0;
    for (int ii = 0; ii < 5; ii++)
#pragma unroll
      for (int jj = 0; jj < 5; jj++)
#pragma unroll
        for (int kk = 0; kk < 5; kk++) {
          const R wx = (ii == 0 || ii == 4) ? R(0.5) : R(1), wy = (jj == 0 || jj == 4) ? R(0.5) : R(1),
                  wz = (kk == 0 || kk == 4) ? R(0.5) : R(1);
          t = A::add(t, wx * wy, wz, neq[(a * 25 + jj * 5 + kk) * kFiltX + v * 4 + ii]);
        }
    const R f = A::result(a, mac + v * 4, t, fac);
    const int kc = w == 0 ? 0 : d.nzc - 1;
    const size_t cstride = (size_t)d.nzc * d.ny * d.nx;
    cdst[(size_t)a * cstride + ((size_t)kc * d.ny + jc) * d.nx + i0 + v] = (typename A::T)f;
    out[v * 19 + a] = f;
  }
  __syncthreads();
  if (threadIdx.x == 0) {  // flow-rate partials, vertices and populations in order
    double mom = 0., den = 0.;
    for (int v = 0; v < kFiltV && i0 + v < d.nx; v++) {
      R vm = 0, vd = 0;
#pragma unroll
      for (int a = 0; a < 19; a++) {
        const R f = out[v * 19 + a];
        vd += f;
        if (ex_of(a) > 0) vm += f;
        if (ex_of(a) < 0) vm -= f;
      }
      mom += vm;
      den += vd;
    }
    part[0] = mom;
    part[1] = den;
  }
}

}  // namespace dns
