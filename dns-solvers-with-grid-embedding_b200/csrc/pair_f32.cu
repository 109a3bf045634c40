// FP32 deviation form, single channel: two fine substeps in one pass (the tile
// work is pair_f32.cuh's).
#include "pair_f32.cuh"

namespace dns {

namespace {

using namespace f32;

template <int MODE>
__global__ void __launch_bounds__(32 * kPairMaxZds, 1)
    fine_pair_f32(const float *__restrict__ src, float *__restrict__ dst, const float *__restrict__ mid,
                  const int8_t *__restrict__ wf, Dims d, PairGrid g, float om, const DevState *st,
                  double *__restrict__ part, double *__restrict__ wpart, unsigned int *__restrict__ lost) {
  extern __shared__ __align__(16) float Mf[];
  __shared__ PairSync S;
  const int nblk = gridDim.x * gridDim.y, blk = blockIdx.y * gridDim.x + blockIdx.x;
  PairTile P;
  P.nx = d.nxf;
  P.ny = d.nyf;
  P.zds = d.zds;
  P.gr = d.gr;
  P.ntx = g.ntx;
  P.bx = blockIdx.x;
  P.y0 = blockIdx.y * g.ly;
  P.L = min(g.ly, d.nyf - P.y0);
  P.upper = blockIdx.z != 0;
  P.om = om;
  P.Gf = (float)((1. / (double)d.gr) * st->force);
  P.src = src;
  P.dst = dst;
  P.mid = mid;
  P.wf = wf;
  P.part = part + ((size_t)blockIdx.z * nblk + blk) * 2;
  P.wpart = wpart + (size_t)blk * 2;
  P.wstride = (size_t)nblk * 2;
  P.lost = lost;
  pair_tile<MODE>(Mf, S, P);
}

}  // namespace

PairGrid make_pair_grid_f32(const Dims &d) {
  PairGrid g;
  // 32-bit byte offsets in a population; pairs of columns
  if (d.zds > kPairMaxZds || 2LL * d.zds * d.nyf * d.nxf >= (1LL << 30) || d.nxf % 2) return g;
  g.ntx = pair_tiles_f32(d.nxf);
  pair_runs(d, d.zds <= 5 ? 3 : (d.zds <= 8 ? 2 : 1), g);
  return g;
}

// The single substeps of the FP32 form run at 88% of the HBM rate beside their
// interface transfers.  A pair takes 204 us on 256x128x83 where two of them take 222,
// at 36% of the HBM rate and 52% of the issue slots: latency, at the 16 warps that its
// shared rows and registers leave an SM.  All its transfers stand in front of it, so it
// pays where a step has two of them and the transfers go out together: GR 4.  Measured us per step, pairs against single
// substeps: GR 4, zds 16: 637 MB 799 / 986, zds 10: 199 MB 410 / 425, 112 MB
// 290 / 260; GR 2, zds 16: 319 MB 349 / 346, zds 8: 160 MB 272 / 248.
bool pairs_pay_f32(const Dims &d, const PairGrid &g) {
  return g.on() && d.gr == 4 && 2. * d.zds * d.nyf * d.nxf * 19 * 4 * 1e-6 >= 180.;
}

int prepare_pair_f32() {
  const int bytes = (int)pair_smem_f32(kPairMaxZds);
  const void *fn[4] = {(const void *)fine_pair_f32<0>, (const void *)fine_pair_f32<1>, (const void *)fine_pair_f32<2>,
                       (const void *)fine_pair_f32<3>};
  for (const void *f : fn)
    if (cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess) return -1;
  return 0;
}

void launch_fine_pair_f32(const float *src, float *dst, const float *mid, const int8_t *wflag, const Dims &d,
                          const PairGrid &g, double om, const DevState *st, double *part, double *wpart,
                          unsigned int *lost, bool first, bool last, cudaStream_t stream) {
  const dim3 grid(g.ntx, g.nly, 2), block(32 * d.zds);
  const size_t smem = pair_smem_f32(d.zds);
  const float omf = (float)om;
  switch ((last ? 1 : 0) | (first ? 2 : 0)) {
    case 0: fine_pair_f32<0><<<grid, block, smem, stream>>>(src, dst, mid, wflag, d, g, omf, st, part, wpart, lost); break;
    case 1: fine_pair_f32<1><<<grid, block, smem, stream>>>(src, dst, mid, wflag, d, g, omf, st, part, wpart, lost); break;
    case 2: fine_pair_f32<2><<<grid, block, smem, stream>>>(src, dst, mid, wflag, d, g, omf, st, part, wpart, lost); break;
    default: fine_pair_f32<3><<<grid, block, smem, stream>>>(src, dst, mid, wflag, d, g, omf, st, part, wpart, lost); break;
  }
}

}  // namespace dns
