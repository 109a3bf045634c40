// FP32 deviation form: two fine substeps in one pass over the fine state, the
// tile work of pair_f32.cu.  The march along y, the live rows in shared memory and
// the barriers are those of pair_f64.cu; here a lane takes two adjacent columns,
// a warp 64, and the collision runs in packed arithmetic (f32x2: two FP32
// operations an instruction, at the scalar rate of the pipe: what it halves is the
// issue slots, which bound the four-node kernels).
#pragma once

#include "f32_core.cuh"
#include "pair_sync.cuh"

namespace dns {
namespace f32 {

constexpr int kPairPlane = kRing * 64;  // floats of one plane's live rows
constexpr int kPairPad = 4;             // before and after the ring
constexpr int kPairOwn = 62;            // columns a tile owns at most (two more complete them)

// ring of zds - 1 planes, 19 rows of the interface plane, the next row of src
inline size_t pair_smem_f32(int zds) {
  return (64 * ((size_t)(zds - 1) * kRing + 19 + zds * 19) + 2 * kPairPad) * sizeof(float);
}

using f2 = unsigned long long;
__device__ __forceinline__ f2 pack2(float a, float b) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ f2 both(float a) { return pack2(a, a); }
__device__ __forceinline__ float lo2(f2 v) {
  float a, b;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
  return a;
}
__device__ __forceinline__ float hi2(f2 v) {
  float a, b;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
  return b;
}
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f2 sub2(f2 a, f2 b) { return fma2(b, both(-1.f), a); }

// Moments of two nodes and their BGK collision in place: collide_f32_pairs's
// deviation equilibrium and update.  The relaxation rate multiplies last, as
// there: rounded products of it with the weights do not sum to it, a bias of the
// mass that 400 substeps made ten times the form's rounding error.
struct Mac2 {
  f2 drho, rho, u0;
};
__device__ __forceinline__ Mac2 collide2(f2 (&d)[19], float om, float G) {
  f2 dr = d[0];
#pragma unroll
  for (int a = 1; a < 19; a++) dr = add2(dr, d[a]);
  const f2 mx = add2(add2(sub2(d[1], d[2]), sub2(d[7], d[8])),
                     add2(sub2(d[10], d[9]), add2(sub2(d[11], d[13]), sub2(d[12], d[14]))));
  const f2 my = add2(add2(sub2(d[3], d[4]), add2(sub2(d[7], d[9]), sub2(d[8], d[10]))),
                     add2(sub2(d[15], d[17]), sub2(d[16], d[18])));
  const f2 mz = add2(add2(sub2(d[5], d[6]), add2(sub2(d[11], d[13]), sub2(d[14], d[12]))),
                     add2(sub2(d[15], d[17]), sub2(d[18], d[16])));
  Mac2 m;
  m.drho = dr;
  m.rho = add2(dr, both(1.f));
  const f2 inv = pack2(1.f / lo2(m.rho), 1.f / hi2(m.rho));
  const f2 u0 = mul2(mx, inv), u1 = mul2(my, inv), u2 = mul2(mz, inv);
  m.u0 = u0;
  const f2 usq15 = mul2(both(-1.5f), fma2(u2, u2, fma2(u1, u1, mul2(u0, u0))));
  const f2 omc = both(1.f - om), om2 = both(om);
  {
    const f2 wr = mul2(both(w_of(0)), m.rho);
    d[0] = fma2(om2, fma2(wr, usq15, mul2(both(w_of(0)), dr)), mul2(omc, d[0]));
  }
#pragma unroll
  for (int c = 1; c <= 2; c++) {
    const int a0 = c == 1 ? 1 : 7, a1 = c == 1 ? 7 : 19;
    const float w = w_of(a0);
    const f2 wr = mul2(both(w), m.rho), wd = mul2(both(w), dr), w3 = mul2(both(3.f), wr);
    const f2 force = mul2(both(bi_of(a0) * G), m.rho);
#pragma unroll
    for (int a = a0; a < a1; a++) {
      const int b = opp_of(a);
      if (b < a) continue;
      auto neg = [](f2 v) { return v ^ 0x8000000080000000ull; };
      f2 eu;
      if (c == 1) eu = a == 1 ? u0 : (a == 3 ? u1 : u2);
      else {
        const f2 p = ex_of(a) > 0 ? u0 : (ex_of(a) < 0 ? neg(u0) : u1);  // 15, 16: e_y = +1
        const f2 q = ey_of(a) && ex_of(a) ? (ey_of(a) > 0 ? u1 : neg(u1)) : (ez_of(a) > 0 ? u2 : neg(u2));
        eu = add2(p, q);
      }
      const f2 s = fma2(wr, fma2(mul2(both(4.5f), eu), eu, usq15), wd), odd = mul2(w3, eu);
      const f2 fa = ex_of(a) == 0 ? mul2(omc, d[a]) : fma2(omc, d[a], ex_of(a) > 0 ? force : neg(force));
      const f2 fb = ex_of(a) == 0 ? mul2(omc, d[b]) : fma2(omc, d[b], ex_of(a) > 0 ? neg(force) : force);
      d[a] = fma2(om2, add2(s, odd), fa);
      d[b] = fma2(om2, sub2(s, odd), fb);
    }
  }
  return m;
}
__device__ __forceinline__ void pin2(f2 (&f)[19]) {
#pragma unroll
  for (int a = 0; a < 19; a++) asm volatile("" : "+l"(f[a]));
}

// where tile i of n along a row of nx nodes starts: whole bulk copies start on
// 16 bytes, which rows of a multiple of 4 nodes allow; else pairs of nodes
__host__ __device__ __forceinline__ int pair_x0_f32(int i, int nx, int n) {
  const int u = nx % 4 == 0 ? 4 : 2;
  return u * (int)((long long)i * (nx / u) / n);
}
__host__ __device__ __forceinline__ int pair_tiles_f32(int nx) {
  return nx % 4 == 0 ? (nx / 4 + 14) / 15 : (nx / 2 + 30) / 31;
}

struct PairSync {
  unsigned long long pushed[kPairMaxZds], taken[kPairMaxZds], staged[kPairMaxZds], middle[kPairMaxZds];
  unsigned long long solid[kMaxRun + 4];
  double sums[kPairMaxZds][4];
  int stop;
};

struct PairTile {
  int nx, ny, zds, gr;        // fine block (nx even)
  int ntx, bx, y0, L;         // tiles along x, this tile, first row and rows of the run
  bool upper;
  float om, Gf;
  const float *src, *mid;     // mid: interface planes between the substeps, [2 walls][19][ny][nx]
  float *dst;
  const int8_t *wf;
  double *part, *wpart;       // this tile's flow-rate pair; wall-shear pairs of row r at wpart[r * wstride]
  size_t wstride;
  unsigned int *lost;         // set where a wait ran out
};

// One tile and run of one fine block.  MODE bits: 1 flow-rate partials, 2
// wall-shear sums.  Block-uniform; at least zds warps; ends with a barrier.
template <int MODE>
__device__ __forceinline__ void pair_tile(float *M, PairSync &S, const PairTile &P) {
  const int zds = P.zds, zdf = zds + 1, gr = P.gr, nx = P.nx, ny = P.ny, L = P.L;
  const int lane = threadIdx.x & 31, warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);  // warp-uniform
  const bool upper = P.upper;
  const int x0 = pair_x0_f32(P.bx, nx, P.ntx), cnt = pair_x0_f32(P.bx + 1, nx, P.ntx) - x0;  // column c is node x0 + c
  const int qi = upper ? 0 : zds - 1, qw = upper ? zds - 1 : 0;
  // pairs of columns in memory: n1 from node x0 on, the row's end continues at its
  // start.  Rows of a multiple of 4 nodes: bulk copies of nb pairs (16-byte
  // multiples: one pair more than the tile needs, except at the row's end), the
  // continuation by its lane; other rows: every lane its own pair.
  const int npair = (cnt + 2) / 2, n1 = min(npair, (nx - x0) / 2);
  const bool bulk = nx % 4 == 0;
  const int nb = bulk ? (x0 + cnt < nx ? npair + 1 : n1) : 0;
  const bool alone = lane >= nb && lane < npair;
  if (threadIdx.x == 0) {
    S.stop = 0;
    for (int w = 0; w < zds; w++) {
      const int n = 1 + (w > 0) + (w < zds - 1), arrivals = (bulk ? 1 : 0) + max(0, npair - nb);
      mb_init(&S.pushed[w], n);
      mb_init(&S.taken[w], n);
      mb_init(&S.staged[w], arrivals);
      mb_init(&S.middle[w], arrivals);
    }
  }
  float *const Sbase = M + 2 * kPairPad + (size_t)(zds - 1) * kPairPlane + 19 * 64;
  if (warp < zds) {
#pragma unroll
    for (int a = 0; a < 19; a++) reinterpret_cast<f2 *>(Sbase + (size_t)(warp * 19 + a) * 64)[lane] = 0;
  }
  for (int r = warp; r < L + 4; r += blockDim.x >> 5) {
    int yr = P.y0 - 2 + r;
    yr = yr < 0 ? yr + ny : (yr >= ny ? yr - ny : yr);
    unsigned long long m = 0;
#pragma unroll
    for (int s = 0; s < 2; s++) {
      int xr = x0 + min(s * 32 + lane, cnt + 1);
      xr = xr >= nx ? xr - nx : xr;
      m |= (unsigned long long)__ballot_sync(0xffffffffu, P.wf[(size_t)yr * nx + xr] == -1) << (s * 32);
    }
    if (lane == 0) S.solid[r] = m;
  }
  fence_async_proxy();
  __syncthreads();
  if (warp < zds) {
    const int q = warp;
    const bool wall = q == qw, iface = q == qi;
    const bool z0 = !iface, zup = q + 1 < zds && q + 1 != qi, zdn = q > 0 && q - 1 != qi;
    const bool inner = z0 && zup && zdn;
    const int p = (upper ? zds : 0) + q, k = upper ? q : q + 1;
    const int c0 = 2 * lane;  // the lane's columns c0, c0 + 1
    const bool own0 = c0 >= 1 && c0 <= cnt, own1 = c0 + 1 <= cnt;
    int x = x0 + min(c0, cnt);  // node of column c0 (even)
    x = x >= nx ? x - nx : x;
    const size_t plane = (size_t)ny * nx, pstride = (size_t)2 * zds * plane;
    const int pos = upper ? zds - 1 - q : q;
    float *const Mq = M + kPairPad + (size_t)pos * kPairPlane + c0;
    float *const Mup = Mq + (upper ? -kPairPlane : kPairPlane), *const Mdn = Mq - (upper ? -kPairPlane : kPairPlane);
    // the columns this lane collides in substep 2: own ones for every lane
    const float *const Mr = Mq - c0 + min(c0, cnt);
    float *const Sw = Sbase + (size_t)warp * 19 * 64;
    const bool wall_sum_plane =
        upper ? (k == zdf - 2 || k == zdf - 3 || k == zdf - 4) : (k == 1 || k == 2 || k == 3);
    const bool wall_rho_plane = upper ? (k == zdf - 4) : (k == 1);
    // encalc2 weights of the destination planes k - 1, k, k + 1 (what heads into the
    // wall stays on plane k; dropped pushes head for planes of weight 0)
    float wz[3];
#pragma unroll
    for (int c = 0; c < 3; c++) {
      const int kd = (wall && c == (upper ? 2 : 0)) ? k : k + c - 1;
      wz[c] = !upper ? ((kd >= 1 && kd < zdf - gr) ? 1.f : 0.f)
                     : ((kd >= gr && kd < zdf - 1) ? (kd == gr ? 0.5f : 1.f) : 0.f);
    }
    const bool unit = wz[0] == 1.f && wz[1] == 1.f && wz[2] == 1.f, none = wz[0] == 0.f && wz[1] == 0.f && wz[2] == 0.f;
    const unsigned rowb = (unsigned)nx * 4u, planeb = (unsigned)plane * 4u;
    const unsigned nodeb = (unsigned)p * planeb + (unsigned)x * 4u;
    const float om = P.om, Gf = P.Gf;
    double acc[2] = {0., 0.}, wacc[2] = {0., 0.};
    bool ok = true, gone = false;  // a wait of the block ran out
    f2 f[19], k0 = 0, p0 = 0;  // population 0 of rows t and t - 1
    // (every lane has collided the rows' old values; the fence puts the reads before
    // the copies, which go by another way to shared memory)
    auto copy = [&](float *row, const float *from, size_t stride, unsigned long long *b) {
      fence_async_proxy();
      __syncwarp();
      if (bulk) {
        if (lane == 0) mb_expect(b, (unsigned)(19 * nb) * 8u);
        __syncwarp();
        if (lane < 19) bulk_copy(row + lane * 64, from + (size_t)lane * stride + x0, (unsigned)nb * 8u, b);
      }
      if (alone) {
        const float *s = from + (lane < n1 ? x0 + c0 : 2 * (lane - n1));
#pragma unroll
        for (int a = 0; a < 19; a++) lane_copy(row + a * 64 + c0, s + (size_t)a * stride);
        lane_copies_arrive(b);
      }
    };
    auto stage = [&](int y) { copy(Sw, P.src + ((size_t)p * ny + y) * nx, pstride, &S.staged[warp]); };
    auto next = [&](int y) { return y == ny - 1 ? 0 : y + 1; };
    int y = P.y0 == 0 ? ny - 1 : P.y0 - 1;  // row t = 0
    int yd = y;                             // the row that substep 2 takes (t - 1)
    int t = 0, s3 = 0;                      // s3: t mod 3
    auto first_half = [&](int t1, int ahead) {
      if (t1 <= L + 1) ok = mb_wait(&S.staged[warp], t1 & 1, &S.stop) && ok;
#pragma unroll
      for (int a = 0; a < 19; a++) f[a] = reinterpret_cast<const f2 *>(Sw + a * 64)[lane];
      const Mac2 m = collide2(f, om, Gf);
      pin2(f);
      gone = !__all_sync(0xffffffffu, ok);
      if (t1 <= L && !gone) stage(ahead);
      if ((MODE & 2) && wall_sum_plane && t1 >= 1 && t1 <= L) {
        if (own0) wacc[0] += (double)lo2(m.u0);
        if (own1) wacc[0] += (double)hi2(m.u0);
        if (wall_rho_plane) {
          if (own0) wacc[1] += 1.0 + (double)lo2(m.drho);
          if (own1) wacc[1] += 1.0 + (double)hi2(m.drho);
        }
      }
    };
    stage(y);
    first_half(0, next(y));
    for (; !gone && t <= L + 1; t++) {
      const int yn = next(y);
      const int r2c = (t & 1) * 64, r2p = 64 - r2c;
      const int r3c = s3 * 64, r3n = (s3 == 2 ? 0 : s3 + 1) * 64, r3p = (s3 == 0 ? 2 : s3 - 1) * 64;
      // the pushes along x store aligned pairs, one value from the lane beside
      if (t > 0) ok = mb_wait(&S.taken[q], (t - 1) & 1, &S.stop) && ok;
      {
        auto slot = [&](int a, int row) {
          const int r = ring_depth(a) == 1 ? 0
                        : ring_depth(a) == 2 ? (row == 0 ? r2c : r2p)
                                             : (row == 0 ? r3c : (row > 0 ? r3n : r3p));
          return ring_off(a) * 64 + r;
        };
        auto to = [&](int a) { return ez_of(a) == 0 ? Mq : (ez_of(a) > 0 ? Mup : Mdn); };
        auto push = [&](int a) {
          f2 v = f[a];
          if (ex_of(a) > 0) v = pack2(__shfl_up_sync(0xffffffffu, hi2(f[a]), 1), lo2(f[a]));
          if (ex_of(a) < 0) v = pack2(hi2(f[a]), __shfl_down_sync(0xffffffffu, lo2(f[a]), 1));
          *reinterpret_cast<f2 *>(to(a) + slot(a, ey_of(a))) = v;
        };
        p0 = k0;
        k0 = f[0];
        if (inner) {
#pragma unroll
          for (int a = 1; a < 19; a++) push(a);
        } else {
#pragma unroll
          for (int c = -1; c <= 1; c++)
            if (c == 0 ? z0 : (c > 0 ? zup : zdn))
#pragma unroll
              for (int a = 1; a < 19; a++)
                if (ez_of(a) == c) push(a);
          if (wall) {
#pragma unroll
            for (int h = 0; h < 2; h++) {
              const int sb = solid_bits(S.solid, t, c0 + h);
#pragma unroll
              for (int a = 1; a < 19; a++) {
                if (ez_of(a) == 0 || (ez_of(a) > 0) != upper) continue;
                Mq[h + ((sb & 1) && (sb & dest_bit(a)) ? slot(opp_of(a), 0) : slot(mir_of(a), ey_of(a)) + ex_of(a))] =
                    h ? hi2(f[a]) : lo2(f[a]);
              }
            }
          }
        }
      }
      mb_arrive(S.pushed, lane, q, zds);
      ok = mb_wait(&S.pushed[q], t & 1, &S.stop) && ok;
      f2 h[19];
      // row t - 1, the copies' (t - 2)nd phase
      if (iface && t >= 2) ok = mb_wait(&S.middle[warp], t & 1, &S.stop) && ok;
#pragma unroll
      for (int a = 1; a < 19; a++)
        h[a] = *reinterpret_cast<const f2 *>(
            Mr + (iface ? a * 64 : ring_off(a) * 64 + (ring_depth(a) == 1 ? 0 : (ring_depth(a) == 2 ? r2p : r3p))));
      h[0] = iface ? *reinterpret_cast<const f2 *>(Mr) : p0;
      mb_arrive(S.taken, lane, q, zds);
      const Mac2 m = collide2(h, om, Gf);
      pin2(h);
      // the interface row that substep 2 takes next (row t)
      if (iface && t >= 1 && t <= L && __all_sync(0xffffffffu, ok))
        copy(Mq - c0, P.mid + ((size_t)(upper ? 19 : 0) * ny + y) * nx, plane, &S.middle[warp]);
      const bool now = t >= 2;
      const bool o0 = own0 && now, o1 = own1 && now;
      if ((MODE & 1) && unit) {
        const f2 mom = fma2(m.rho, both(Gf), mul2(m.rho, m.u0));
        if (o0) {
          acc[0] += (double)lo2(mom);
          acc[1] += (double)lo2(m.drho);
        }
        if (o1) {
          acc[0] += (double)hi2(mom);
          acc[1] += (double)hi2(m.drho);
        }
      }
      {
        const int ym = yd == 0 ? ny - 1 : yd - 1;  // rows yd - 1, yd, y
        const unsigned o = nodeb + (unsigned)yd * rowb;
        const unsigned dym = (unsigned)(ym - yd) * rowb, dyp = (unsigned)(y - yd) * rowb;
        auto offy = [&](int a) { return ey_of(a) > 0 ? dyp : (ey_of(a) < 0 ? dym : 0u); };
        auto offz = [&](int a) { return ez_of(a) > 0 ? planeb : (ez_of(a) < 0 ? 0u - planeb : 0u); };
        // Aligned pairs: e_x = +1 columns (c0, c0 + 1) from (c0 - 1, c0), lanes 1..cnt / 2;
        // e_x = -1 from (c0 + 1, c0 + 2), lanes 0..cnt / 2 - 1; e_x = 0 whole pairs in
        // between, the tile's first and last column alone.
        const bool right = now && lane >= 1 && 2 * lane <= cnt, left = now && 2 * lane + 2 <= cnt;
        const bool whole = o0 && o1;
        auto store = [&](int a) {
          float *d = at(P.dst + (size_t)a * pstride, o + offy(a) + offz(a));
          if (ex_of(a) > 0) {
            const f2 v = pack2(__shfl_up_sync(0xffffffffu, hi2(h[a]), 1), lo2(h[a]));
            if (right) *reinterpret_cast<f2 *>(d) = v;
          } else if (ex_of(a) < 0) {
            const f2 v = pack2(hi2(h[a]), __shfl_down_sync(0xffffffffu, lo2(h[a]), 1));
            if (left) *reinterpret_cast<f2 *>(d) = v;
          } else if (whole) {
            *reinterpret_cast<f2 *>(d) = h[a];
          } else {
            if (o0) d[0] = lo2(h[a]);
            if (o1) d[1] = hi2(h[a]);
          }
        };
        if (inner) {
#pragma unroll
          for (int a = 0; a < 19; a++) store(a);
        } else {
#pragma unroll
          for (int c = -1; c <= 1; c++)
            if (c == 0 ? z0 : (c > 0 ? zup : zdn))
#pragma unroll
              for (int a = 0; a < 19; a++)
                if (ez_of(a) == c) store(a);
          if (wall) {
#pragma unroll
            for (int hh = 0; hh < 2; hh++) {
              const int sb = solid_bits(S.solid, t - 1, c0 + hh), xh = x + hh;
              const unsigned oh = o + 4u * hh;
              const unsigned dxm = (unsigned)(xh == 0 ? nx - 1 : -1) * 4u, dxp = (unsigned)(xh == nx - 1 ? 1 - nx : 1) * 4u;
#pragma unroll
              for (int a = 0; a < 19; a++) {
                if (ez_of(a) == 0 || (ez_of(a) > 0) != upper) continue;
                const float v = hh ? hi2(h[a]) : lo2(h[a]);
                const bool bounce = (sb & 1) && (sb & dest_bit(a));
                const unsigned off = bounce ? oh : oh + offy(a) + (ex_of(a) > 0 ? dxp : (ex_of(a) < 0 ? dxm : 0u));
                if (hh ? o1 : o0) {
                  *at(bounce ? P.dst + (size_t)opp_of(a) * pstride : P.dst + (size_t)mir_of(a) * pstride, off) = v;
                  // a bounce reverses its momentum
                  if ((MODE & 1) && ex_of(a) != 0 && bounce) acc[0] -= (double)(2.f * ex_of(a) * wz[1] * v);
                }
              }
            }
          }
        }
        if ((MODE & 1) && !unit && !none) {
          // mass and momentum by destination plane
          const f2 m0 = add2(add2(add2(add2(h[0], h[1]), add2(h[2], h[3])), add2(add2(h[4], h[7]), add2(h[8], h[9]))), h[10]);
          const f2 mp = add2(add2(add2(h[5], h[11]), add2(h[14], h[15])), h[18]);
          const f2 mm = add2(add2(add2(h[6], h[12]), add2(h[13], h[16])), h[17]);
          const f2 px = add2(add2(sub2(h[1], h[2]), sub2(h[7], h[8])), sub2(h[10], h[9]));
          const f2 den = fma2(both(wz[0]), mm, fma2(both(wz[1]), m0, mul2(both(wz[2]), mp)));
          const f2 mom = fma2(both(wz[0]), sub2(h[12], h[13]), fma2(both(wz[1]), px, mul2(both(wz[2]), sub2(h[11], h[14]))));
          if (o0) {
            acc[0] += (double)lo2(mom);
            acc[1] += (double)lo2(den);
          }
          if (o1) {
            acc[0] += (double)hi2(mom);
            acc[1] += (double)hi2(den);
          }
        }
      }
      first_half(t + 1, next(yn));
      yd = y;
      y = yn;
      s3 = s3 == 2 ? 0 : s3 + 1;
    }
    if (gone) {
      S.stop = 1;
      *P.lost = 1u;
      drain(&S.staged[warp], min(t, L + 1));
      if (iface) drain(&S.middle[warp], min(t - 1, L) - 1);
    }
    if (MODE) {
      double v[4] = {acc[0], acc[1], wacc[0], wacc[1]};
#pragma unroll
      for (int c = 0; c < 4; c++) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[c] += __shfl_down_sync(0xffffffffu, v[c], o);
        if (lane == 0) S.sums[warp][c] = v[c];
      }
    }
  }
  __syncthreads();
  if ((MODE & 1) && threadIdx.x < 2) {
    double s = 0.;
    for (int w = 0; w < zds; w++) s += S.sums[w][threadIdx.x];
    P.part[threadIdx.x] = s;
  }
  // wall-shear rows: lower k = 1, 2, 3, upper k = zdf - 2, -3, -4
  if ((MODE & 2) && threadIdx.x >= 32 && threadIdx.x < 38) {
    const int r = ((int)threadIdx.x - 32) >> 1, c = threadIdx.x & 1;
    P.wpart[(size_t)(upper ? 3 + r : r) * P.wstride + c] = S.sums[upper ? zds - 1 - r : r][2 + c];
  }
  if (threadIdx.x == 0)
    for (int w = 0; w < zds; w++) {
      mb_inval(&S.pushed[w]);
      mb_inval(&S.taken[w]);
      mb_inval(&S.staged[w]);
      mb_inval(&S.middle[w]);
    }
  __syncthreads();
}

}  // namespace f32
}  // namespace dns
