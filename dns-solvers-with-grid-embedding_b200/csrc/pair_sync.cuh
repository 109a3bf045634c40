// What the kernels that take two fine substeps in one pass share (pair_f64.cu,
// pair_f32.cuh): the live rows of each population, and the barriers.
#pragma once

#include "lattice.cuh"

namespace dns {

// Rows of population a that are live at a time: pushes with e_y = -1 complete the
// row that is taken next (1 row; 2 for populations 17 and 18, which half-way
// bounce-back also writes one row early), e_y = 0 two rows, e_y = +1 three;
// population 0 stays in its lane's registers.
__host__ __device__ constexpr int ring_depth(int a) {
  return a == 0 ? 0 : ey_of(a) < 0 ? ((a == 17 || a == 18) ? 2 : 1) : (ey_of(a) == 0 ? 2 : 3);
}
// where they start
__host__ __device__ constexpr int ring_off(int a) {
  int o = 0;
  for (int b = 0; b < a; b++) o += ring_depth(b);
  return o;
}
constexpr int kRing = ring_off(19);
static_assert(kRing == 38, "live rows per plane");
constexpr int kMaxRun = 256;  // rows of a run (the wall flags of a run are kept as one mask a row)

// Split barriers, one a plane: its warps and those of the planes beside it arrive
// (only they push into its rows, and only it reads them), its warps wait for the
// phase.  The waits are bounded: kTries attempts, 1.5 us each where the phase does not
// complete, so about 0.1 s, which only a fault of these files could take (every warp
// makes the same arrivals).
__device__ __forceinline__ void mb_init(unsigned long long *b, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"((unsigned)__cvta_generic_to_shared(b)), "r"(count)
               : "memory");
}
__device__ __forceinline__ void mb_inval(unsigned long long *b) {
  asm volatile("mbarrier.inval.shared::cta.b64 [%0];\n" ::"r"((unsigned)__cvta_generic_to_shared(b)) : "memory");
}
// arrive at the barriers of planes q - 1, q, q + 1
__device__ __forceinline__ void mb_arrive(unsigned long long *b, int lane, int q, int zds) {
  __syncwarp();
  const int n = q - 1 + lane;
  if (lane < 3 && n >= 0 && n < zds)
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"((unsigned)__cvta_generic_to_shared(b + n))
                 : "memory");
}
// False for a lane whose wait ran out or found the block's stop set: its warp goes on to
// the middle of its row and leaves there.  (A vote and a branch at every wait cost 10% of
// the two-substep pass, one a row 1.4%.)
constexpr int kTries = 1 << 16;
__device__ __forceinline__ bool mb_wait(unsigned long long *b, int parity, volatile int *stop, int tries = kTries) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(b);
  for (int n = 0; n < tries; n++) {
    unsigned ok;
    asm volatile(
        "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(a), "r"(parity)
        : "memory");
    if (ok) return true;
    if (*stop) break;
  }
  return false;
}

// Bulk copies into a warp's rows: the warp's barrier completes when `bytes` have landed.
__device__ __forceinline__ void mb_expect(unsigned long long *b, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"((unsigned)__cvta_generic_to_shared(b)),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void bulk_copy(void *smem, const void *gmem, unsigned bytes, unsigned long long *b) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
                   (unsigned)__cvta_generic_to_shared(smem)),
               "l"(gmem), "r"(bytes), "r"((unsigned)__cvta_generic_to_shared(b))
               : "memory");
}

// 8 bytes by the calling lane, its arrival at the barrier once they have landed
__device__ __forceinline__ void lane_copy(void *smem, const void *gmem) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(gmem)
               : "memory");
}
__device__ __forceinline__ void lane_copies_arrive(unsigned long long *b) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];\n" ::"r"((unsigned)__cvta_generic_to_shared(b))
               : "memory");
}
__device__ __forceinline__ void fence_async_proxy() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }

// A warp that leaves sets stop, takes no further row and issues no further copy.  The
// launch is reported in *lost: the step's log row and every later one carry a NaN wall
// stress, and dns_step returns an error.  The warp's own copies land before it goes:
// phases up to `copies` of its barrier b (the last one may not have been issued).
__device__ __forceinline__ void drain(unsigned long long *b, int copies) {
  int none = 0;
  for (int c = max(copies - 1, 0); c <= copies; c++) mb_wait(b, c & 1, &none, 4096);
  asm volatile("cp.async.wait_all;\n" ::: "memory");
}

// a thread-uniform base plus a 32-bit byte offset (population arrays are below 4 GB)
template <class T>
__device__ __forceinline__ T *at(T *base, unsigned off) {
  return reinterpret_cast<T *>(reinterpret_cast<char *>(base) + off);
}

// bits of the wall flags around a column: 0 own, 1 x + 1, 2 x - 1, 3 y + 1, 4 y - 1
// (set: solid); the bit of the column population a heads for
__host__ __device__ constexpr int dest_bit(int a) {
  return ex_of(a) > 0 ? 2 : (ex_of(a) < 0 ? 4 : (ey_of(a) > 0 ? 8 : (ey_of(a) < 0 ? 16 : 1)));
}
// solid: one mask of the tile's columns a row, row t at solid[t + 1]
__device__ __forceinline__ int solid_bits(const unsigned long long *solid, int t, int col) {
  const unsigned long long m = solid[t + 1];
  return (int)((m >> col) & 1) | (int)(((m >> 1) >> col) & 1) << 1 | (int)(((m << 1) >> col) & 1) << 2 |
         (int)((solid[t + 2] >> col) & 1) << 3 | (int)((solid[t] >> col) & 1) << 4;
}

}  // namespace dns
