// split_epilogue.cuh -- the end of a GEMM tile whose reduction the CTAs of a cluster share, and the staging of
// per-channel requantisation parameters; for blocks of 256 threads.
#pragma once

#include "internal.cuh"
#include "sm100_primitives.cuh"

namespace pulpnn {

// k and lambda' of channels n0 .. n0+ncols-1 (32-bit values in the 32-bit modes). The bias is folded into lambda:
// k*(acc+b)+lambda == k*acc + (k*b+lambda) in wrap-around arithmetic.
template <int MODE>
__device__ __forceinline__ void stage_channel_params(const Epilogue &e, int n0, int ncols, long long *par_k, long long *par_l,
                                                     int first, int step)
{
  for (int i = first; i < ncols; i += step) {
    const int n = n0 + i;
    if (MODE == EPI_BN32) {
      const int k = __ldg(reinterpret_cast<const int *>(e.k) + n), l = __ldg(reinterpret_cast<const int *>(e.lambda) + n);
      const int b = e.bias ? (int)__ldg(reinterpret_cast<const int8_t *>(e.bias) + n) : 0;
      reinterpret_cast<int *>(par_k)[i] = k;
      reinterpret_cast<int *>(par_l)[i] = (int)((unsigned)k * (unsigned)b + (unsigned)l);
    } else if (MODE == EPI_BN64) {
      const long long k = __ldg(reinterpret_cast<const long long *>(e.k) + n), l = __ldg(reinterpret_cast<const long long *>(e.lambda) + n);
      const long long b = e.bias ? (long long)__ldg(reinterpret_cast<const int8_t *>(e.bias) + n) : 0;
      par_k[i] = k;
      par_l[i] = (long long)((unsigned long long)k * (unsigned long long)b + (unsigned long long)l);
    } else if (MODE == EPI_RAW32) {
      reinterpret_cast<int *>(par_l)[i] = e.bias ? __ldg(reinterpret_cast<const int *>(e.bias) + n) : 0;
    } else {
      reinterpret_cast<int *>(par_l)[i] = e.bias ? (int)__ldg(reinterpret_cast<const int8_t *>(e.bias) + n) : 0;
    }
  }
}

// 32 accumulator columns c0.. of the calling lane's row -> 32 bytes, parameters staged by stage_channel_params (whole
// warps: 64-bit parameters are looked at together). Columns past ncols give bytes nobody may store.
template <int MODE>
__device__ __forceinline__ void requant32_cols(const uint32_t (&v)[32], int c0, int ncols, const long long *par_k, const long long *par_l,
                                               const Epilogue &e, int K, unsigned (&w)[8])
{
  const int lane = threadIdx.x & 31;
  const bool fits = MODE == EPI_BN64 &&
      __all_sync(0xffffffffu, c0 + lane >= ncols || bn_fits_32(par_k[c0 + lane], par_l[c0 + lane], acc_bound(K), e.shift));
#pragma unroll
  for (int j = 0; j < 32; j += 4) {
    int t[4];
    // columns past the last channel read stale parameters; their bytes are never stored
    if (MODE == EPI_BN32) {
      const int4 kk = *reinterpret_cast<const int4 *>(reinterpret_cast<const int *>(par_k) + c0 + j);
      const int4 ll = *reinterpret_cast<const int4 *>(reinterpret_cast<const int *>(par_l) + c0 + j);
      t[0] = (int)((unsigned)kk.x * v[j] + (unsigned)ll.x) >> e.shift;
      t[1] = (int)((unsigned)kk.y * v[j + 1] + (unsigned)ll.y) >> e.shift;
      t[2] = (int)((unsigned)kk.z * v[j + 2] + (unsigned)ll.z) >> e.shift;
      t[3] = (int)((unsigned)kk.w * v[j + 3] + (unsigned)ll.w) >> e.shift;
    } else if (MODE == EPI_BN64) {
      requant4_bn64(par_k + c0 + j, par_l + c0 + j, v[j], v[j + 1], v[j + 2], v[j + 3], e.shift, fits, t);
    } else {
      const int4 bb = *reinterpret_cast<const int4 *>(reinterpret_cast<const int *>(par_l) + c0 + j);
      const int a4[4] = {(int)v[j] + bb.x, (int)v[j + 1] + bb.y, (int)v[j + 2] + bb.z, (int)v[j + 3] + bb.w};
#pragma unroll
      for (int u = 0; u < 4; u++)
        t[u] = MODE == EPI_MULT ? (int)(short)((int)((unsigned)e.out_mult * (unsigned)a4[u]) >> e.shift) : a4[u] >> e.shift;
    }
    w[j >> 2] = pack4_sat_u8(t[0], t[1], t[2], t[3]);
  }
}

template <int MODE>
__device__ __forceinline__ int requant_param(int a, int col, const long long *par_k, const long long *par_l, const Epilogue &e)
{
  const int *k32 = reinterpret_cast<const int *>(par_k), *l32 = reinterpret_cast<const int *>(par_l);
  if (MODE == EPI_BN32) return (int)((unsigned)k32[col] * (unsigned)a + (unsigned)l32[col]) >> e.shift;
  if (MODE == EPI_BN64)
    return (int)((long long)((unsigned long long)par_k[col] * (unsigned long long)(long long)a + (unsigned long long)par_l[col]) >> e.shift);
  if (MODE == EPI_MULT) return (int)(short)((int)((unsigned)e.out_mult * (unsigned)(a + l32[col])) >> e.shift);
  return (a + l32[col]) >> e.shift;
}

// The CTAs of a cluster hold partial sums of the same 128-row tile: each puts its own into its shared memory
// (`ring`, 128 rows of bn + 4 words), takes an equal share of the rows, adds the others' through the cluster and
// finishes them. The sums are integers, so their order does not matter. row_of(r) is the row of the output (of N
// channels) that row r of the tile is, or -1. A cluster of one CTA works as well.
template <int MODE, typename RowOf>
__device__ __forceinline__ void split_epilogue(const Epilogue &e, void *out_base, int N, int bn, int k_split, int ks, int n0,
                                               int ncols, uint8_t *ring, uint32_t tmem, const long long *par_k,
                                               const long long *par_l, bool dead, RowOf row_of)
{
  using namespace sm100;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int pitch = bn + 4;                        // words; rows 16-byte aligned, an odd number of 16-byte pieces
  const int quad = warp & 3, r = quad * 32 + lane;
  if (!dead) {
    for (int c0 = (warp >> 2) * 32; c0 < ncols; c0 += 64) {
      uint32_t v[32];
      tmem_ld_32(tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)c0, v);
      tmem_wait_ld();
      const uint32_t row = smem_u32(ring) + (uint32_t)((r * pitch + c0) * 4);
#pragma unroll
      for (int j = 0; j < 32; j += 4)
        if (c0 + j < bn) sts128(row + 4 * j, v[j], v[j + 1], v[j + 2], v[j + 3]);
    }
  }
  tc_fence_before();
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  tc_fence_after();
  const int share = 128 / k_split, r0 = ks * share;
  const int per = (ncols + 3) >> 2;
  if (!dead) {
    for (int i = tid; i < share * per; i += 256) {
      const int rr = i / per, c = (i - rr * per) * 4;
      const long long row = row_of(r0 + rr);
      if (row < 0) continue;
      const uint32_t mine = smem_u32(ring) + (uint32_t)(((r0 + rr) * pitch + c) * 4);
      int s0 = 0, s1 = 0, s2 = 0, s3 = 0;
      for (int k0 = 0; k0 < k_split; k0 += 4) {
        uint32_t x[4][4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
          x[k][0] = x[k][1] = x[k][2] = x[k][3] = 0;
          if (k0 + k < k_split) {
            uint32_t a;
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(mine), "r"(k0 + k));
            asm volatile("ld.shared::cluster.v4.b32 {%0, %1, %2, %3}, [%4];"
                         : "=r"(x[k][0]), "=r"(x[k][1]), "=r"(x[k][2]), "=r"(x[k][3]) : "r"(a) : "memory");
          }
        }
#pragma unroll
        for (int k = 0; k < 4; k++) { s0 += (int)x[k][0]; s1 += (int)x[k][1]; s2 += (int)x[k][2]; s3 += (int)x[k][3]; }
      }
      const size_t o = (size_t)row * N + n0 + c;
      const int sum[4] = {s0, s1, s2, s3};
      if (MODE == EPI_RAW32) {
        int *out = reinterpret_cast<int *>(out_base) + o;
#pragma unroll
        for (int j = 0; j < 4; j++)
          if (c + j < ncols) out[j] = sum[j] + reinterpret_cast<const int *>(par_l)[c + j];
      } else {
        uint8_t *out = static_cast<uint8_t *>(out_base) + o;
        int t[4];
#pragma unroll
        for (int j = 0; j < 4; j++) t[j] = requant_param<MODE>(sum[j], c + j, par_k, par_l, e);
        const unsigned w = pack4_sat_u8(t[0], t[1], t[2], t[3]);
        if (c + 4 <= ncols && (reinterpret_cast<uintptr_t>(out) & 3) == 0) *reinterpret_cast<unsigned *>(out) = w;
        else {
#pragma unroll
          for (int j = 0; j < 4; j++)
            if (c + j < ncols) out[j] = (uint8_t)(w >> (8 * j));
        }
      }
    }
  }
  // nobody's sums are overwritten, and no CTA leaves, before all have read them
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

}  // namespace pulpnn
