// conv_gather_tc.cu -- convolution, pointwise and fully connected layers on the sm_100a tensor cores
// for the shapes whose rows no TMA box can describe: channel counts that are not a multiple of 16 (or
// 32 for a spatial kernel), operands that are not 16-byte aligned. Arithmetic as in igemm_tc.cu
// (32bit/src/pulp_nn_conv_Ho_parallel.c:80-249, pulp_nn_matmul.c:27-298).
//
// In HWC memory the kx * ch_in bytes that one output pixel reads from one filter row are CONTIGUOUS. So
// the im2col row of a pixel is ky runs of L = kx*ch_in bytes at arbitrary byte addresses, and a weight
// row is ky runs of the same length. Both are laid out in shared memory with every run padded to
// Lp = 16*ceil(L/16) bytes, K' = ky*Lp: a 16-byte chunk then belongs to one run and costs two aligned
// 16-byte loads and a byte shift (one load when everything is a multiple of 16). The padding bytes of W
// are zero, so whatever the padding bytes of A hold contributes nothing; pixels outside the image are
// masked to zero, the zero padding of the reference.
//
// One CTA (8 warps, all of them gather, one thread issues the MMAs) computes 128 output pixels x BN
// channels: per 128-byte slab of K' the warps fill a stage of the ring (128-byte swizzle, K-major) and
// go on to the next while tcgen05.mma works on it; the accumulator is requantised from tensor memory
// into a staging tile and leaves as the contiguous run of bytes that 128 consecutive pixels are. Two
// CTAs share an SM, so one gathers while the other drains. W stays in shared memory when it fits beside
// the ring (read once per CTA), otherwise its slab is gathered with every slab of A. A problem with few
// tiles and a long reduction is shared by the CTAs of a cluster, which add their sums through
// distributed shared memory.
//
// What bounds it: instruction issue of the gather (64x56x56x48 -> 48: 45 % of the issue slots, 33 % of the
// shared-memory cycles, tensor pipe 6 %), so divisions are multiplications, offsets 32 bits and the edge
// cases out of line: 31.7 -> 26.5 us there. The dp4a kernel it replaces takes 64 x 64 x 32 per 128
// cycles at best. Measured against it (us, graph replay): 48x48x20 -> 40 at batch 32 12.3 / 33.6, 56x56x181 ->
// 250 at batch 8 55 / 719, 14x14x999 -> 1000 pointwise at batch 8 19 / 145, linear 4090 -> 1000 at batch
// 100 13.3 / 362 (79 before the reduction was shared in a cluster), 7x7x16 -> 16 3.8 / 7.3.
#include "internal.cuh"
#include "sm100_primitives.cuh"
#include "split_epilogue.cuh"
#include "unaligned16.cuh"

namespace pulpnn {

namespace {

using namespace sm100;

constexpr int GT = 256;                  // threads
constexpr int GBM = 128;                 // output pixels per tile
constexpr int A_STAGE = GBM * 128;       // bytes of A per slab
constexpr int MAX_G_STAGES = 4;
constexpr int ST_G_EMPTY = 0x1000, ST_G_FULL = 0x2000;

struct GatherParams {
  ConvProblem p;
  FastDiv by_pixels, by_wo, by_chunks, by_cols;   // Ho*Wo, Wo, run_chunks; 16-byte pieces of a tile's row
  FastDiv by_bn, by_last;                         // columns of a tile, of the last one
  int M, K;                // M = B*Ho*Wo output pixels, K = ky*kx*Cin bytes per weight row
  int run, run_chunks;     // L and Lp/16
  int chunks, slabs;       // chunks of K' in all, 128-byte slabs
  int m_tiles, n_tiles, bn;
  int k_split, slabs_per;  // CTAs of a cluster that share a tile's reduction, slabs of each
  int stages, tmem_cols;
  int out_vec;             // store width in bytes: 16, 4 or 1
  int *status;
};

// ALIGNED: ch_in a multiple of 16 and 16-byte aligned operands, so that every chunk is one aligned load of one pixel
// W_RES: the CTA's rows of W stay in shared memory
template <int MODE, bool ALIGNED, bool W_RES>
__global__ void __launch_bounds__(GT, 2) conv_gather_tc_kernel(const __grid_constant__ GatherParams g)
{
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  __shared__ uint64_t empty_bar[MAX_G_STAGES], full_bar;
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_word;
  __shared__ __align__(16) long long par_k[256];     // k and lambda' of the CTA's channels (int in the 32-bit modes)
  __shared__ __align__(16) long long par_l[256];
  volatile int *abort_flag = &abort_word;

  const ConvProblem &p = g.p;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int bn = g.bn;
  const int w_slab = bn * 128;
  const int stage_bytes = W_RES ? A_STAGE : A_STAGE + w_slab;
  uint8_t *ring = smem + (W_RES ? g.slabs_per * w_slab : 0);
  uint8_t *staging = ring;                           // the output tile, once the MMAs have read the ring

  // CTAs k_split*i .. k_split*i + k_split-1 (a cluster) share a tile, each with its own slabs
  const int ks = g.k_split == 1 ? 0 : (int)(blockIdx.x % (unsigned)g.k_split);
  const unsigned cta = g.k_split == 1 ? blockIdx.x : blockIdx.x / (unsigned)g.k_split;
  const int nt = (int)(cta % (unsigned)g.n_tiles);
  const int m_first = (int)(cta / (unsigned)g.n_tiles), m_step = (int)(gridDim.x / (unsigned)(g.n_tiles * g.k_split));
  const int slab0 = ks * g.slabs_per, slab1 = min(slab0 + g.slabs_per, g.slabs);
  const int n0 = nt * bn, ncols = min(bn, p.Cout - n0);

  if (tid == 0) {
    for (int s = 0; s < g.stages; s++) mbar_init(&empty_bar[s], 1);
    mbar_init(&full_bar, 1);
    abort_word = 0;
    mbar_fence_init();
  }
  if (warp == 1) tmem_alloc(&tmem_slot, (uint32_t)g.tmem_cols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  pdl_wait();
  pdl_launch_dependents();

  stage_channel_params<MODE>(p.epi, n0, ncols, par_k, par_l, tid, GT);
  const Epilogue &e = p.epi;

  const int ck = tid & 7, row0 = tid >> 3;           // this thread's chunk of a slab, its first row
  const Bytes wt(p.w, p.Cout * g.K), at(p.in, p.B * p.H * p.W * p.Cin);
  const int w_first = wt.start + n0 * g.K;

  // Chunk ck of rows r[0..3] of slab s[0..3] of W: zero past the end of a run, past the last channel
  auto w_off = [&](int s, int &left) {
    const int q = s * 8 + ck;
    const int fy = g.by_chunks.div(q), j = q - fy * g.run_chunks;
    left = q < g.chunks ? g.run - 16 * j : 0;        // bytes of the run from this chunk on
    return w_first + fy * g.run + 16 * j;
  };
  auto w_store = [&](uint8_t *dst, int r, uint4 v) {
    sts128(smem_u32(dst) + (uint32_t)(r * 128 + ((ck ^ (r & 7)) << 4)), v.x, v.y, v.z, v.w);
  };
  auto w_get = [&](const Chunk &t, int left) {
    uint4 v = make_uint4(0, 0, 0, 0);
    if (left > 0) {
      if (ALIGNED) v = t.a;
      else {
        v = t.get(wt);
        if (left < 16) mask16(v, 0, left);
      }
    }
    return v;
  };
  auto fetch = [&](Chunk &t, const Bytes &b, int off, bool need) {
    if (ALIGNED) t.a = ldg16_if(b.base + off, need);
    else         t.fetch(b, off, need);
  };

  if (W_RES) {
    // rows of all slabs as one list, four chunks of a thread in flight
    const int total = (slab1 - slab0) * bn;
    for (int f = row0; f < total; f += 4 * (GT / 8)) {
      Chunk t[4];
      int left[4];
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const int x = f + i * (GT / 8);
        const int s = x / bn, r = x - s * bn;
        const int off = w_off(slab0 + s, left[i]) + r * g.K;
        if (r >= ncols || x >= total) left[i] = 0;
        fetch(t[i], wt, off, left[i] > 0);
      }
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const int x = f + i * (GT / 8);
        const int s = x / bn, r = x - s * bn;
        if (x < total) w_store(smem + s * w_slab, r, w_get(t[i], left[i]));
      }
    }
  }

  const uint32_t idesc = umma_idesc_u8s8(bn);
  bool dead = false;
  int st = 0;                                        // stage of the current slab
  uint32_t lap = 0;                                  // times round the ring
  uint32_t tile_parity = 0;
  // this thread's four pixels of the tile being gathered: offset of the window's first byte, first window
  // row, and the bytes [from, to) of a window row that lie inside the image
  int src[4], iy0[4], from[4], to[4];
  auto set_tile = [&](int mt) {
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const int m = mt * GBM + row0 + 32 * i;
      const int mm = m < g.M ? m : 0;
      const int b = g.by_pixels.div(mm), r = mm - b * (p.Ho * p.Wo);
      const int oy = g.by_wo.div(r), ox = r - oy * p.Wo;
      const int iy = oy * p.sy - p.pt, ix = ox * p.sx - p.pl;
      iy0[i] = m < g.M ? iy : -(1 << 30);            // a row past the last pixel reads as padding
      from[i] = min(max(-ix, 0), p.kx) * p.Cin;
      to[i] = p.W - ix < p.kx ? max(p.W - ix, 0) * p.Cin : 1 << 29;
      src[i] = at.start + ((b * p.H + iy) * p.W + ix) * p.Cin;
    }
  };
  Chunk t[4];
  unsigned inside = 0;                               // bit i: chunk i is not padding as a whole
  int j = 0;                                         // its position in the run
  auto fetch_a = [&](int s) {
    const int q = s * 8 + ck;
    const int fy = g.by_chunks.div(q);
    j = q - fy * g.run_chunks;
    const int off = fy * p.W * p.Cin + 16 * j;
    inside = 0;
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const bool in = q < g.chunks && (unsigned)(iy0[i] + fy) < (unsigned)p.H && from[i] < 16 * j + 16 && to[i] > 16 * j;
      if (in) inside |= 1u << i;
      fetch(t[i], at, src[i] + off, in);
    }
  };
  if (ALIGNED && m_first < g.m_tiles) { set_tile(m_first); fetch_a(slab0); }
  for (int mt = m_first; mt < g.m_tiles; mt += m_step) {
    if (!ALIGNED) set_tile(mt);
    for (int s = slab0; s < slab1; s++) {
      if (!ALIGNED) fetch_a(s);
      Chunk tw[4];
      int left = 0, woff = 0;
      if (!W_RES) {
        woff = w_off(s, left);
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const int r = row0 + 32 * i;
          fetch(tw[i], wt, woff + r * g.K, r < ncols && left > 0);
        }
      }
      if (lap > 0 && !dead && !mbar_wait(&empty_bar[st], (lap - 1) & 1u, abort_flag, g.status, ST_G_EMPTY)) dead = true;
      uint8_t *a_dst = ring + st * stage_bytes;
#pragma unroll
      for (int i = 0; i < 4; i++) {
        uint4 v = make_uint4(0, 0, 0, 0);
        if (ALIGNED) v = t[i].a;                     // a chunk of one pixel is inside or outside as a whole
        else if (inside & (1u << i)) {
          v = t[i].get(at);
          if (from[i] > 16 * j || to[i] < 16 * j + 16) mask16(v, from[i] - 16 * j, to[i] - 16 * j);
        }
        const int r = row0 + 32 * i;
        sts128(smem_u32(a_dst) + (uint32_t)(r * 128 + ((ck ^ (r & 7)) << 4)), v.x, v.y, v.z, v.w);
      }
      if (!W_RES) {
        for (int r0 = row0;;) {
#pragma unroll
          for (int i = 0; i < 4; i++) {
            const int r = r0 + 32 * i;
            if (r < bn) w_store(a_dst + A_STAGE, r, w_get(tw[i], r < ncols ? left : 0));
          }
          r0 += 4 * 32;
          if (r0 >= bn) break;
#pragma unroll
          for (int i = 0; i < 4; i++) {
            const int r = r0 + 32 * i;
            fetch(tw[i], wt, woff + r * g.K, r < ncols && left > 0);
          }
        }
      }
      // the next slab's (or tile's) loads are on their way while this one is multiplied and drained
      // (unaligned chunks hold twice the registers: they would spill)
      if (ALIGNED) {
        if (s + 1 < slab1) fetch_a(s + 1);
        else if (mt + m_step < g.m_tiles) { set_tile(mt + m_step); fetch_a(slab0); }
      }
      fence_proxy_async();
      __syncthreads();
      if (tid == 0 && !dead) {
        tc_fence_after();
        const uint32_t a_addr = smem_u32(a_dst);
        const uint32_t b_addr = W_RES ? smem_u32(smem + (s - slab0) * w_slab) : a_addr + A_STAGE;
        const uint64_t da = umma_smem_desc<128>(a_addr), db = umma_smem_desc<128>(b_addr);
        const int n_mma = (min(g.chunks - s * 8, 8) + 1) >> 1;   // 32 bytes of K' each
        for (int j2 = 0; j2 < n_mma; j2++)
          umma_i8(tmem, da + (uint64_t)(2 * j2), db + (uint64_t)(2 * j2), idesc, (s > slab0 || j2 > 0) ? 1u : 0u);
        umma_commit(&empty_bar[st]);
        if (s == slab1 - 1) umma_commit(&full_bar);
      }
      if (++st == g.stages) { st = 0; lap++; }
    }
    if (!dead && !mbar_wait(&full_bar, tile_parity, abort_flag, g.status, ST_G_FULL)) dead = true;
    tile_parity ^= 1;
    dead = __syncthreads_or(dead);                   // tensor-memory loads need whole warps
    tc_fence_after();

    if (g.k_split > 1) {
      const int m0 = mt * GBM;
      split_epilogue<MODE>(p.epi, p.out, p.Cout, bn, g.k_split, ks, n0, ncols, ring, tmem, par_k, par_l, dead,
                           [&](int r) { return m0 + r < g.M ? (long long)(m0 + r) : -1ll; });
      continue;
    }

    // ---- epilogue: warp w drains rows 32*(w%4).. and every other 32-column chunk -----------------
    const int quad = warp & 3;
    const int r = quad * 32 + lane;
    const int pitch = g.out_vec == 16 ? ((bn >> 4) | 1) << 4 : bn + 4;   // odd number of 16-byte pieces / words: no bank conflicts
    // ragged rows of the only channel tile: staged as the one run of bytes that they are in memory
    const bool linear = MODE != EPI_RAW32 && g.n_tiles == 1 && g.out_vec != 1 && p.Cout % 16 != 0;
    const uint32_t t_row = tmem + ((uint32_t)(quad * 32) << 16);
    if (!dead) {
      for (int c0 = (warp >> 2) * 32; c0 < ncols; c0 += 64) {
        uint32_t v[32];
        tmem_ld_32(t_row + (uint32_t)c0, v);
        tmem_wait_ld();
        if (MODE == EPI_RAW32) {
          // 32 x 32 words through shared memory, so that a warp stores runs of a row
          int *tile = reinterpret_cast<int *>(staging) + warp * (32 * 33);
          const int *pb = reinterpret_cast<const int *>(par_l);
          __syncwarp();
#pragma unroll
          for (int j = 0; j < 32; j++) tile[lane * 33 + j] = (int)v[j] + ((c0 + j) < ncols ? pb[c0 + j] : 0);
          __syncwarp();
          const int col = c0 + lane;
          int *o = reinterpret_cast<int *>(p.out) + (size_t)n0 + col;
          const int mb = mt * GBM + quad * 32;
          for (int rr = 0; rr < 32; rr++)
            if (mb + rr < g.M && col < ncols) o[(size_t)(mb + rr) * p.Cout] = tile[rr * 33 + lane];
        } else {
          unsigned w[8];
          const bool fits = MODE == EPI_BN64 &&
              __all_sync(0xffffffffu, c0 + lane >= ncols || bn_fits_32(par_k[c0 + lane], par_l[c0 + lane], acc_bound(g.K), e.shift));
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
          if (linear) {
            // bytes [from, from + len) of the tile's run: whole words shifted into place, the ends byte by byte
            const int from_b = r * ncols + c0, len = min(32, ncols - c0);
            const int head = -from_b & 3, n_words = len > head ? (len - head) >> 2 : 0;
            const uint32_t at_s = smem_u32(staging) + (uint32_t)from_b;
            unsigned last = 0;
#pragma unroll
            for (int j = 0; j < 9; j++) {
              const unsigned x = __funnelshift_r(j < 8 ? w[j < 8 ? j : 7] : 0u, j < 7 ? w[j < 7 ? j + 1 : 7] : 0u, 8 * head);
              if (j < n_words) asm volatile("st.shared.b32 [%0], %1;" ::"r"(at_s + head + 4 * j), "r"(x) : "memory");
              if (j == n_words) last = x;
            }
            const int tail = len > head ? (len - head) & 3 : 0;
#pragma unroll
            for (int b = 0; b < 3; b++) {
              if (b < min(head, len)) asm volatile("st.shared.b8 [%0], %1;" ::"r"(at_s + b), "r"(w[0] >> (8 * b)) : "memory");
              if (b < tail) asm volatile("st.shared.b8 [%0], %1;" ::"r"(at_s + len - tail + b), "r"(last >> (8 * b)) : "memory");
            }
            continue;
          }
          uint8_t *row = staging + r * pitch + c0;
          // bn is a multiple of 16: a chunk is 16 or 32 columns of the tile
          if (g.out_vec == 16) {
            sts128(smem_u32(row), w[0], w[1], w[2], w[3]);
            if (c0 + 16 < bn) sts128(smem_u32(row) + 16, w[4], w[5], w[6], w[7]);
          } else {
#pragma unroll
            for (int j = 0; j < 8; j++)
              if (c0 + 4 * j < bn) reinterpret_cast<unsigned *>(row)[j] = w[j];
          }
        }
      }
    }
    tc_fence_before();
    if (MODE != EPI_RAW32) {
      __syncthreads();
      const int rows = min(GBM, g.M - mt * GBM);
      if (!dead) {
        uint8_t *out = static_cast<uint8_t *>(p.out) + (size_t)mt * GBM * p.Cout + n0;
        if (g.out_vec == 16 && p.Cout % 16 == 0) {
          // rows are whole 16-byte pieces
          const int per = ncols >> 4;
          for (int i = tid; i < rows * per; i += GT) {
            const int rr = ncols == bn ? g.by_cols.div(i) : i / per, c = i - rr * per;
            *reinterpret_cast<uint4 *>(out + (size_t)rr * p.Cout + 16 * c) = *reinterpret_cast<const uint4 *>(staging + rr * pitch + 16 * c);
          }
        } else if (linear) {
          // the run starts at a multiple of 128 bytes of the output
          const int total = rows * ncols;
          int done;
          if ((reinterpret_cast<uintptr_t>(p.out) & 15) == 0) {
            done = total & ~15;
            for (int o = 16 * tid; o < done; o += 16 * GT) *reinterpret_cast<uint4 *>(out + o) = *reinterpret_cast<const uint4 *>(staging + o);
          } else {
            done = total & ~3;
            for (int o = 4 * tid; o < done; o += 4 * GT) *reinterpret_cast<unsigned *>(out + o) = *reinterpret_cast<const unsigned *>(staging + o);
          }
          for (int o = done + tid; o < total; o += GT) out[o] = staging[o];
        } else if (g.out_vec >= 4 && p.Cout % 4 == 0) {
          const int per = ncols >> 2;
          for (int i = tid; i < rows * per; i += GT) {
            const int rr = i / per, c = i - rr * per;
            *reinterpret_cast<unsigned *>(out + (size_t)rr * p.Cout + 4 * c) = *reinterpret_cast<const unsigned *>(staging + rr * pitch + 4 * c);
          }
        } else {
          // byte by byte: a warp to a row while that fills its lanes
          if (ncols >= 64) {
#pragma unroll 2
            for (int rr = warp; rr < rows; rr += GT / 32)
              for (int c = lane; c < ncols; c += 32) out[(size_t)rr * p.Cout + c] = staging[rr * pitch + c];
          } else {
            const FastDiv &by = nt == g.n_tiles - 1 ? g.by_last : g.by_bn;
#pragma unroll 4
            for (int i = tid; i < rows * ncols; i += GT) {
              const int rr = by.div(i), c = i - rr * ncols;
              out[(size_t)rr * p.Cout + c] = staging[rr * pitch + c];
            }
          }
        }
      }
    }
    __syncthreads();           // the staging tile and the accumulator are free for the next tile
    tc_fence_after();
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, (uint32_t)g.tmem_cols);
  }
}

constexpr int SMEM_SM = 227 * 1024;
constexpr int STATIC_SMEM = 4096 + 256;       // parameters, barriers
constexpr int SMEM_RESERVED = 1024;           // taken by the system per CTA

template <int MODE, bool ALIGNED, bool W_RES>
bool launch_gather(Context &c, const GatherParams &g, int grid, int smem)
{
  auto kern = conv_gather_tc_kernel<MODE, ALIGNED, W_RES>;
  static PerDeviceInt attr_set;
  if (!attr_set.get(c.device)) {
    if (!cuda_ok(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_SM / 2), "cudaFuncSetAttribute(conv_gather_tc)"))
      return false;
    attr_set.set(c.device, 1);
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid); cfg.blockDim = dim3(GT); cfg.dynamicSmemBytes = (size_t)smem; cfg.stream = c.stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = (unsigned)g.k_split; attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr; cfg.numAttrs = g.k_split > 1 ? 2 : 1;
  const cudaError_t le = cudaLaunchKernelEx(&cfg, kern, g);
  count_launch("conv_gather_tc_kernel");
  return cuda_ok(le, "conv_gather_tc launch") && cuda_ok(cudaGetLastError(), "conv_gather_tc launch");
}

template <bool ALIGNED, bool W_RES>
bool launch_gather_mode(Context &c, const GatherParams &g, int grid, int smem)
{
  switch (g.p.epi.mode) {
    case EPI_NONE: return launch_gather<EPI_NONE, ALIGNED, W_RES>(c, g, grid, smem);
    case EPI_MULT: return launch_gather<EPI_MULT, ALIGNED, W_RES>(c, g, grid, smem);
    case EPI_BN32: return launch_gather<EPI_BN32, ALIGNED, W_RES>(c, g, grid, smem);
    case EPI_BN64: return launch_gather<EPI_BN64, ALIGNED, W_RES>(c, g, grid, smem);
    default:       return launch_gather<EPI_RAW32, ALIGNED, W_RES>(c, g, grid, smem);
  }
}

}  // namespace

bool conv_gather_tc_supported(const ConvProblem &p)
{
  // 32-bit offsets into the tensors, padding rows and a chunk of slack included
  const long long lim = 0x7fff0000LL, row = (long long)p.W * p.Cin, run = (long long)p.kx * p.Cin;
  const long long M = (long long)p.B * p.Ho * p.Wo;
  if (M < 1 || M > lim || (long long)p.B * p.H * row + (long long)(p.pt + p.ky) * row + (long long)p.pl * p.Cin > lim) return false;
  return (long long)p.Cout * p.ky * run <= lim && p.ky * ((run + 15) / 16) <= (1 << 20);
}

// Cuts the problem into tiles and a reduction into the CTAs of a cluster; returns the rounds of tiles
static long long plan_gather(const ConvProblem &p, int sms, GatherParams &g)
{
  g.p = p;
  g.M = p.B * p.Ho * p.Wo;
  g.K = p.ky * p.kx * p.Cin;
  g.run = p.kx * p.Cin;
  g.run_chunks = (g.run + 15) / 16;
  g.chunks = p.ky * g.run_chunks;
  g.slabs = (g.chunks + 7) / 8;
  g.m_tiles = (g.M + GBM - 1) / GBM;

  // How many ways to cut the channels (bn = 16 .. 256) and the reduction (1 .. 8 CTAs of a cluster): the
  // cheapest count of gathered rows on the busiest SM's pair of CTAs. A tile's set-up, drain and stores
  // weigh about 300 rows, the exchange through the cluster 150 more; at least two slabs per CTA.
  // Rows of no whole words in several tiles leave byte by byte.
  const bool bytewise = p.epi.mode != EPI_RAW32 && (p.Cout % 4 != 0 || (reinterpret_cast<uintptr_t>(p.out) & 3));
  long long best = -1, best_rounds = 1;
  for (int split = 1; split <= 8; split *= 2) {
    const int per = (g.slabs + split - 1) / split;
    if (split > 1 && (per < 2 || (split - 1) * per >= g.slabs)) break;
    const int fewest = (p.Cout + 255) / 256;
    for (int want = fewest; want == fewest || (long long)g.m_tiles * want * split <= 2 * sms; want += (want + 3) / 4) {
      const int bn = ((p.Cout + want - 1) / want + 15) & ~15, nt = (p.Cout + bn - 1) / bn;
      if (split > 1 && bn > 64) continue;              // the partial sums have to fit the ring
      const long long rounds = ((long long)g.m_tiles * nt * split + 2 * sms - 1) / (2 * sms);
      const long long cost = rounds * ((long long)per * (GBM + bn) + 300 + (split > 1 ? 150 : 0) + (bytewise && nt > 1 && split == 1 ? 100 + bn : 0));
      if (best < 0 || cost < best) { best = cost; best_rounds = rounds; g.bn = bn; g.n_tiles = nt; g.k_split = split; g.slabs_per = per; }
      if (bn == 16) break;
    }
  }
  return best_rounds;
}

static bool gather_aligned(const ConvProblem &p)
{
  return p.Cin % 16 == 0 && ((reinterpret_cast<uintptr_t>(p.in) | reinterpret_cast<uintptr_t>(p.w)) & 15) == 0;
}

// Fitted to 1900 calls of 2 to 300 us (standard deviation 11 %): a tile's slabs by the rows gathered for each, twice as
// dear where chunks cross pixels, its drain by the columns, and the exchange of a shared reduction.
double conv_gather_tc_estimate(const Context &c, const ConvProblem &p, double worth)
{
  if (!conv_gather_tc_supported(p)) return -1;
  // one round of the smallest tiles over an eighth of the slabs: the plan is looked for only if that is of interest
  const int eighth = ((p.ky * ((p.kx * p.Cin + 15) / 16) + 7) / 8 + 7) / 8;
  const double least = 2960 + (gather_aligned(p) ? 4.7 : 8.3) * eighth * (GBM + 16);
  if (least >= worth) return least;
  GatherParams g = {};
  const double rounds = (double)plan_gather(p, c.sm_count > 0 ? c.sm_count : 148, g);
  return 2060 + rounds * (900 + (gather_aligned(p) ? 4.7 : 8.3) * g.slabs_per * (GBM + g.bn) + 10 * g.bn) + (g.k_split > 1 ? 46 * g.bn : 0);
}

bool launch_conv_gather_tc(Context &c, const ConvProblem &p)
{
  GatherParams g = {};
  const int sms = c.sm_count > 0 ? c.sm_count : 148;
  plan_gather(p, sms, g);
  g.by_pixels.set((unsigned)(p.Ho * p.Wo));
  g.by_wo.set((unsigned)p.Wo);
  g.by_chunks.set((unsigned)g.run_chunks);
  g.tmem_cols = 32;
  while (g.tmem_cols < g.bn) g.tmem_cols *= 2;
  const uintptr_t out_a = reinterpret_cast<uintptr_t>(p.out);
  g.out_vec = (p.Cout % 16 == 0 && (out_a & 15) == 0) ? 16 : ((out_a & 3) == 0 ? 4 : 1);

  g.by_bn.set((unsigned)g.bn);
  g.by_last.set((unsigned)(p.Cout - (g.n_tiles - 1) * g.bn));
  g.by_cols.set((unsigned)(g.bn / 16));              // 16-byte pieces of a full tile's row

  // two CTAs per SM: the ring, which also holds the output tile, and, if it fits beside three stages, all of W (two
  // stages where 256 columns of W are streamed)
  const int half_sm = SMEM_SM / 2 - STATIC_SMEM - SMEM_RESERVED - 1024;
  const long long w_all = (long long)g.slabs_per * g.bn * 128;
  const bool w_res = w_all + 3 * A_STAGE <= half_sm;
  const int stage = w_res ? A_STAGE : A_STAGE + g.bn * 128;
  int stages = (int)((half_sm - (w_res ? w_all : 0)) / stage);
  if (stages > MAX_G_STAGES) stages = MAX_G_STAGES;
  g.stages = stages;
  const int smem = (int)(w_res ? w_all : 0) + stages * stage + 1024;

  if (!ctx_status_word_unless_capturing(c, &g.status)) return false;

  const int lanes = g.n_tiles * g.k_split;             // CTAs that work on one row of tiles
  int per = 2 * sms / lanes;
  if (per < 1) per = 1;
  const int grid = lanes * (per < g.m_tiles ? per : g.m_tiles);
  if (gather_aligned(p)) return w_res ? launch_gather_mode<true, true>(c, g, grid, smem) : launch_gather_mode<true, false>(c, g, grid, smem);
  return w_res ? launch_gather_mode<false, true>(c, g, grid, smem) : launch_gather_mode<false, false>(c, g, grid, smem);
}

}  // namespace pulpnn
