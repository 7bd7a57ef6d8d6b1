// igemm_split.cu -- the u8 x s8 -> s32 GEMM of igemm_tc.cu for problems of FEW tiles: small batches, single
// images, fully connected layers. A persistent kernel with wide tiles leaves most SMs idle there and walks a
// long reduction alone; here the reduction of a tile is shared by the CTAs of a cluster (up to eight), which add
// their partial sums through distributed shared memory (split_epilogue.cuh), in ONE kernel and without scratch.
// Arithmetic and operand layouts as in igemm_tc.cu (32bit/src/pulp_nn_matmul.c:27-298, pulp_nn_linear.c:58-108,
// pulp_nn_conv_Ho_parallel.c:80-249).
//
// One CTA (8 warps) computes 128 rows (a patch of 128 output pixels of a spatial convolution) x BN columns over its
// share of the K-slabs: two threads keep a ring of TMA loads in flight, one issues the MMAs, all eight warps drain
// the accumulator and finish their share of the rows.
//
// What bounds it: the fixed cost of a kernel (launch, barriers, tensor memory, one round trip to L2, the exchange:
// some 4 us), then the bytes into an SM. Columns and slices are chosen by plan_split's estimate of both. Measured (us,
// graph replay; the two-kernel split through scratch or dp4a before): 4096 -> 4096 at 128 vectors 87 -> 10.3, at 256
// 17.4 -> 12.5 (50 MB into the SMs), 14x14x512 -> 512 of one image 13.7 -> 4.1 (5.6 with the tile
// put together in shared memory, which a tile of one CTA does without), 7x7x1024 -> 1024 at batch 4 19.8 -> 5.7.
#include "internal.cuh"
#include "split_epilogue.cuh"
#include "sm100_primitives.cuh"
#include "tensor_maps.cuh"

namespace pulpnn {

namespace {

using namespace sm100;

constexpr int SBM = 128, STHREADS = 256, MAX_S_STAGES = 12;
constexpr int ST_S_EMPTY = 0x10000, ST_S_FULL = 0x20000, ST_S_DONE = 0x40000, ST_S_DRAIN = 0x80000;

struct SplitParams {
  Epilogue epi;
  void *out;
  int M, N, K;
  int m_tiles, n_tiles, bn;
  int k_split, slabs_per, slabs;
  int stages, tmem_cols;
  int direct;              // one CTA per tile and whole 16-byte pieces: rows leave from registers
  int const_weights;       // W belongs to a network: no kernel writes it
  int conv, tw_log2, tiles_x, tiles_y, chunks_per_tap, kx, sx, sy, pl, pt, Ho, Wo;    // as in igemm_tc.cu
  int *status;
};

template <int MODE, int BKB>
__global__ void __launch_bounds__(STHREADS, 2)
igemm_split_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const SplitParams g)
{
  extern __shared__ uint8_t smem_raw[];
  uint8_t *ring = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  __shared__ uint64_t full_bar[MAX_S_STAGES], empty_bar[MAX_S_STAGES], done_bar;
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_word;
  __shared__ __align__(16) long long par_k[256], par_l[256];
  volatile int *abort_flag = &abort_word;

  const int tid = threadIdx.x, warp = tid >> 5;
  const int a_bytes = SBM * BKB, stage_bytes = a_bytes + g.bn * BKB;
  const int ks = (int)(blockIdx.x % (unsigned)g.k_split);
  const unsigned tile = blockIdx.x / (unsigned)g.k_split;
  const int nt = (int)(tile % (unsigned)g.n_tiles), mt = (int)(tile / (unsigned)g.n_tiles);
  const int n0 = nt * g.bn, ncols = min(g.bn, g.N - n0);
  const int slab0 = ks * g.slabs_per, nslabs = min(slab0 + g.slabs_per, g.slabs) - slab0;

  // first output pixel of a convolution's patch
  int cb = 0, cy = 0, cx = 0;
  if (g.conv) {
    const int r = mt / g.tiles_x;
    cx = (mt - r * g.tiles_x) << g.tw_log2;
    cb = r / g.tiles_y;
    cy = (r - cb * g.tiles_y) << (7 - g.tw_log2);
  }

  if (tid == 0) {
    for (int s = 0; s < g.stages; s++) { mbar_init(&full_bar[s], 2); mbar_init(&empty_bar[s], 1); }
    mbar_init(&done_bar, 1);
    abort_word = 0;
    mbar_fence_init();
  }
  if (warp == 1) tmem_alloc(&tmem_slot, (uint32_t)g.tmem_cols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;

  if (tid == 0 || tid == 64) {
    // ------------------------------ TMA producers: A and W --------------------------------------
    // (getting a load on its way takes a thread several hundred cycles: one thread for both operands was what
    // bounded the narrow slabs of a spatial convolution)
    const bool is_a = tid == 0;
    auto load = [&](int i) {
      const int st = i % g.stages, s = slab0 + i;
      uint8_t *dst = ring + st * stage_bytes;
      mbar_arrive_expect_tx(&full_bar[st], (uint32_t)(is_a ? a_bytes : stage_bytes - a_bytes));
      if (!is_a) tma_load_2d(dst + a_bytes, &map_b, &full_bar[st], s * BKB, n0);
      else if (g.conv) {
        const int tap = s / g.chunks_per_tap, chunk = s - tap * g.chunks_per_tap;
        const int fy = tap / g.kx, fx = tap - fy * g.kx;
        tma_load_4d(dst, &map_a, &full_bar[st], chunk * BKB, cx * g.sx - g.pl + fx, cy * g.sy - g.pt + fy, cb);
      } else tma_load_2d(dst, &map_a, &full_bar[st], s * BKB, mt * SBM);
    };
    // a network's weights are constants: their first slabs may come before the previous kernel has ended
    int issued = 0;
    if (!is_a && g.const_weights)
      for (; issued < min(g.stages, nslabs); issued++) load(issued);
    pdl_wait();
    if (is_a) pdl_launch_dependents();
    for (; issued < nslabs; issued++) {
      if (issued >= g.stages &&
          !mbar_wait(&empty_bar[issued % g.stages], (uint32_t)(issued / g.stages - 1) & 1u, abort_flag, g.status, ST_S_EMPTY)) break;
      load(issued);
    }
    if (*abort_flag) {
      // none of the loads may still be on its way into this CTA's memory when it leaves
      for (int i = max(issued - g.stages, 0); i < issued; i++) {
        const unsigned long long t0 = global_ns();
        while (!mbar_try_wait(&full_bar[i % g.stages], (uint32_t)(i / g.stages) & 1u))
          if (global_ns() - t0 > WAIT_LIMIT_NS) { if (g.status) atomicOr(g.status, ST_S_DRAIN); break; }
      }
    }
  } else {
    pdl_wait();
  }
  if (tid == 32) {
    // ------------------------------ MMA issuer --------------------------------------------------
    const uint32_t idesc = umma_idesc_u8s8(g.bn);
    bool ok = true;
    for (int i = 0; i < nslabs && ok; i++) {
      const int st = i % g.stages;
      ok = mbar_wait(&full_bar[st], (uint32_t)(i / g.stages) & 1u, abort_flag, g.status, ST_S_FULL);
      if (!ok) break;
      tc_fence_after();
      const uint32_t a_addr = smem_u32(ring + st * stage_bytes);
      const uint64_t da = umma_smem_desc<BKB>(a_addr), db = umma_smem_desc<BKB>(a_addr + a_bytes);
      const int kbytes = min(BKB, g.K - (slab0 + i) * BKB);      // the rest of the slab is zero-filled
      const int n_mma = (kbytes + 31) / 32;
      for (int j = 0; j < n_mma; j++) umma_i8(tmem, da + (uint64_t)(2 * j), db + (uint64_t)(2 * j), idesc, (i > 0 || j > 0) ? 1u : 0u);
      umma_commit(&empty_bar[st]);
    }
    if (ok) umma_commit(&done_bar);
  }
  if (tid >= 96) stage_channel_params<MODE>(g.epi, n0, ncols, par_k, par_l, tid - 96, STHREADS - 96);
  __syncwarp();
  bool dead = !mbar_wait(&done_bar, 0, abort_flag, g.status, ST_S_DONE);
  dead = __syncthreads_or(dead);
  tc_fence_after();
  const int m0 = mt * SBM;
  auto row_of = [&](int r) -> long long {
    if (!g.conv) return m0 + r < g.M ? m0 + r : -1;
    const int y = cy + (r >> g.tw_log2), x = cx + (r & ((1 << g.tw_log2) - 1));
    return y < g.Ho && x < g.Wo ? ((long long)cb * g.Ho + y) * g.Wo + x : -1;
  };
  if (MODE != EPI_RAW32 && g.direct) {
    if (!dead) {
      const int quad = warp & 3;
      const long long row = row_of(quad * 32 + (tid & 31));
      uint8_t *out = static_cast<uint8_t *>(g.out) + (size_t)(row < 0 ? 0 : row) * g.N + n0;
      for (int c0 = (warp >> 2) * 32; c0 < ncols; c0 += 64) {
        uint32_t v[32];
        tmem_ld_32(tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)c0, v);
        tmem_wait_ld();
        unsigned w[8];
        requant32_cols<MODE == EPI_RAW32 ? EPI_NONE : MODE>(v, c0, ncols, par_k, par_l, g.epi, g.K, w);
        if (row >= 0) {
          *reinterpret_cast<uint4 *>(out + c0) = make_uint4(w[0], w[1], w[2], w[3]);
          if (c0 + 16 < ncols) *reinterpret_cast<uint4 *>(out + c0 + 16) = make_uint4(w[4], w[5], w[6], w[7]);
        }
      }
    }
  } else {
    split_epilogue<MODE>(g.epi, g.out, g.N, g.bn, g.k_split, ks, n0, ncols, ring, tmem, par_k, par_l, dead, row_of);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, (uint32_t)g.tmem_cols);
  }
}

constexpr int SPLIT_SMEM = 220 * 1024, SPLIT_SMEM_TWO = 108 * 1024;     // one / two CTAs on an SM

// CTAs of clusters of `split` that are on the GPU at the same time: a cluster sits in one GPC, whose SMs are no
// multiple of four or eight (cudaOccupancyMaxActiveClusters on 148 SMs: 132 and 120 at one CTA an SM, 284 and 264 at two)
int resident(int sms, int split, bool two)
{
  if (two) return split <= 2 ? 2 * sms : (split == 4 ? sms * 284 / 148 : sms * 264 / 148);
  return split <= 2 ? sms : (split == 4 ? sms * 132 / 148 : sms * 120 / 148);
}

template <int MODE, int BKB>
bool launch_split(Context &c, const CUtensorMap &a, const CUtensorMap &b, const SplitParams &g, int smem)
{
  auto kern = igemm_split_kernel<MODE, BKB>;
  static PerDeviceInt attr_set;
  if (!attr_set.get(c.device)) {
    if (!cuda_ok(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SPLIT_SMEM), "cudaFuncSetAttribute(igemm_split)"))
      return false;
    attr_set.set(c.device, 1);
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(g.m_tiles * g.n_tiles * g.k_split));
  cfg.blockDim = dim3(STHREADS); cfg.dynamicSmemBytes = (size_t)smem; cfg.stream = c.stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = (unsigned)g.k_split; attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr; cfg.numAttrs = g.k_split > 1 ? 2 : 1;
  const cudaError_t le = cudaLaunchKernelEx(&cfg, kern, a, b, g);
  count_launch("igemm_split_kernel");
  return cuda_ok(le, "igemm_split launch") && cuda_ok(cudaGetLastError(), "igemm_split launch");
}

template <int MODE>
bool launch_split_bk(Context &c, const CUtensorMap &a, const CUtensorMap &b, const SplitParams &g, int bkb, int smem)
{
  if (bkb == 32) return launch_split<MODE, 32>(c, a, b, g, smem);
  if (bkb == 64) return launch_split<MODE, 64>(c, a, b, g, smem);
  return launch_split<MODE, 128>(c, a, b, g, smem);
}

// The cut of the problem with the least estimated time; returns that time in ns, or -1 when the tiles alone are more
// than the SMs (igemm_tc.cu's persistent CTAs are the better form then).
double plan_split(const ConvProblem &p, int sms, SplitParams &g, int &bkb, int &smem)
{
  g.epi = p.epi; g.out = p.out;
  g.M = p.B * p.Ho * p.Wo; g.N = p.Cout; g.K = p.ky * p.kx * p.Cin;
  g.conv = igemm_is_plain(p) ? 0 : 1;
  g.kx = p.kx; g.sx = p.sx; g.sy = p.sy; g.pl = p.pl; g.pt = p.pt; g.Ho = p.Ho; g.Wo = p.Wo;
  g.tw_log2 = 7; g.tiles_x = g.tiles_y = 1; g.chunks_per_tap = 1;
  long long m_tiles;
  if (g.conv) {
    bkb = p.Cin % 128 == 0 ? 128 : (p.Cin % 64 == 0 ? 64 : 32);
    g.chunks_per_tap = p.Cin / bkb;
    g.tw_log2 = pick_patch_width_log2(p.Ho, p.Wo, p.sx, p.sy);
    g.tiles_x = (p.Wo + (1 << g.tw_log2) - 1) >> g.tw_log2;
    g.tiles_y = (p.Ho + (128 >> g.tw_log2) - 1) / (128 >> g.tw_log2);
    m_tiles = (long long)p.B * g.tiles_x * g.tiles_y;
  } else {
    bkb = g.K <= 32 ? 32 : (g.K <= 64 ? 64 : (g.K < 128 && g.K % 64 != 0 ? 32 : 128));
    m_tiles = (g.M + SBM - 1) / SBM;
  }
  if (m_tiles > 2 * sms) return -1;
  g.m_tiles = (int)m_tiles;
  g.slabs = (g.K + bkb - 1) / bkb;
  const bool pieces = p.epi.mode != EPI_RAW32 && p.Cout % 16 == 0 && (reinterpret_cast<uintptr_t>(p.out) & 15) == 0;
  double best = -1;
  bool best_two = false;
  for (int bn = 256; bn >= 32; bn /= 2) {
    if (bn > 32 && bn / 2 >= g.N) continue;
    const int nt = (g.N + bn - 1) / bn;
    for (int split = 1; split <= 8; split *= 2) {
      const int per = (g.slabs + split - 1) / split, ctas = g.m_tiles * nt * split;
      if (split > 1 && (split - 1) * per >= g.slabs) break;
      const bool two = ctas > resident(sms, split, false);
      if (two && (bn > 128 || ctas > resident(sms, split, true))) break;
      // bytes into the busiest SM at 70 per ns and into all of them at 9000; the tensor pipe's BN/2 cycles per 32 bytes
      // of K; the drain, the finishing of a CTA's rows and, for a shared reduction, its way through the cluster at 40
      // bytes per ns (fitted to 20 shapes between 8 x 256 x 512 and 3136 x 512 x 512)
      const double load = (two ? 2.0 : 1.0) * per * bkb * (SBM + bn) / 70.0;
      const double l2 = (double)g.m_tiles * nt * g.slabs * bkb * (SBM + bn) / 9000.0;
      const double mma = (two ? 2.0 : 1.0) * per * bkb / 32 * bn / 3.8;
      double t = load > l2 ? load : l2;
      t = (t > mma ? t : mma) + bn * 6.0 + (split == 1 && pieces ? 0.0 : 25.0 * bn / split) +
          (split > 1 ? 400.0 + 512.0 * bn * (split - 1) / split / 40.0 : 0.0);
      if (best < 0 || t < best) { best = t; best_two = two; g.bn = bn; g.n_tiles = nt; g.k_split = split; g.slabs_per = per; }
    }
  }
  if (best < 0) return -1;
  g.tmem_cols = g.bn;
  g.direct = pieces && g.k_split == 1;
  const int stage = (SBM + g.bn) * bkb, tile = SBM * (g.bn + 4) * 4;
  int stages = ((best_two || g.slabs_per * stage <= SPLIT_SMEM_TWO ? SPLIT_SMEM_TWO : SPLIT_SMEM) - 1024) / stage;
  if (stages > MAX_S_STAGES) stages = MAX_S_STAGES;
  if (stages > g.slabs_per) stages = g.slabs_per;
  g.stages = stages;
  smem = (stages * stage > tile ? stages * stage : tile) + 1024;
  return best;
}

}  // namespace

double igemm_split_estimate(const Context &c, const ConvProblem &p)
{
  if (!igemm_tc_supported(c, p)) return -1;
  SplitParams g = {};
  int bkb = 0, smem = 0;
  const double ns = plan_split(p, c.sm_count > 0 ? c.sm_count : 148, g, bkb, smem);
  if (ns < 0 || !g.conv) return ns < 0 ? -1 : 3400.0 + ns;
  // a spatial convolution waits for getting its boxes on their way, 400 to 480 ns a slab (fitted to 466 calls of 4 to 100 us)
  const double slabs = (bkb == 128 ? 403.0 : (bkb == 64 ? 463.0 : 483.0)) * g.slabs_per;
  return 2470.0 + (1.33 * ns > slabs ? 1.33 * ns : slabs);
}

bool launch_igemm_split(Context &c, const ConvProblem &p)
{
  SplitParams g = {};
  int bkb = 128, smem = 0;
  if (plan_split(p, c.sm_count > 0 ? c.sm_count : 148, g, bkb, smem) < 0) return false;
  g.const_weights = p.folded != nullptr;
  if (!ctx_status_word_unless_capturing(c, &g.status)) return false;
  CUtensorMap a, b;
  if (g.conv) {
    if (!make_map_4d(&a, p.in, p.Cin, p.W, p.H, p.B, bkb, 1 << g.tw_log2, 128 >> g.tw_log2, p.sx, p.sy)) return false;
  } else if (!make_map(&a, p.in, g.M, g.K, SBM, bkb)) return false;
  if (!make_map(&b, p.w, g.N, g.K, g.bn, bkb)) return false;
  switch (p.epi.mode) {
    case EPI_NONE: return launch_split_bk<EPI_NONE>(c, a, b, g, bkb, smem);
    case EPI_MULT: return launch_split_bk<EPI_MULT>(c, a, b, g, bkb, smem);
    case EPI_BN32: return launch_split_bk<EPI_BN32>(c, a, b, g, bkb, smem);
    case EPI_BN64: return launch_split_bk<EPI_BN64>(c, a, b, g, bkb, smem);
    default:       return launch_split_bk<EPI_RAW32>(c, a, b, g, bkb, smem);
  }
}

}  // namespace pulpnn
