// conv_halo_tc.cu -- spatial convolution, strides 1 and 2, on the tensor cores with every input pixel fetched ONCE
// per tile (arithmetic of igemm_tc.cu; 32bit/src/pulp_nn_conv_Ho_parallel.c:80-249).
//
// igemm_tc.cu fetches a tile's operand tap by tap: nine TMA boxes of the same pixels for a 3x3 kernel, and with
// the weights streamed beside them that traffic into the SM is what its convolutions wait for. Here a tile is a
// patch of 8 x 16 output pixels, and ONE box per chunk of channels brings the (8 + kx - 1) x (16 + ky - 1) input
// pixels it reads (zeros outside the image). In shared memory a pixel is a row of BKB bytes, swizzled; the A
// operand of tap (fy, fx) is the box read from pixel (fy, fx) on: its 16 groups of eight rows are runs of eight
// pixels, one box row apart (the descriptor's stride). The swizzle is a function of the absolute shared-memory
// address for TMA and MMA alike, so a shifted start needs nothing else. The CTA's slice of W stays in shared
// memory for its lifetime; a 128-channel 3x3 tile then takes 23 KB from L2 instead of 295.
//
// Roles of a CTA (persistent, 18 warps): warp 0 TMA, warp 1 MMA issue, warps 2..17 four epilogue groups that take the
// tiles in turn from a ring of accumulators in tensor memory and store the requantised rows from registers.
//
// What bounds it: the MMAs -- one costs some 80 cycles, bound by reading 32 bytes of each of its rows, so the issuing
// thread adds a tabled offset per tap and nothing else (with the offsets computed there a tap of one MMA took 270
// cycles) --, for 32- and 64-channel slabs the rows of the TMA box, and a last round of tiles that is not full.
// Measured (us, graph replay, the kernel before / this one): 3x3 28x28x128 -> 128 at batch 32 11.9 / 8.3, at batch 1 6.7 /
// 4.6; 56x56x64 -> 64 at batch 64 31.3 / 20.1; 112x112x64 -> 64 at batch 16 31.4 / 17.8; 56x56x96 -> 96 at batch 32
// 27.8 / 20.6; 32x32x32 -> 64 at batch 1 4.5 / 3.4; 5x5 28x28x64 -> 64 at batch 32 17.0 / 9.0; stride 2 56x56x64 -> 128 at
// batch 32 8.8 / 6.9. Tried: a staging tile and 16-byte pieces instead of 32-byte stores, with 8 warps: 8.0 and 22.3
// us on the first two (before the issue loop was cut down; with four groups of epilogue warps 8.8 and 23.3).
#include "internal.cuh"
#include "split_epilogue.cuh"
#include "sm100_primitives.cuh"
#include "tensor_maps.cuh"

namespace pulpnn {

namespace {

using namespace sm100;

constexpr int HTW = 8, HTH = 16;                     // output pixels of a patch
constexpr int H_GROUPS = 4, HTHREADS = 64 + 128 * H_GROUPS;   // warps 2..17: groups of four, one per TMEM lane quarter
constexpr int MAX_BOXES = 4, MAX_ACC = 4, MAX_TAPS = 81;
constexpr int ST_H_BOX = 0x100000, ST_H_FULL = 0x200000, ST_H_ACC = 0x400000, ST_H_EPI = 0x800000;

struct HaloParams {
  Epilogue epi;
  uint8_t *out;
  int N, K, Ho, Wo, pt, pl, ky, kx;
  int chunks;                        // channel chunks of BKB bytes
  int sx, sy;                        // 1 or 2: sx * sy boxes of every sx-th, sy-th pixel per chunk
  int box_w, box_h, box_bytes, box_pitch, box_stride, n_boxes;      // one box, to the next box, all boxes of a chunk
  int tiles_x, tiles_y, m_tiles, n_tiles, bn, acc_cols, n_acc;
  int wide_store;                    // 32-byte stores
  int const_weights;
  FastDiv by_tx, by_ty;
  int *status;
};

// K-major operand whose groups of eight rows are `sbo` bytes apart (see umma_smem_desc)
template <int BKB>
__device__ __forceinline__ uint64_t strided_desc(uint32_t saddr, uint32_t sbo)
{
  constexpr uint64_t layout = BKB == 128 ? 2 : (BKB == 64 ? 4 : 6);
  return (uint64_t)((saddr & 0x3ffffu) >> 4) | (uint64_t)1 << 16 | (uint64_t)(sbo >> 4) << 32 | (uint64_t)1 << 46 | layout << 61;
}

template <int MODE, int BKB>
__global__ void __launch_bounds__(HTHREADS, 1)
conv_halo_tc_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w, const HaloParams g)
{
  extern __shared__ uint8_t smem_raw[];
  uint8_t *smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  __shared__ uint64_t box_full[MAX_BOXES], box_empty[MAX_BOXES], t_full[MAX_ACC], t_empty[MAX_ACC], w_bar;
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_word;
  __shared__ uint32_t tap_off[MAX_TAPS + 1];           // start of each tap's operand in the boxes, 16-byte units
  __shared__ __align__(16) long long par_k[256], par_l[256];
  volatile int *abort_flag = &abort_word;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int taps = g.ky * g.kx, w_slab = g.bn * BKB, slabs = taps * g.chunks;
  uint8_t *boxes = smem + slabs * w_slab;
  const int nt = (int)(blockIdx.x % (unsigned)g.n_tiles);
  const int m0 = (int)(blockIdx.x / (unsigned)g.n_tiles), m_step = (int)(gridDim.x / (unsigned)g.n_tiles);
  const int n0 = nt * g.bn, ncols = min(g.bn, g.N - n0);

  if (tid == 0) {
    for (int s = 0; s < g.n_boxes; s++) { mbar_init(&box_full[s], 1); mbar_init(&box_empty[s], 1); }
    for (int a = 0; a < g.n_acc; a++) { mbar_init(&t_full[a], 1); mbar_init(&t_empty[a], 4 * H_GROUPS / g.n_acc); }
    mbar_init(&w_bar, 1);
    abort_word = 0;
    mbar_fence_init();
  }
  for (int t = tid; t <= taps; t += HTHREADS) {
    const int fy = t / g.kx, fx = t - fy * g.kx;
    const int q = (fy % g.sy) * g.sx + fx % g.sx;       // the box of this tap's pixels
    tap_off[t] = (uint32_t)(q * g.box_pitch + (fy / g.sy * g.box_w + fx / g.sx) * BKB) >> 4;
  }
  if (warp == 1) tmem_alloc(&tmem_slot, (uint32_t)(g.n_acc * g.acc_cols));
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  auto patch = [&](int mt, int &b, int &y, int &x) {
    const int r = g.by_tx.div(mt);
    x = (mt - r * g.tiles_x) * HTW;
    b = g.by_ty.div(r);
    y = (r - b * g.tiles_y) * HTH;
  };

  if (warp == 0) {
    if (lane == 0) {
      // ------------------------------ TMA ------------------------------------------------------
      auto load_w = [&] {
        mbar_arrive_expect_tx(&w_bar, (uint32_t)(slabs * w_slab));
        for (int s = 0; s < slabs; s++) tma_load_2d(smem + s * w_slab, &map_w, &w_bar, s * BKB, n0);
      };
      if (g.const_weights) load_w();       // a network's weights are constants
      pdl_wait();
      pdl_launch_dependents();
      if (!g.const_weights) load_w();
      int st = 0, issued = 0;
      uint32_t lap = 0;
      bool ok = true;
      for (int mt = m0; mt < g.m_tiles && ok; mt += m_step) {
        int b, y, x;
        patch(mt, b, y, x);
        for (int c = 0; c < g.chunks; c++) {
          if (lap > 0 && !mbar_wait(&box_empty[st], (lap - 1) & 1u, abort_flag, g.status, ST_H_BOX)) { ok = false; break; }
          mbar_arrive_expect_tx(&box_full[st], (uint32_t)(g.sx * g.sy * g.box_bytes));
          for (int q = 0; q < g.sx * g.sy; q++)
            tma_load_4d(boxes + st * g.box_stride + q * g.box_pitch, &map_a, &box_full[st], c * BKB, x * g.sx - g.pl + q % g.sx,
                        y * g.sy - g.pt + q / g.sx, b);
          issued++;
          if (++st == g.n_boxes) { st = 0; lap++; }
        }
      }
      if (*abort_flag) {
        // none of the loads may still be on its way into this CTA's memory when it leaves
        for (int i = max(issued - g.n_boxes, 0); i <= issued; i++) {
          const unsigned long long t0 = global_ns();
          while (!(i == issued ? mbar_try_wait(&w_bar, 0) : mbar_try_wait(&box_full[i % g.n_boxes], (uint32_t)(i / g.n_boxes) & 1u)))
            if (global_ns() - t0 > WAIT_LIMIT_NS) break;
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      // ------------------------------ MMA ------------------------------------------------------
      const uint32_t idesc = umma_idesc_u8s8(g.bn), sbo = (uint32_t)(g.box_w * BKB);
      const uint64_t w_step = (uint64_t)((g.chunks * w_slab) >> 4);
      bool ok = mbar_wait(&w_bar, 0, abort_flag, g.status, ST_H_FULL);
      int st = 0, i = 0;
      uint32_t lap = 0;
      for (int mt = m0; mt < g.m_tiles && ok; mt += m_step, i++) {
        const int acc = i % g.n_acc;
        if (!mbar_wait(&t_empty[acc], ((uint32_t)(i / g.n_acc) & 1u) ^ 1u, abort_flag, g.status, ST_H_ACC)) break;
        tc_fence_after();
        const uint32_t d = tmem + (uint32_t)(acc * g.acc_cols);
        for (int c = 0; c < g.chunks && ok; c++) {
          ok = mbar_wait(&box_full[st], lap & 1u, abort_flag, g.status, ST_H_FULL);
          if (!ok) break;
          tc_fence_after();
          // one thread issues everything: what it does per tap is an addition to each descriptor's start address
          const uint64_t a0 = strided_desc<BKB>(smem_u32(boxes + st * g.box_stride), sbo);
          uint64_t db = umma_smem_desc<BKB>(smem_u32(smem + c * w_slab));
          uint32_t off = tap_off[0];
#pragma unroll 3
          for (int tap = 0; tap < taps; tap++) {
            const uint64_t da = a0 + off;
            off = tap_off[tap + 1];
#pragma unroll
            for (int j = 0; j < BKB / 32; j++)
              umma_i8(d, da + (uint64_t)(2 * j), db + (uint64_t)(2 * j), idesc, (c > 0 || tap > 0 || j > 0) ? 1u : 0u);
            db += w_step;
          }
          umma_commit(&box_empty[st]);
          if (++st == g.n_boxes) { st = 0; lap++; }
        }
        if (ok) umma_commit(&t_full[acc]);
      }
    }
  } else {
    // ------------------------------ epilogue -----------------------------------------------------
    const int et = tid - 64, grp = (warp - 2) >> 2;
    const Epilogue &e = g.epi;
    pdl_wait();                            // the output buffer may still be read by the previous kernel
    stage_channel_params<MODE>(e, n0, ncols, par_k, par_l, et, 128 * H_GROUPS);
    asm volatile("bar.sync 1, %0;" ::"n"(128 * H_GROUPS) : "memory");
    // a group takes every n_acc-th tile, always in the same accumulator; with fewer accumulators than groups the groups
    // of a tile take its 32-column chunks in turn
    const int quad = warp & 3, r = quad * 32 + lane;
    const int acc = grp % g.n_acc, share = grp / g.n_acc, shares = H_GROUPS / g.n_acc;
    const uint32_t t_row = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(acc * g.acc_cols);
    int i = acc;
    for (int mt = m0 + acc * m_step; mt < g.m_tiles; mt += g.n_acc * m_step, i += g.n_acc) {
      if (!mbar_wait(&t_full[acc], (uint32_t)(i / g.n_acc) & 1u, abort_flag, g.status, ST_H_EPI)) break;
      __syncwarp();                        // tensor-memory loads need whole warps
      tc_fence_after();
      int b, y, x;
      patch(mt, b, y, x);
      y += r >> 3;
      x += r & 7;
      const bool store = y < g.Ho && x < g.Wo;
      uint8_t *out = g.out + (((size_t)b * g.Ho + (store ? y : 0)) * g.Wo + (store ? x : 0)) * g.N + n0;
      for (int c0 = share * 32; c0 < ncols; c0 += 32 * shares) {
        uint32_t v[32];
        tmem_ld_32(t_row + (uint32_t)c0, v);
        tmem_wait_ld();
        unsigned w[8];
        requant32_cols<MODE>(v, c0, ncols, par_k, par_l, e, g.K, w);
        if (store) {
          // whole 32-byte sectors of a pixel where the channel count allows
          uint8_t *o = out + c0;
          if (g.wide_store)
            asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                         ::"l"(o), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7]) : "memory");
          else {
            *reinterpret_cast<uint4 *>(o) = make_uint4(w[0], w[1], w[2], w[3]);
            if (c0 + 16 < ncols) *reinterpret_cast<uint4 *>(o + 16) = make_uint4(w[4], w[5], w[6], w[7]);
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&t_empty[acc]);
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem, (uint32_t)(g.n_acc * g.acc_cols));
  }
}

constexpr int HALO_SMEM = 220 * 1024;

template <int MODE, int BKB>
bool launch_halo(Context &c, const CUtensorMap &a, const CUtensorMap &w, const HaloParams &g, int grid, int smem)
{
  auto kern = conv_halo_tc_kernel<MODE, BKB>;
  static PerDeviceInt attr_set;
  if (!attr_set.get(c.device)) {
    if (!cuda_ok(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, HALO_SMEM), "cudaFuncSetAttribute(conv_halo_tc)"))
      return false;
    attr_set.set(c.device, 1);
  }
  const cudaError_t le = launch_pdl(kern, dim3((unsigned)grid), dim3(HTHREADS), (size_t)smem, c.stream, a, w, g);
  count_launch("conv_halo_tc_kernel");
  return cuda_ok(le, "conv_halo_tc launch") && cuda_ok(cudaGetLastError(), "conv_halo_tc launch");
}

template <int MODE>
bool launch_halo_bk(Context &c, const CUtensorMap &a, const CUtensorMap &w, const HaloParams &g, int bkb, int grid, int smem)
{
  if (bkb == 32) return launch_halo<MODE, 32>(c, a, w, g, grid, smem);
  if (bkb == 64) return launch_halo<MODE, 64>(c, a, w, g, grid, smem);
  return launch_halo<MODE, 128>(c, a, w, g, grid, smem);
}

// Lays the problem out and returns the estimated ns, -1 where it does not fit. The channels are cut into the tiles with
// the least estimated time: an MMA takes 80 cycles or BN / 2, whichever is more, a row of a TMA box some 12, the CTA's
// slice of W 80 bytes per ns, and the tiles come in rounds of as many as there are SMs. Cutting the channels multiplies
// the MMAs that narrow tiles leave half idle: beyond twice those of one tile, and more than two rounds, igemm_tc.cu is
// faster (-1 as well: 14x14x256 -> 256 at batch 64, four tiles of 64: 17.8 us against 12.9; 28x28x224 -> 224 at batch 16
// 19.9 / 18.3; 28x28x160 -> 160 at batch 32 18.8 / 19.1; in one or two rounds 14x14x256 at batch 32 10.8 / 12.3, at
// batch 8 6.6 / 10.4).
double plan_halo(const ConvProblem &p, int sms, HaloParams &g, int &bkb, int &smem)
{
  if (p.sx < 1 || p.sx > 2 || p.sy < 1 || p.sy > 2 || p.ky * p.kx < 2 || p.kx > 9 || p.ky > 9 || p.Cin % 32 != 0 || p.Cout % 16 != 0)
    return -1;
  if (p.epi.mode == EPI_RAW32) return -1;
  if ((reinterpret_cast<uintptr_t>(p.in) | reinterpret_cast<uintptr_t>(p.w) | reinterpret_cast<uintptr_t>(p.out)) & 15) return -1;
  bkb = p.Cin % 128 == 0 ? 128 : (p.Cin % 64 == 0 ? 64 : 32);
  g.epi = p.epi; g.out = static_cast<uint8_t *>(p.out);
  g.N = p.Cout; g.K = p.ky * p.kx * p.Cin; g.Ho = p.Ho; g.Wo = p.Wo; g.pt = p.pt; g.pl = p.pl; g.ky = p.ky; g.kx = p.kx;
  g.chunks = p.Cin / bkb;
  g.sx = p.sx; g.sy = p.sy;
  g.box_w = HTW + (p.kx - 1) / p.sx; g.box_h = HTH + (p.ky - 1) / p.sy;
  g.box_bytes = g.box_w * g.box_h * bkb;
  g.box_pitch = (g.box_bytes + 1023) & ~1023;
  g.box_stride = p.sx * p.sy * g.box_pitch;
  g.tiles_x = (p.Wo + HTW - 1) / HTW; g.tiles_y = (p.Ho + HTH - 1) / HTH;
  const long long m_tiles = (long long)p.B * g.tiles_x * g.tiles_y;
  if (m_tiles > 0x7fffffffLL) return -1;
  g.m_tiles = (int)m_tiles;
  double best = -1;
  for (int nt = (p.Cout + 255) / 256;; nt++) {
    const int bn = ((p.Cout + nt - 1) / nt + 15) & ~15, n_tiles = (p.Cout + bn - 1) / bn;
    // (with more channel tiles than SMs not even the first candidate has a round)
    if (n_tiles > sms || (nt > (p.Cout + 255) / 256 && bn < 32)) break;
    const long long fixed = (long long)g.K * bn + 1024;
    const long long boxes = (HALO_SMEM - fixed) / g.box_stride;
    if (fixed >= HALO_SMEM || boxes < 2) continue;
    const long long rounds = (m_tiles + sms / n_tiles - 1) / (sms / n_tiles);
    const double wide = bn > 160 ? bn / 2.0 : 80.0, one = p.Cout > 160 ? p.Cout / 2.0 : 80.0;
    if (rounds > 2 && n_tiles * wide > 2.0 * one) continue;
    const double mma = p.ky * p.kx * (p.Cin / 32) * wide + 400, tma = 12.0 * g.chunks * p.sx * p.sy * g.box_w * g.box_h;
    const double t = (double)rounds * (mma > tma ? mma : tma) / 1.9 + (double)g.K * bn / 80;
    if (best >= 0 && t >= best) continue;
    best = t;
    g.bn = bn; g.n_tiles = n_tiles;
    g.n_boxes = (int)(boxes < MAX_BOXES ? boxes : MAX_BOXES);
    smem = (int)(fixed + (long long)g.n_boxes * g.box_stride);
  }
  if (best < 0) return -1;
  g.acc_cols = 32;
  while (g.acc_cols < g.bn) g.acc_cols *= 2;
  g.n_acc = 512 / g.acc_cols < MAX_ACC ? 512 / g.acc_cols : MAX_ACC;
  g.wide_store = p.Cout % 32 == 0 && g.bn % 32 == 0 && (reinterpret_cast<uintptr_t>(p.out) & 31) == 0;
  // What the cut takes, to be compared with other kernels' estimates: fitted to 188 calls of 3 to 80 us over odd image
  // sizes, strides and kernels (standard deviation 9 %). The start of a chunk and of a tile cost the MMA thread some 480
  // and 930 cycles, a row of a box 2.3 to 3.9 in the long run.
  const double rounds = (double)((m_tiles + sms / g.n_tiles - 1) / (sms / g.n_tiles));
  const double mma = 0.94 * p.ky * p.kx * (p.Cin / 32) * (g.bn > 160 ? g.bn / 2.0 : 80.0) + 480.0 * g.chunks + 930;
  const double rows = (bkb == 128 ? 3.9 : (bkb == 64 ? 3.05 : 2.3)) * g.chunks * p.sx * p.sy * g.box_w * g.box_h;
  return 2470 + rounds * (mma > rows ? mma : rows) / 1.9 + (double)g.K * g.bn / 46;
}

}  // namespace

double conv_halo_tc_estimate(const Context &c, const ConvProblem &p)
{
  HaloParams g = {};
  int bkb, smem;
  const double ns = plan_halo(p, c.sm_count > 0 ? c.sm_count : 148, g, bkb, smem);
  return encode_tiled_fn() ? ns : -1;
}

bool launch_conv_halo_tc(Context &c, const ConvProblem &p)
{
  HaloParams g = {};
  int bkb = 128, smem = 0;
  const int sms = c.sm_count > 0 ? c.sm_count : 148;
  if (plan_halo(p, sms, g, bkb, smem) < 0) return false;
  g.const_weights = p.folded != nullptr;
  g.by_tx.set((unsigned)g.tiles_x);
  g.by_ty.set((unsigned)g.tiles_y);
  if (!ctx_status_word_unless_capturing(c, &g.status)) return false;
  CUtensorMap a, w;
  if (!make_map_4d(&a, p.in, p.Cin, p.W, p.H, p.B, bkb, g.box_w, g.box_h, p.sx, p.sy)) return false;
  if (!make_map(&w, p.w, p.Cout, g.K, g.bn, bkb)) return false;
  const int per = sms / g.n_tiles;
  const int grid = g.n_tiles * (per < g.m_tiles ? per : g.m_tiles);
  switch (p.epi.mode) {
    case EPI_NONE: return launch_halo_bk<EPI_NONE>(c, a, w, g, bkb, grid, smem);
    case EPI_MULT: return launch_halo_bk<EPI_MULT>(c, a, w, g, bkb, grid, smem);
    case EPI_BN32: return launch_halo_bk<EPI_BN32>(c, a, w, g, bkb, grid, smem);
    default:       return launch_halo_bk<EPI_BN64>(c, a, w, g, bkb, grid, smem);
  }
}

}  // namespace pulpnn
