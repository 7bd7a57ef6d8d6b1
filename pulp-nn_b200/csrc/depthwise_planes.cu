// depthwise_planes.cu -- 3x3 and 5x5 depthwise convolution, stride 1 or 2, of ANY channel count, row
// length and alignment, from HWC or CHW input (arithmetic of 32bit/src/pulp_nn_depthwise_generic.c:133-180).
//
// A CTA takes one image, a group of 32 (16) channels and a band of output rows, cut into strips of columns
// where bands alone are too large or too few. It stages the input rows of the band in shared memory as one
// PLANE per channel, [channel][row][x - first column it reads], zeros outside the image: HWC input through 4x4 byte transposes (four pixels x four channels), CHW input as it lies.
// A lane is a channel, so a warp stores runs of 32 bytes of the HWC output and an odd pitch in words
// keeps the lanes on different banks. A lane computes four adjacent output columns of R rows: their
// windows lie in two (stride 1) or three (stride 2) aligned words of a plane row, and a filter row costs
// one or two dp4a per output against copies of its taps shifted to the byte the window starts at -- no
// unpacking and no funnel shifts. Each plane row is read once for the R rows it feeds.
//
// What bounds it: instruction issue -- a warp of 3x3 outputs costs some 12 instructions in the dp4a and
// the requantised byte stores and about as many again to stage its share of the input, halo included (64 % of
// the issue slots taken on 70x70x187). So a filter row is expanded once per CTA and not per warp, offsets are
// 32 bits, and pixels that lie across words are two word loads and a funnel shift. Measured (us, graph replay;
// the kernels it replaces / now): 28x28x120 5x5 HWC at batch 32 39.3 / 8.8, the same from CHW 97.8 / 9.9,
// 14x14x475 5x5 stride 2 at batch 20 15.9 / 5.6, 56x56x61 3x3 at batch 8 25.5 / 4.7, 30x30x64 3x3 CHW at batch
// 64 70.9 / 8.4, 70x70x187 3x3 at batch 32 458 / 33.7.
#include "internal.cuh"
#include "unaligned16.cuh"

namespace pulpnn {

namespace {

constexpr int DT = 256;
constexpr int PLANES_BAND = 48 * 1024;       // planes of a CTA: four CTAs share an SM
constexpr int PLANES_SMEM = PLANES_BAND + 5 * 4 * 2 * 32 * 4;      // and its expanded filter rows

struct PlanesParams {
  DepthwiseProblem p;
  int groups, bands, band;      // channel groups, bands of `band` output rows (a multiple of R)
  int rows_in, row_pitch;       // staged rows, bytes of a plane row
  int plane;                    // bytes of a plane, an odd number of words
  int words;                    // HWC: channels in whole aligned words
  int quads;                    // groups of four output columns
  int strips, sq;               // strips of sq such groups
  FastDiv by_groups, by_bands, by_strips;
  FastDiv by_qw, by_per, by_sq; // words (CHW: 16-byte pieces) of a plane row, of a plane; sq
};

__device__ __forceinline__ unsigned prmt_b(unsigned a, unsigned b, unsigned sel)
{
  unsigned d;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(sel));
  return d;
}

// STRIPS: more than one strip (as a branch of its own the check of the last strip's groups costs the 5x5 layers of one
// strip 2.5 %)
template <int MODE, int K, int S, int CG, bool STRIPS>
__global__ void __launch_bounds__(DT) depthwise_planes_kernel(const __grid_constant__ PlanesParams g)
{
  constexpr int R = S == 1 ? 4 : 2;                         // output rows of a lane
  constexpr int NW = ((3 * S + K - 1) >> 2) + 1;            // plane words its four columns touch
  constexpr int NV = 4 / S;                                 // window starts modulo a word
  extern __shared__ __align__(16) uint8_t planes[];
  const DepthwiseProblem &p = g.p;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int t0 = g.by_groups.div((int)blockIdx.x), grp = (int)blockIdx.x - t0 * g.groups;
  const int t1 = STRIPS ? g.by_strips.div(t0) : t0, xq0 = STRIPS ? (t0 - t1 * g.strips) * g.sq : 0;
  const int b = g.by_bands.div(t1), band = t1 - b * g.bands;
  const int c0 = grp * CG, nch = min(CG, p.C - c0);
  const int oy0 = band * g.band;
  const int iy0 = oy0 * S - p.pt, ix0 = (STRIPS ? 4 * S * xq0 : 0) - p.pl;
  const int qw = g.row_pitch >> 2;                          // words of a plane row

  pdl_wait();
  pdl_launch_dependents();

  // what the compute phase needs of the parameters is on its way while the rows are staged: a filter row of one
  // channel per thread, the lane's channel's requantisation
  const Epilogue &e = p.epi;
  const int cl = lane % CG, sub = lane / CG;
  const int c = c0 + min(cl, nch - 1);
  long long kk = 0, ll = 0;
  if (MODE == EPI_BN32) {
    kk = __ldg(reinterpret_cast<const int *>(e.k) + c);
    ll = __ldg(reinterpret_cast<const int *>(e.lambda) + c);
  } else if (MODE == EPI_BN64) {
    kk = __ldg(reinterpret_cast<const long long *>(e.k) + c);
    ll = __ldg(reinterpret_cast<const long long *>(e.lambda) + c);
  }
  const int bias = e.bias ? (int)__ldg(reinterpret_cast<const int8_t *>(e.bias) + c) : 0;
  static_assert(K * CG <= DT, "a filter row per thread");
  const int wc = tid % CG, wfy = tid / CG;
  unsigned taps[K];
#pragma unroll
  for (int fx = 0; fx < K; fx++)
    taps[fx] = wfy < K && wc < nch ? (unsigned)(uint8_t)__ldg(p.w + ((size_t)(c0 + wc) * K + wfy) * K + fx) : 0u;

  // ---- stage the planes -----------------------------------------------------------------------
  if (p.in_is_hwc) {
    constexpr int CQ = CG / 4;
    // 32-bit offsets into the image from the word at or below its first byte
    const int own = p.H * p.W * p.C;
    const size_t off = (size_t)b * own;
    const int lead = (int)(reinterpret_cast<uintptr_t>(p.in + off) & 3);
    const uint8_t *img = p.in + off - lead;
    const ImageSpan span(lead, own, off, (size_t)(p.B - 1 - b) * own);
    const int items = g.rows_in * qw;                       // words of four pixels, the thread's four channels
    const int cq = tid % CQ, left = nch - 4 * cq;           // channels of this word that exist
    constexpr int STEP = DT / CQ;
    constexpr int U = 2;                                    // items of a thread in flight
    for (int it0 = tid / CQ; it0 < items; it0 += U * STEP) {
      unsigned v[U][4], v1[U][4];
      int dst[U], at[U];
#pragma unroll
      for (int u = 0; u < U; u++) {
        const int it = it0 + u * STEP;
        const int row = g.by_qw.div(it), q = it - row * qw;
        const int iy = iy0 + row, ix = ix0 + 4 * q;
        const bool ok = it < items && (unsigned)iy < (unsigned)p.H && left > 0;
        at[u] = (iy * p.W + ix) * p.C + c0 + 4 * cq + lead;
        dst[u] = it < items ? 4 * cq * g.plane + row * g.row_pitch + 4 * q : -1;
        if (g.words) {
#pragma unroll
          for (int i = 0; i < 4; i++) v[u][i] = ldg4_if(img + at[u] + i * p.C, ok && (unsigned)(ix + i) < (unsigned)p.W);
        } else if (!ok || span.holds_words(at[u], p.C)) {
#pragma unroll
          for (int i = 0; i < 4; i++) {
            const bool in = ok && (unsigned)(ix + i) < (unsigned)p.W;
            const uint8_t *w = img + ((at[u] + i * p.C) & ~3);
            v[u][i] = ldg4_if(w, in);
            v1[u][i] = ldg4_if(w + 4, in);
          }
        } else {
          // the ends of the tensor: byte by byte, put where the shift takes them
#pragma unroll
          for (int i = 0; i < 4; i++) {
            const int o = at[u] + i * p.C;
            const bool in = (unsigned)(ix + i) < (unsigned)p.W;
            unsigned x = 0;
#pragma unroll
            for (int k = 0; k < 4; k++) x |= ldg1_if(img + o + k, in && k < left) << (8 * k);
            const unsigned sh = (unsigned)(o & 3) * 8;
            v[u][i] = x << sh;
            v1[u][i] = sh ? x >> (32 - sh) : 0;
          }
        }
      }
      if (!g.words) {
#pragma unroll
        for (int u = 0; u < U; u++)
#pragma unroll
          for (int i = 0; i < 4; i++) v[u][i] = __funnelshift_r(v[u][i], v1[u][i], (unsigned)(at[u] + i * p.C) * 8);
      }
#pragma unroll
      for (int u = 0; u < U; u++) {
        if (dst[u] < 0) continue;
        const unsigned a = prmt_b(v[u][0], v[u][1], 0x5140), bb = prmt_b(v[u][0], v[u][1], 0x7362);
        const unsigned cc = prmt_b(v[u][2], v[u][3], 0x5140), d = prmt_b(v[u][2], v[u][3], 0x7362);
        uint8_t *to = planes + dst[u];
        *reinterpret_cast<unsigned *>(to) = prmt_b(a, cc, 0x5410);
        *reinterpret_cast<unsigned *>(to + g.plane) = prmt_b(a, cc, 0x7632);
        *reinterpret_cast<unsigned *>(to + 2 * g.plane) = prmt_b(bb, d, 0x5410);
        *reinterpret_cast<unsigned *>(to + 3 * g.plane) = prmt_b(bb, d, 0x7632);
      }
    }
  } else {
    // offsets from the group's first byte, with up to 64 bytes of the tensor on either side: a piece is read as two
    // aligned blocks of 16, which only at the very ends of the tensor are not its own
    const size_t off = ((size_t)b * p.C + c0) * p.H * p.W, all = (size_t)p.B * p.C * p.H * p.W;
    const int own = nch * p.H * p.W;
    const int before = (int)min(off, (size_t)64), after = (int)min(all - off - (size_t)own, (size_t)64);
    const Bytes in(p.in + off - before, before + own + after);
    const int first = in.start + before;
    const int pw = g.row_pitch >> 4, per = g.rows_in * pw, items = per * nch;   // 16-byte pieces
    constexpr int U = 2;
    for (int it0 = tid; it0 < items; it0 += U * DT) {
      Chunk t[U];
      int from[U], to[U], dst[U];                           // bytes [from, to) of the piece lie inside the image
#pragma unroll
      for (int u = 0; u < U; u++) {
        const int it = it0 + u * DT;
        const int ch = g.by_per.div(it), rq = it - ch * per;
        const int row = g.by_qw.div(rq), q = rq - row * pw;
        const int iy = iy0 + row, ix = ix0 + 16 * q;
        from[u] = max(-ix, 0);
        to[u] = it < items && (unsigned)iy < (unsigned)p.H && from[u] < 16 ? min(p.W - ix, 16) : 0;
        t[u].fetch(in, first + (ch * p.H + iy) * p.W + ix, to[u] > 0);
        dst[u] = it < items ? ch * g.plane + row * g.row_pitch + 16 * q : -1;
      }
#pragma unroll
      for (int u = 0; u < U; u++) {
        if (dst[u] < 0) continue;
        uint4 v = make_uint4(0, 0, 0, 0);
        if (to[u] > 0) {
          v = t[u].get(in);
          if (from[u] > 0 || to[u] < 16) mask16(v, from[u], to[u]);
        }
        unsigned *d = reinterpret_cast<unsigned *>(planes + dst[u]);
        d[0] = v.x; d[1] = v.y; d[2] = v.z; d[3] = v.w;
      }
    }
  }

  // ---- the filter rows shifted to every window start, [row][start][word][channel] ------------------
  unsigned *wsm = reinterpret_cast<unsigned *>(planes + CG * g.plane);
  if (wfy < K) {
    unsigned long long t = 0;
#pragma unroll
    for (int fx = 0; fx < K; fx++) t |= (unsigned long long)taps[fx] << (8 * fx);
#pragma unroll
    for (int v = 0; v < NV; v++) {
      wsm[((wfy * NV + v) * 2 + 0) * CG + wc] = (unsigned)(t << (8 * v * S));
      wsm[((wfy * NV + v) * 2 + 1) * CG + wc] = (unsigned)((t << (8 * v * S)) >> 32);
    }
  }
  const bool fits = MODE == EPI_BN64 && __all_sync(0xffffffffu, bn_fits_32(kk, ll, K * K * ACC_PER_TERM + 128, e.shift));
  __syncthreads();
  unsigned wv[K][NV][2];
#pragma unroll
  for (int fy = 0; fy < K; fy++)
#pragma unroll
    for (int v = 0; v < NV; v++) {
      wv[fy][v][0] = wsm[((fy * NV + v) * 2 + 0) * CG + cl];
      wv[fy][v][1] = wsm[((fy * NV + v) * 2 + 1) * CG + cl];
    }
  // the shifted value before it is cut to a byte
  auto scaled = [&](int a) {
    if (MODE == EPI_BN32 || fits) return (int)((unsigned)(int)kk * (unsigned)a + (unsigned)(int)ll) >> e.shift;
    if (MODE == EPI_BN64) return (int)((long long)((unsigned long long)kk * (unsigned long long)(long long)a + (unsigned long long)ll) >> e.shift);
    if (MODE == EPI_MULT) return (int)(short)((int)((unsigned)e.out_mult * (unsigned)a) >> e.shift);
    return a >> e.shift;
  };

  // ---- compute: a unit is four columns x R rows of the warp's channels ------------------------------
  const int rows = min(g.band, p.Ho - oy0);
  const int units = ((rows + R - 1) / R) * g.sq;
  const uint8_t *mine = planes + (size_t)cl * g.plane;
  uint8_t *out = p.out + (size_t)b * p.Ho * p.Wo * p.C;
  for (int u = warp * (32 / CG) + sub; u < units; u += (DT / 32) * (32 / CG)) {
    const int rb = g.by_sq.div(u), xq = u - rb * g.sq;
    int acc[R][4];
#pragma unroll
    for (int r = 0; r < R; r++)
#pragma unroll
      for (int i = 0; i < 4; i++) acc[r][i] = bias;
    const uint8_t *at = mine + (rb * R * S) * g.row_pitch + xq * 4 * S;
#pragma unroll
    for (int ir = 0; ir < S * (R - 1) + K; ir++) {
      unsigned w[NW];
#pragma unroll
      for (int j = 0; j < NW; j++) w[j] = *reinterpret_cast<const unsigned *>(at + ir * g.row_pitch + 4 * j);
#pragma unroll
      for (int r = 0; r < R; r++) {
        const int fy = ir - S * r;
        if (fy < 0 || fy >= K) continue;
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const int off = (i * S) & 3, j = (i * S) >> 2;
          acc[r][i] = dp4a_us(w[j], (int)wv[fy][off / S][0], acc[r][i]);
          if (off + K > 4) acc[r][i] = dp4a_us(w[j + 1 < NW ? j + 1 : j], (int)wv[fy][off / S][1], acc[r][i]);
        }
      }
    }
    const int oy = oy0 + rb * R, ox = (STRIPS ? xq0 + xq : xq) * 4;
    const bool whole = ox + 4 <= p.Wo;
    unsigned o = (unsigned)((oy * p.Wo + ox) * p.C + c);
#pragma unroll
    for (int r = 0; r < R; r++, o += (unsigned)(p.Wo * p.C)) {
      const unsigned w = pack4_sat_u8(scaled(acc[r][0]), scaled(acc[r][1]), scaled(acc[r][2]), scaled(acc[r][3]));
      if (cl >= nch || oy + r >= p.Ho || (STRIPS && ox >= p.Wo)) continue;
      out[o] = (uint8_t)w;
      if (whole) {
        out[o + p.C] = (uint8_t)(w >> 8);
        out[o + 2 * p.C] = (uint8_t)(w >> 16);
        out[o + 3 * p.C] = (uint8_t)(w >> 24);
      } else {
        if (ox + 1 < p.Wo) out[o + p.C] = (uint8_t)(w >> 8);
        if (ox + 2 < p.Wo) out[o + 2 * p.C] = (uint8_t)(w >> 16);
      }
    }
  }
}

template <int MODE, int K, int S, int CG, bool STRIPS>
bool launch_planes(Context &c, const PlanesParams &g, int smem)
{
  auto kern = depthwise_planes_kernel<MODE, K, S, CG, STRIPS>;
  static PerDeviceInt attr_set;
  if (!attr_set.get(c.device)) {
    if (!cuda_ok(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, PLANES_SMEM), "cudaFuncSetAttribute(depthwise_planes)"))
      return false;
    attr_set.set(c.device, 1);
  }
  const cudaError_t le = launch_pdl(kern, dim3((unsigned)(g.groups * g.strips * g.bands * g.p.B)), dim3(DT), (size_t)smem, c.stream, g);
  count_launch("depthwise_planes_kernel");
  return cuda_ok(le, "depthwise_planes launch") && cuda_ok(cudaGetLastError(), "depthwise_planes launch");
}

template <int MODE, int CG, bool STRIPS>
bool launch_planes_ks(Context &c, const PlanesParams &g, int smem)
{
  if (g.p.kx == 3) return g.p.sx == 1 ? launch_planes<MODE, 3, 1, CG, STRIPS>(c, g, smem) : launch_planes<MODE, 3, 2, CG, STRIPS>(c, g, smem);
  return g.p.sx == 1 ? launch_planes<MODE, 5, 1, CG, STRIPS>(c, g, smem) : launch_planes<MODE, 5, 2, CG, STRIPS>(c, g, smem);
}

template <int MODE>
bool launch_planes_mode(Context &c, const PlanesParams &g, int cg, int smem)
{
  if (g.strips > 1) return cg == 16 ? launch_planes_ks<MODE, 16, true>(c, g, smem) : launch_planes_ks<MODE, 32, true>(c, g, smem);
  return cg == 16 ? launch_planes_ks<MODE, 16, false>(c, g, smem) : launch_planes_ks<MODE, 32, false>(c, g, smem);
}

// lays the work out; false when the offsets or the grid are too large
bool configure(const DepthwiseProblem &p, int sms, PlanesParams &g, int &cg, int &smem)
{
  const int S = p.sx, K = p.kx, R = S == 1 ? 4 : 2;
  g.p = p;
  cg = p.C <= 16 ? 16 : 32;
  g.groups = (p.C + cg - 1) / cg;
  g.quads = (p.Wo + 3) / 4;
  g.words = p.C % 4 == 0 && (reinterpret_cast<uintptr_t>(p.in) & 3) == 0;
  auto pitch_of = [&](int sq) {
    const long long pitch = (long long)(sq - 1) * 4 * S + 4 * (((3 * S + K - 1) >> 2) + 1);
    return p.in_is_hwc ? pitch : (pitch + 15) & ~15LL;      // CHW rows are staged in 16-byte pieces
  };
  auto plane_of = [&](int band, int sq) {
    const long long w = ((long long)(band - 1) * S + K) * (pitch_of(sq) / 4);
    return (w | 1) * 4;
  };
  // whole images while they fit, shorter bands until the GPU is full
  const int rb = (p.Ho + R - 1) / R;
  int blocks = rb;
  while (blocks > 1 && (plane_of(blocks * R, g.quads) * cg > PLANES_BAND || (long long)p.B * g.groups * ((rb + blocks - 1) / blocks) < 2LL * sms))
    blocks = (blocks + 1) / 2;
  g.band = blocks * R;
  g.bands = (p.Ho + g.band - 1) / g.band;
  // Strips of no fewer than 32 columns where bands of R rows are still too large, or too few for the GPU: one row of 1038
  // pixels of 154 channels was staged and computed by five CTAs, in 23.7 us against 3.1 in strips.
  const long long ctas = (long long)p.B * g.groups * g.bands;
  long long n = ctas < 2LL * sms ? (2LL * sms + ctas - 1) / ctas : 1;
  if (n > (g.quads + 7) / 8) n = (g.quads + 7) / 8;
  g.sq = (int)((g.quads + n - 1) / n);
  while (g.sq > 8 && plane_of(g.band, g.sq) * cg > PLANES_BAND) g.sq = (g.sq + 1) / 2;
  g.strips = (g.quads + g.sq - 1) / g.sq;
  const int filters = K * (4 / S) * 2 * cg * 4;
  if (plane_of(g.band, g.sq) * cg + filters > PLANES_SMEM) return false;
  // 32-bit offsets inside a group of channels, the rows above and below its image included
  if (((long long)cg * p.H + p.pt + g.band * S + K) * p.W > 0x7fff0000LL) return false;
  if ((long long)p.Ho * p.Wo * p.C > 0x7fff0000LL || ((long long)p.H + p.pt + g.band * S + K) * p.W * p.C > 0x7fff0000LL) return false;
  if (ctas * g.strips > 0x7fffffffLL) return false;
  g.row_pitch = (int)pitch_of(g.sq);
  g.rows_in = (g.band - 1) * S + K;
  g.plane = (int)plane_of(g.band, g.sq);
  smem = g.plane * cg + filters;
  g.by_groups.set((unsigned)g.groups);
  g.by_bands.set((unsigned)g.bands);
  g.by_strips.set((unsigned)g.strips);
  const int piece = p.in_is_hwc ? 4 : 16;
  g.by_qw.set((unsigned)(g.row_pitch / piece));
  g.by_per.set((unsigned)(g.rows_in * (g.row_pitch / piece)));
  g.by_sq.set((unsigned)g.sq);
  return true;
}

}  // namespace

bool depthwise_planes_supported(const DepthwiseProblem &p)
{
  if (p.kx != p.ky || (p.kx != 3 && p.kx != 5) || p.sx != p.sy || (p.sx != 1 && p.sx != 2)) return false;
  PlanesParams g = {};
  int cg, smem;
  return configure(p, 148, g, cg, smem);
}

bool launch_depthwise_planes(Context &c, const DepthwiseProblem &p)
{
  PlanesParams g = {};
  int cg, smem;
  if (!configure(p, c.sm_count > 0 ? c.sm_count : 148, g, cg, smem)) return false;
  switch (p.epi.mode) {
    case EPI_NONE: return launch_planes_mode<EPI_NONE>(c, g, cg, smem);
    case EPI_MULT: return launch_planes_mode<EPI_MULT>(c, g, cg, smem);
    case EPI_BN32: return launch_planes_mode<EPI_BN32>(c, g, cg, smem);
    default:       return launch_planes_mode<EPI_BN64>(c, g, cg, smem);
  }
}

}  // namespace pulpnn
