// pool_add.cu -- max pooling, average pooling and the residual add. All three are one pass over
// the input and one over the output; threads are laid out along the channel axis (HWC), four
// channels (one 32-bit word) per thread where the channel count allows, sixteen for the add.
#include "internal.cuh"
#include "unaligned16.cuh"

namespace pulpnn {

namespace {

__device__ __forceinline__ unsigned ld_bytes(const uint8_t *p, int n)
{
  unsigned v = 0;
  for (int j = 0; j < n; j++) v |= (unsigned)__ldg(p + j) << (8 * j);
  return v;
}
__device__ __forceinline__ void st_bytes(uint8_t *p, unsigned v, int n)
{
  for (int j = 0; j < n; j++) p[j] = (uint8_t)(v >> (8 * j));
}

// ---- max pooling ---------------------------------------------------------------------------
// The reference pools along x in place and then along y (32bit/src/pulp_nn_maxpool.c:58-144);
// with stride_x > padding_l (checked on the host) that equals the maximum over the window
// clipped to the image: rows [max(0, oy*sy - pt), min(oy*sy - pt + ky, H)), columns likewise
// with padding_l. padding_b / padding_r are never read by the reference.
template <bool VEC>
__global__ void __launch_bounds__(256) maxpool_kernel(const PoolProblem p, int CW, long long total)
{
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= total) return;
  const int cw = (int)(t % CW);
  long long r = t / CW;
  const int ox = (int)(r % p.Wo); r /= p.Wo;
  const int oy = (int)(r % p.Ho);
  const int b = (int)(r / p.Ho);
  const int c = VEC ? cw * 4 : cw, nb = VEC ? 4 : 1;
  const int y0 = max(oy * p.sy - p.pt, 0), y1 = min(oy * p.sy - p.pt + p.ky, p.H);
  const int x0 = max(ox * p.sx - p.pl, 0), x1 = min(ox * p.sx - p.pl + p.kx, p.W);
  const uint8_t *img = p.in + (size_t)b * p.H * p.W * p.C + c;
  unsigned m = 0;
  for (int y = y0; y < y1; y++)
    for (int x = x0; x < x1; x++) {
      const uint8_t *q = img + ((size_t)y * p.W + x) * p.C;
      const unsigned v = VEC ? __ldg(reinterpret_cast<const unsigned *>(q)) : ld_bytes(q, nb);
      m = __vmaxu4(m, v);
    }
  uint8_t *o = p.out + (((size_t)b * p.Ho + oy) * p.Wo + ox) * p.C + c;
  if (VEC) *reinterpret_cast<unsigned *>(o) = m; else st_bytes(o, m, nb);
}

// Reproduces what the reference leaves in Im_in: after its x pass, column ox of every input row
// holds the maximum over that row's window for output column ox (pulp_nn_maxpool.c:63,85-92).
// Reads the untouched input copy `src` and writes into `dst` (the caller's Im_in).
__global__ void __launch_bounds__(256) maxpool_clobber_kernel(const PoolProblem p, const uint8_t *src,
                                                              uint8_t *dst, long long total)
{
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= total) return;
  const int c = (int)(t % p.C);
  long long r = t / p.C;
  const int ox = (int)(r % p.Wo); r /= p.Wo;
  const int y = (int)(r % p.H);
  const int b = (int)(r / p.H);
  const int x0 = max(ox * p.sx - p.pl, 0), x1 = min(ox * p.sx - p.pl + p.kx, p.W);
  const uint8_t *row = src + (((size_t)b * p.H + y) * p.W) * p.C + c;
  int m = 0;
  for (int x = x0; x < x1; x++) m = max(m, (int)__ldg(row + (size_t)x * p.C));
  dst[(((size_t)b * p.H + y) * p.W + ox) * p.C + c] = (uint8_t)m;
}

// ---- average pooling -----------------------------------------------------------------------
// 32bit/src/pulp_nn_avgpool.c:71-119. Window start in y uses padding_b and window end in x uses
// padding_r, as written there; the divisor is always kx*ky. The requantised form is unsigned
// 32-bit arithmetic in the 32-bit tree and signed 64-bit arithmetic in the 64-bit tree.
template <bool VEC>
__global__ void __launch_bounds__(256) avgpool_kernel(const PoolProblem p, int CW, long long total)
{
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= total) return;
  const int cw = (int)(t % CW);
  long long r = t / CW;
  const int ox = (int)(r % p.Wo); r /= p.Wo;
  const int oy = (int)(r % p.Ho);
  const int b = (int)(r / p.Ho);
  const int c = VEC ? cw * 4 : cw, nb = VEC ? 4 : 1;
  const int y0 = max(oy * p.sy - p.pb, 0), y1 = min(oy * p.sy - p.pt + p.ky, p.H);
  const int x0 = max(ox * p.sx - p.pl, 0), x1 = min(ox * p.sx - p.pr + p.kx, p.W);
  const uint8_t *img = p.in + (size_t)b * p.H * p.W * p.C + c;
  unsigned s[4] = {0, 0, 0, 0};
  for (int y = y0; y < y1; y++)
    for (int x = x0; x < x1; x++) {
      const uint8_t *q = img + ((size_t)y * p.W + x) * p.C;
      const unsigned v = VEC ? __ldg(reinterpret_cast<const unsigned *>(q)) : ld_bytes(q, nb);
      s[0] += v & 0xff; s[1] += (v >> 8) & 0xff; s[2] += (v >> 16) & 0xff; s[3] += v >> 24;
    }
  const unsigned ktot = (unsigned)(p.kx * p.ky);
  unsigned o = 0;
  for (int j = 0; j < nb; j++) {
    int res;
    if (p.requant) {
      if (p.bn_bits == 32) {
        const unsigned tq = s[j] * (unsigned)(int)p.lambda / ktot + (unsigned)(int)p.out_add;
        res = (int)(tq >> p.shift);
      } else {
        const long long tq = (long long)s[j] * p.lambda / (long long)ktot + p.out_add;
        res = (int)(tq >> p.shift);
      }
    } else {
      res = (int)(s[j] / ktot);
    }
    o |= (unsigned)clip_u8(res) << (8 * j);
  }
  uint8_t *dst = p.out + (((size_t)b * p.Ho + oy) * p.Wo + ox) * p.C + c;
  if (VEC) *reinterpret_cast<unsigned *>(dst) = o; else st_bytes(dst, o, nb);
}

// ---- both, at any channel count ---------------------------------------------------------------
// One thread takes VB adjacent channels of one output pixel: 16 (one aligned load per window pixel) where
// channel count and alignment allow, else 4, from one aligned word or (UNAL) from the two words it lies
// across. All loads of a 2x2 or 3x3 window are in flight at once (K = 2, 3; K = 0: any window, eight at
// a time). Bytes are compared as 16-bit pairs: the high byte of a pair decides its maximum
// whatever the low byte holds, so v and v & 0x00ff00ff give all four for three instructions a word, where
// a byte-wise maximum takes three times that; sums (at most 257 pixels) are 16-bit pairs as well.
// Index arithmetic is 32 bits with multiplications for divisions. Measured (us, graph replay, before / after):
// max 3x3 stride 2 of 112x112x64 at batch 32 13.8 / 7.5 (32 MB: 4.3 TB/s), of 17x17x429 at batch 64 32.4 / 10.8, of
// 56x56x64 at batch 1 3.1 / 1.9; average 3x3 stride 2 of 56x56x64 at batch 64 15.1 / 6.4.
struct PoolParams {
  PoolProblem p;
  FastDiv by_cw, by_wo, by_ho, by_taps;
  int cw;                  // groups of VB channels per pixel
  int total;               // threads
};

__device__ __forceinline__ unsigned max_u16x2(unsigned a, unsigned b)
{
  unsigned d;
  asm("max.u16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}

template <bool AVG>
__device__ __forceinline__ void pool_word(unsigned v, unsigned &lo, unsigned &hi)
{
  if (AVG) { lo += v & 0x00ff00ffu; hi += (v >> 8) & 0x00ff00ffu; }
  else     { lo = max_u16x2(lo, v & 0x00ff00ffu); hi = max_u16x2(hi, v); }
}

__device__ __forceinline__ int pool_mean(unsigned s, const PoolParams &g)
{
  const PoolProblem &p = g.p;
  if (!p.requant) return g.by_taps.div((int)s);
  const unsigned ktot = (unsigned)(p.kx * p.ky);
  if (p.bn_bits == 32) return (int)((s * (unsigned)(int)p.lambda / ktot + (unsigned)(int)p.out_add) >> p.shift);
  return (int)(((long long)s * p.lambda / (long long)ktot + p.out_add) >> p.shift);
}

template <int VB, bool UNAL, bool AVG, int K>
__global__ void __launch_bounds__(256) pool_kernel(const PoolParams g)
{
  constexpr int NW = VB / 4;
  pdl_wait();
  pdl_launch_dependents();
  const PoolProblem &p = g.p;
  const int t = (int)(blockIdx.x * 256u + threadIdx.x);
  if (t >= g.total) return;
  int r = g.by_cw.div(t);
  const int c = (t - r * g.cw) * VB;
  int q = g.by_wo.div(r);
  const int ox = r - q * p.Wo;
  const int b = g.by_ho.div(q), oy = q - b * p.Ho;
  // where the windows begin and end: see the kernels above
  const int yb = oy * p.sy - (AVG ? p.pb : p.pt), xb = ox * p.sx - p.pl;
  const int y1 = min(oy * p.sy - p.pt + p.ky, p.H), x1 = min(ox * p.sx - (AVG ? p.pr : p.pl) + p.kx, p.W);
  const uint8_t *img = p.in + (size_t)b * p.H * p.W * p.C + c;
  const uint8_t *end = p.in + (size_t)p.B * p.H * p.W * p.C;
  unsigned lo[NW], hi[NW];
#pragma unroll
  for (int i = 0; i < NW; i++) lo[i] = hi[i] = 0;

  struct Px { uint4 v; unsigned w1; const uint8_t *at; };
  auto load = [&](Px &x, int y, int xx, bool ok) {
    const uint8_t *s = img + ((size_t)(ok ? y : 0) * p.W + (ok ? xx : 0)) * p.C;
    if (VB == 16) x.v = ldg16_if(s, ok);
    else if (!UNAL) x.v.x = ldg4_if(s, ok);
    else {
      const uint8_t *w = reinterpret_cast<const uint8_t *>(reinterpret_cast<uintptr_t>(s) & ~(uintptr_t)3);
      const bool whole = ok && w >= p.in && w + 8 <= end;
      x.v.x = ldg4_if(w, whole);
      x.w1 = ldg4_if(w + 4, whole);
      x.at = s;
      if (ok && !whole) {                                  // the ends of the tensor
        unsigned v = 0;
        for (int k = 0; k < 4 && c + k < p.C; k++) v |= (unsigned)__ldg(s + k) << (8 * k);
        const unsigned sh = (unsigned)(reinterpret_cast<uintptr_t>(s) & 3) * 8;
        x.v.x = v << sh;
        x.w1 = sh ? v >> (32 - sh) : 0;
      }
    }
  };
  auto take = [&](const Px &x) {
    if (VB == 16) {
      pool_word<AVG>(x.v.x, lo[0], hi[0]); pool_word<AVG>(x.v.y, lo[1 % NW], hi[1 % NW]);
      pool_word<AVG>(x.v.z, lo[2 % NW], hi[2 % NW]); pool_word<AVG>(x.v.w, lo[3 % NW], hi[3 % NW]);
    } else if (!UNAL) pool_word<AVG>(x.v.x, lo[0], hi[0]);
    else pool_word<AVG>(__funnelshift_r(x.v.x, x.w1, (unsigned)(reinterpret_cast<uintptr_t>(x.at) & 3) * 8), lo[0], hi[0]);
  };
  if (K > 0) {
    Px px[K * K > 0 ? K * K : 1];
#pragma unroll
    for (int f = 0; f < K * K; f++) {
      const int y = yb + f / (K > 0 ? K : 1), xx = xb + f % (K > 0 ? K : 1);
      load(px[f], y, xx, y >= 0 && y < y1 && xx >= 0 && xx < x1);
    }
#pragma unroll
    for (int f = 0; f < K * K; f++) take(px[f]);
  } else {
    // the window's pixels as one sequence, eight loads in flight
    const int y0 = max(yb, 0), x0 = max(xb, 0);
    const int tot = x1 > x0 && y1 > y0 ? (x1 - x0) * (y1 - y0) : 0;
    int y = y0, xx = x0;
    for (int n = 0; n < tot; n += 8) {
      Px px[8];
#pragma unroll
      for (int i = 0; i < 8; i++) {
        load(px[i], y, xx, n + i < tot);
        if (++xx == x1) { xx = x0; y++; }
      }
#pragma unroll
      for (int i = 0; i < 8; i++) take(px[i]);
    }
  }

  unsigned o[NW];
#pragma unroll
  for (int i = 0; i < NW; i++) {
    if (AVG)
      o[i] = (unsigned)clip_u8(pool_mean(lo[i] & 0xffffu, g)) | ((unsigned)clip_u8(pool_mean(hi[i] & 0xffffu, g)) << 8) |
             ((unsigned)clip_u8(pool_mean(lo[i] >> 16, g)) << 16) | ((unsigned)clip_u8(pool_mean(hi[i] >> 16, g)) << 24);
    else o[i] = lo[i] | (hi[i] & 0xff00ff00u);
  }
  uint8_t *dst = p.out + (size_t)r * p.C + c;
  if (VB == 16) *reinterpret_cast<uint4 *>(dst) = make_uint4(o[0], o[1 % NW], o[2 % NW], o[3 % NW]);
  else if (!UNAL) *reinterpret_cast<unsigned *>(dst) = o[0];
  else {
#pragma unroll
    for (int k = 0; k < 4; k++)
      if (c + k < p.C) dst[k] = (uint8_t)(o[0] >> (8 * k));
  }
}

// the form of a pooling call: 16 aligned channels per thread, 4 aligned ones, 4 at any address. An average of 16 channels
// is 16 divisions one after the other, so while there are fewer than 256 such threads an SM, four channels each finish
// sooner (us, 16 channels / 4: 4x1 over 20x4x64 3.7 / 2.0, 1x1 stride 3 over 42x42x384 4.6 / 2.8; 2x2, 49392 threads of 16
// 5.0, of 4 6.3).
int pool_form(const PoolProblem &p, bool avg, int sms)
{
  const uintptr_t a = reinterpret_cast<uintptr_t>(p.in) | reinterpret_cast<uintptr_t>(p.out);
  const bool enough = !avg || (long long)p.B * p.Ho * p.Wo * (p.C / 16) >= 256LL * sms;
  return enough && p.C % 16 == 0 && (a & 15) == 0 ? 0 : (p.C % 4 == 0 && (a & 3) == 0 ? 1 : 2);
}
// 32-bit thread indices; an average's window of at most 257 pixels, so that its sums fit 16 bits
bool pool_fits(const PoolProblem &p, bool avg, int sms)
{
  const int vb = pool_form(p, avg, sms) == 0 ? 16 : 4;
  if ((long long)p.B * p.Ho * p.Wo * ((p.C + vb - 1) / vb) > 0x7fffff00LL) return false;
  return !avg || ((long long)(p.kx + max(p.pl - p.pr, 0)) * (p.ky + max(p.pb - p.pt, 0)) <= 257);
}

template <bool AVG>
bool launch_pool(Context &c, const PoolProblem &p)
{
  const int form = pool_form(p, AVG, c.sm_count), vb = form == 0 ? 16 : 4;
  const long long pixels = (long long)p.B * p.Ho * p.Wo, cw = (p.C + vb - 1) / vb;
  PoolParams g = {};
  g.p = p;
  g.cw = (int)cw;
  g.total = (int)(pixels * cw);
  g.by_cw.set((unsigned)cw); g.by_wo.set((unsigned)p.Wo); g.by_ho.set((unsigned)p.Ho); g.by_taps.set((unsigned)(p.kx * p.ky));
  const int k = p.kx == p.ky && (p.kx == 2 || p.kx == 3) && (!AVG || (p.pt == p.pb && p.pl == p.pr)) ? p.kx : 0;
  const dim3 grid((unsigned)((g.total + 255) / 256));
  auto go = [&](auto kern) { return launch_pdl(kern, grid, dim3(256), 0, c.stream, g); };
  cudaError_t le;
  if (form == 0)      le = k == 2 ? go(pool_kernel<16, false, AVG, 2>) : k == 3 ? go(pool_kernel<16, false, AVG, 3>) : go(pool_kernel<16, false, AVG, 0>);
  else if (form == 1) le = k == 2 ? go(pool_kernel<4, false, AVG, 2>) : k == 3 ? go(pool_kernel<4, false, AVG, 3>) : go(pool_kernel<4, false, AVG, 0>);
  else                le = k == 2 ? go(pool_kernel<4, true, AVG, 2>) : k == 3 ? go(pool_kernel<4, true, AVG, 3>) : go(pool_kernel<4, true, AVG, 0>);
  count_launch("pool_kernel");
  return cuda_ok(le, "pool launch");
}

// The same for 16 channels per thread (C a multiple of 16, 16-byte aligned tensors): 16-byte loads,
// four of them in flight, so that a window of many pixels (a global pool) keeps HBM busy.
__global__ void __launch_bounds__(256) avgpool16_kernel(const PoolProblem p, int CW, long long total)
{
  pdl_wait();
  pdl_launch_dependents();
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= total) return;
  const int cw = (int)(t % CW);
  long long r = t / CW;
  const int ox = (int)(r % p.Wo); r /= p.Wo;
  const int oy = (int)(r % p.Ho);
  const int b = (int)(r / p.Ho);
  const int c = cw * 16;
  const int y0 = max(oy * p.sy - p.pb, 0), y1 = min(oy * p.sy - p.pt + p.ky, p.H);
  const int x0 = max(ox * p.sx - p.pl, 0), x1 = min(ox * p.sx - p.pr + p.kx, p.W);
  const uint8_t *img = p.in + (size_t)b * p.H * p.W * p.C + c;
  unsigned s[16];
#pragma unroll
  for (int j = 0; j < 16; j++) s[j] = 0;
  auto add16 = [&](const uint4 &v) {
    const unsigned w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; i++) {
      s[4 * i + 0] += w[i] & 0xff; s[4 * i + 1] += (w[i] >> 8) & 0xff;
      s[4 * i + 2] += (w[i] >> 16) & 0xff; s[4 * i + 3] += w[i] >> 24;
    }
  };
  // the window's pixels in one sequence, eight loads in flight at a time
  const int tot = (x1 > x0 && y1 > y0) ? (x1 - x0) * (y1 - y0) : 0;
  int yy = y0, xx = x0;
  for (int n = 0; n < tot; n += 8) {
    uint4 v[8];
#pragma unroll
    for (int i = 0; i < 8; i++) {
      v[i] = make_uint4(0, 0, 0, 0);
      if (n + i < tot) {
        v[i] = __ldg(reinterpret_cast<const uint4 *>(img + ((size_t)yy * p.W + xx) * p.C));
        if (++xx == x1) { xx = x0; yy++; }
      }
    }
#pragma unroll
    for (int i = 0; i < 8; i++) add16(v[i]);
  }
  const unsigned ktot = (unsigned)(p.kx * p.ky);
  unsigned o[4] = {0, 0, 0, 0};
#pragma unroll
  for (int j = 0; j < 16; j++) {
    int res;
    if (p.requant) {
      if (p.bn_bits == 32) {
        const unsigned tq = s[j] * (unsigned)(int)p.lambda / ktot + (unsigned)(int)p.out_add;
        res = (int)(tq >> p.shift);
      } else {
        const long long tq = (long long)s[j] * p.lambda / (long long)ktot + p.out_add;
        res = (int)(tq >> p.shift);
      }
    } else {
      res = (int)(s[j] / ktot);
    }
    o[j >> 2] |= (unsigned)clip_u8(res) << (8 * (j & 3));
  }
  uint8_t *dst = p.out + (((size_t)b * p.Ho + oy) * p.Wo + ox) * p.C + c;
  *reinterpret_cast<uint4 *>(dst) = make_uint4(o[0], o[1], o[2], o[3]);
}

// Large windows (a global pool): one thread per window would leave most of the GPU idle and make
// every thread walk the whole window alone. Here a block takes one output pixel and 128 channels:
// lane = four channels (a warp reads 128 contiguous bytes of a pixel), the block's eight warps share
// out the window's pixels, and shared memory adds up the eight partial sums. Same arithmetic.
// (VEC: channel count and pointers in whole words, else byte by byte.)
template <bool VEC>
__global__ void __launch_bounds__(256) avgpool_window_kernel(const PoolProblem p, int chunks)
{
  __shared__ unsigned part[8][32][4];
  pdl_wait();
  pdl_launch_dependents();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned t = blockIdx.x;
  const int chunk = (int)(t % (unsigned)chunks); t /= (unsigned)chunks;
  const int ox = (int)(t % (unsigned)p.Wo); t /= (unsigned)p.Wo;
  const int oy = (int)(t % (unsigned)p.Ho);
  const int b = (int)(t / (unsigned)p.Ho);
  const int c = chunk * 128 + lane * 4;
  const bool on = c < p.C;
  const int y0 = max(oy * p.sy - p.pb, 0), y1 = min(oy * p.sy - p.pt + p.ky, p.H);
  const int x0 = max(ox * p.sx - p.pl, 0), x1 = min(ox * p.sx - p.pr + p.kx, p.W);
  const int wx = x1 - x0, tot = (wx > 0 && y1 > y0) ? wx * (y1 - y0) : 0;
  const uint8_t *img = p.in + (size_t)b * p.H * p.W * p.C + (on ? c : 0);
  unsigned s[4] = {0, 0, 0, 0};
  // a window as wide as the image (a global pool) is one contiguous run of pixels: no division
  const bool run = wx == p.W;
  for (int n = warp; n < tot; n += 32) {          // four loads in flight per thread
    unsigned v[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const int q = n + 8 * i;
      v[i] = 0;
      if (q < tot && on) {
        const size_t pix = run ? (size_t)y0 * p.W + q : (size_t)(y0 + q / wx) * p.W + x0 + q % wx;
        const uint8_t *at = img + pix * p.C;
        if (VEC) v[i] = __ldg(reinterpret_cast<const unsigned *>(at));
        else {
#pragma unroll
          for (int k = 0; k < 4; k++) v[i] |= ldg1_if(at + k, c + k < p.C) << (8 * k);
        }
      }
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
      s[0] += v[i] & 0xff; s[1] += (v[i] >> 8) & 0xff; s[2] += (v[i] >> 16) & 0xff; s[3] += v[i] >> 24;
    }
  }
#pragma unroll
  for (int j = 0; j < 4; j++) part[warp][lane][j] = s[j];
  __syncthreads();
  if (warp != 0 || !on) return;
#pragma unroll
  for (int w = 1; w < 8; w++)
#pragma unroll
    for (int j = 0; j < 4; j++) s[j] += part[w][lane][j];
  const unsigned ktot = (unsigned)(p.kx * p.ky);
  unsigned o = 0;
#pragma unroll
  for (int j = 0; j < 4; j++) {
    int res;
    if (p.requant) {
      if (p.bn_bits == 32) {
        const unsigned tq = s[j] * (unsigned)(int)p.lambda / ktot + (unsigned)(int)p.out_add;
        res = (int)(tq >> p.shift);
      } else {
        const long long tq = (long long)s[j] * p.lambda / (long long)ktot + p.out_add;
        res = (int)(tq >> p.shift);
      }
    } else {
      res = (int)(s[j] / ktot);
    }
    o |= (unsigned)clip_u8(res) << (8 * j);
  }
  uint8_t *dst = p.out + (((size_t)b * p.Ho + oy) * p.Wo + ox) * p.C + c;
  if (VEC) *reinterpret_cast<unsigned *>(dst) = o; else st_bytes(dst, o, min(4, p.C - c));
}

// ---- residual add --------------------------------------------------------------------------
// 32bit/src/pulp_nn_utils.c:47-60: uint32 sum of the two int16-scaled bytes, logical shift,
// cut to 16 bits, then clamp to 255.
__device__ __forceinline__ unsigned add_word(unsigned a, unsigned b, int m1, int m2, int d)
{
  unsigned o = 0;
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const unsigned t = (unsigned)((int)((a >> (8 * j)) & 0xff) * m1 + (int)((b >> (8 * j)) & 0xff) * m2);
    const unsigned x = (t >> d) & 0xffffu;
    o |= min(x, 255u) << (8 * j);
  }
  return o;
}

// n16 pieces of 16 bytes; the threads of the last block add what is left of n
__global__ void __launch_bounds__(256) add_kernel(const uint8_t *a, const uint8_t *b, uint8_t *out, size_t n16, size_t n,
                                                  int m1, int m2, int d)
{
  pdl_wait();
  pdl_launch_dependents();
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n16; i += stride) {
    const uint4 x = __ldg(reinterpret_cast<const uint4 *>(a) + i), y = __ldg(reinterpret_cast<const uint4 *>(b) + i);
    uint4 o;
    o.x = add_word(x.x, y.x, m1, m2, d); o.y = add_word(x.y, y.y, m1, m2, d);
    o.z = add_word(x.z, y.z, m1, m2, d); o.w = add_word(x.w, y.w, m1, m2, d);
    reinterpret_cast<uint4 *>(out)[i] = o;
  }
  for (size_t i = n16 * 16 + (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
    out[i] = (uint8_t)add_word(a[i], b[i], m1, m2, d);
}

}  // namespace

bool launch_maxpool(Context &c, const PoolProblem &p, uint8_t *clobber_in)
{
  if (!pool_fits(p, false, c.sm_count)) {
    // index arithmetic of more than 32 bits
    const bool vec = (p.C % 4 == 0) && ((reinterpret_cast<uintptr_t>(p.in) & 3) == 0) &&
                     ((reinterpret_cast<uintptr_t>(p.out) & 3) == 0);
    const int CW = vec ? p.C / 4 : p.C;
    const long long total = (long long)p.B * p.Ho * p.Wo * CW;
    const unsigned blocks = (unsigned)((total + 255) / 256);
    if (vec) maxpool_kernel<true><<<blocks, 256, 0, c.stream>>>(p, CW, total);
    else     maxpool_kernel<false><<<blocks, 256, 0, c.stream>>>(p, CW, total);
    count_launch("maxpool_kernel");
    if (!cuda_ok(cudaGetLastError(), "maxpool launch")) return false;
  } else if (!launch_pool<false>(c, p)) return false;
  if (clobber_in) {
    // the x-pass image must be computed from the untouched input: copy it aside first
    const size_t bytes = (size_t)p.B * p.H * p.W * p.C;
    void *copy = ctx_scratch(c, bytes);
    if (!copy) return false;
    if (!cuda_ok(cudaMemcpyAsync(copy, clobber_in, bytes, cudaMemcpyDeviceToDevice, c.stream), "D2D copy"))
      return false;
    const long long tot2 = (long long)p.B * p.H * p.Wo * p.C;
    maxpool_clobber_kernel<<<(unsigned)((tot2 + 255) / 256), 256, 0, c.stream>>>(
        p, static_cast<const uint8_t *>(copy), clobber_in, tot2);
    count_launch();
    if (!cuda_ok(cudaGetLastError(), "maxpool clobber launch")) return false;
  }
  return true;
}

bool launch_avgpool(Context &c, const PoolProblem &p)
{
  const bool vec = (p.C % 4 == 0) && ((reinterpret_cast<uintptr_t>(p.in) & 3) == 0) &&
                   ((reinterpret_cast<uintptr_t>(p.out) & 3) == 0);
  // windows of at least 32 pixels: a block per output pixel and 128 channels
  const int chunks = (p.C + 127) / 128;
  const long long blocks_w = (long long)p.B * p.Ho * p.Wo * chunks;
  const long long threads16 = (long long)p.B * p.Ho * p.Wo * (p.C / 16);
  const bool fills_gpu = p.C % 16 == 0 && threads16 >= 32768;      // measured: from batch 512 of a 7x7x1024 pool on
  // (byte by byte only while a block per window still has the GPU to itself: 7x7x333 at batch 64 3.6 us against 8.9 in
  // pool_kernel, 784 windows of 101 channels 7.3 / 9.0, 3136 of them 20.3 / 15.4)
  if (p.kx * p.ky >= 32 && blocks_w < 0x7fffffffLL && !fills_gpu && (vec || blocks_w <= 8LL * c.sm_count)) {
    const cudaError_t le = launch_pdl(vec ? avgpool_window_kernel<true> : avgpool_window_kernel<false>, dim3((unsigned)blocks_w), dim3(256), 0, c.stream, p, chunks);
    count_launch("avgpool_window_kernel");
    return cuda_ok(le, "avgpool launch") && cuda_ok(cudaGetLastError(), "avgpool launch");
  }
  // windows of at least 16 pixels: fewer threads with more bytes in flight each
  if (p.C % 16 == 0 && p.kx * p.ky >= 16 && ((reinterpret_cast<uintptr_t>(p.in) | reinterpret_cast<uintptr_t>(p.out)) & 15) == 0) {
    const int CW16 = p.C / 16;
    const long long total16 = (long long)p.B * p.Ho * p.Wo * CW16;
    const cudaError_t le = launch_pdl(avgpool16_kernel, dim3((unsigned)((total16 + 255) / 256)), dim3(256), 0, c.stream,
                                      p, CW16, total16);
    count_launch("avgpool16_kernel");
    return cuda_ok(le, "avgpool launch") && cuda_ok(cudaGetLastError(), "avgpool launch");
  }
  if (pool_fits(p, true, c.sm_count)) return launch_pool<true>(c, p);
  const int CW = vec ? p.C / 4 : p.C;
  const long long total = (long long)p.B * p.Ho * p.Wo * CW;
  const unsigned blocks = (unsigned)((total + 255) / 256);
  if (vec) avgpool_kernel<true><<<blocks, 256, 0, c.stream>>>(p, CW, total);
  else     avgpool_kernel<false><<<blocks, 256, 0, c.stream>>>(p, CW, total);
  count_launch("avgpool_kernel");
  return cuda_ok(cudaGetLastError(), "avgpool launch");
}

bool launch_add(Context &c, const uint8_t *a, const uint8_t *b, uint8_t *out, size_t n, int m1,
                int m2, int shift)
{
  const bool aligned = ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) |
                         reinterpret_cast<uintptr_t>(out)) & 15) == 0;
  const size_t n16 = aligned ? n / 16 : 0;
  const size_t items = n16 > n - n16 * 16 ? n16 : n - n16 * 16;
  const size_t want = (items + 255) / 256, most = (size_t)c.sm_count * 16;
  const cudaError_t le = launch_pdl(add_kernel, dim3((unsigned)(want < most ? want : most)), dim3(256), 0, c.stream, a, b, out, n16, n,
                                    m1, m2, shift);
  count_launch("add_kernel");
  return cuda_ok(le, "add launch");
}

}  // namespace pulpnn
