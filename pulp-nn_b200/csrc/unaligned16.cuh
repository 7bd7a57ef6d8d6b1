// unaligned16.cuh -- 16-byte pieces of a byte tensor at any address, read with aligned 16-byte loads
// that never touch a byte outside the tensor. Shared by the kernels that gather rows of HWC or CHW data
// whose starts are not aligned.
#pragma once

#include "internal.cuh"

namespace pulpnn {

// A byte tensor addressed by 32-bit offsets from the 16-byte boundary at or below its start: it
// occupies [start, end). A block of 32 bytes at offset o (a multiple of 16) lies wholly inside when
// (unsigned)(o - whole_lo) < whole_n.
struct Bytes {
  const uint8_t *base;
  int start, end, whole_lo;
  unsigned whole_n;
  __device__ __forceinline__ Bytes(const void *p, int n)
  {
    const uintptr_t a = reinterpret_cast<uintptr_t>(p);
    base = reinterpret_cast<const uint8_t *>(a & ~(uintptr_t)15);
    start = (int)(a & 15);
    end = start + n;
    whole_lo = (start + 15) & ~15;
    whole_n = (unsigned)max(end - 31 - whole_lo, 0);
  }
};

__device__ __forceinline__ uint4 ldg16_if(const uint8_t *p, bool ok)
{
  uint4 v;
  asm volatile(
      "{\n\t.reg .pred q;\n\t"
      "setp.ne.b32 q, %5, 0;\n\t"
      "mov.b32 %0, 0;\n\tmov.b32 %1, 0;\n\tmov.b32 %2, 0;\n\tmov.b32 %3, 0;\n\t"
      "@q ld.global.nc.v4.b32 {%0, %1, %2, %3}, [%4];\n\t}"
      : "=&r"(v.x), "=&r"(v.y), "=&r"(v.z), "=&r"(v.w)
      : "l"(p), "r"((int)ok));
  return v;
}

__device__ __forceinline__ unsigned ldg4_if(const uint8_t *p, bool ok)
{
  unsigned v;
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %2, 0;\n\tmov.b32 %0, 0;\n\t@q ld.global.nc.b32 %0, [%1];\n\t}"
               : "=&r"(v) : "l"(p), "r"((int)ok));
  return v;
}
__device__ __forceinline__ unsigned ldg1_if(const uint8_t *p, bool ok)
{
  unsigned v;
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %2, 0;\n\tmov.b32 %0, 0;\n\t@q ld.global.nc.u8 %0, [%1];\n\t}"
               : "=&r"(v) : "l"(p), "r"((int)ok));
  return v;
}

// The 16 bytes at offset o of a tensor, in two steps so that several chunks are in flight at once:
// fetch() issues the loads without a branch, get() does the rest. Bytes outside the tensor are never
// touched and read as zero: a chunk whose aligned 32 bytes are not wholly inside goes byte by byte.
struct Chunk {
  uint4 a, b;
  int o;
  __device__ __forceinline__ void fetch(const Bytes &t, int off, bool need)
  {
    o = off;
    const int ob = off & ~15;
    const bool ok = need && (unsigned)(ob - t.whole_lo) < t.whole_n;
    const uint8_t *at = t.base + ob;
    a = ldg16_if(at, ok);
    b = ldg16_if(at + 16, ok);
  }
  __device__ __forceinline__ uint4 get(const Bytes &t) const
  {
    if ((unsigned)((o & ~15) - t.whole_lo) >= t.whole_n) return bytes(t.base, o, t.start, t.end);
    const bool s2 = o & 8, s1 = o & 4;
    const unsigned t0 = s2 ? a.z : a.x, t1 = s2 ? a.w : a.y, t2 = s2 ? b.x : a.z, t3 = s2 ? b.y : a.w,
                   t4 = s2 ? b.z : b.x, t5 = s2 ? b.w : b.y;
    const unsigned u0 = s1 ? t1 : t0, u1 = s1 ? t2 : t1, u2 = s1 ? t3 : t2, u3 = s1 ? t4 : t3, u4 = s1 ? t5 : t4;
    const unsigned bs = (unsigned)o * 8;             // the funnel shift takes it modulo 32
    return make_uint4(__funnelshift_r(u0, u1, bs), __funnelshift_r(u1, u2, bs), __funnelshift_r(u2, u3, bs),
                      __funnelshift_r(u3, u4, bs));
  }
  __device__ __noinline__ static uint4 bytes(const uint8_t *base, int o, int start, int end)
  {
    unsigned w[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
      w[i] = 0;
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const int q = o + 4 * i + j;
        if (q >= start && q < end) w[i] |= (unsigned)__ldg(base + q) << (8 * j);
      }
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
  }
};

// One image of a tensor of bytes, by offsets from the word at or below its first byte (`lead` bytes before it): between
// lo and hi lie the image's own bytes and up to 64 of the `before` and `after` that the tensor has on either side.
struct ImageSpan {
  int lo, hi;
  __host__ __device__ ImageSpan(int lead, int own, size_t before, size_t after)
      : lo(lead - (int)(before < 64 ? before : 64)), hi(lead + own + (int)(after < 64 ? after : 64)) {}
  // four pixels of C bytes from offset `at` on, each read as the two words that its first four bytes lie across
  __host__ __device__ bool holds_words(int at, int C) const { return (at & ~3) >= lo && at + 3 * C + 8 <= hi; }
};

// bytes [from, to) of word i of a 16-byte chunk
__device__ __forceinline__ unsigned word_mask(int i, int from, int to)
{
  const int f = min(max(from - 4 * i, 0), 4), t = min(max(to - 4 * i, 0), 4);
  const unsigned mt = t == 4 ? 0xffffffffu : ((1u << (8 * t)) - 1u);
  const unsigned mf = f == 4 ? 0xffffffffu : ((1u << (8 * f)) - 1u);
  return mt & ~mf;
}
__device__ __forceinline__ void mask16(uint4 &v, int from, int to)
{
  v.x &= word_mask(0, from, to); v.y &= word_mask(1, from, to);
  v.z &= word_mask(2, from, to); v.w &= word_mask(3, from, to);
}

}  // namespace pulpnn
