// internal.cuh -- shared declarations of the library's translation units.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>
#include <stddef.h>
#include <atomic>

#include "../../include/pulpnn_b200.h"

namespace pulpnn {

// ---------------------------------------------------------------------------------------------
// Requantisation epilogues. The mode is decided on the host from (flag_relu, flag_batch_norm)
// exactly as the reference does (32bit/src/pulp_nn_matmul.c:144-216, pulp_nn_linear.c:88-107,
// pulp_nn_depthwise_generic.c:167-178).
// ---------------------------------------------------------------------------------------------
enum EpiMode : int {
  EPI_NONE = 0,   // clip(acc >> d)
  EPI_MULT = 1,   // clip((int16)((int16)out_mult * acc >> d))
  EPI_BN32 = 2,   // clip((int32)(k*acc + lambda) >> d), int32 wrap-around
  EPI_BN64 = 3,   // clip((int32)(((int64)k*acc + lambda) >> d))
  EPI_RAW32 = 4   // store the int32 accumulator (pulp_nn_linear_out_32)
};

struct Epilogue {
  const void *k;        // int32[] or int64[] per output channel (BN modes)
  const void *lambda;
  const void *bias;     // int8[] per output channel, int32[] for EPI_RAW32, or nullptr
  int mode;
  int out_mult;         // already converted to int16 range semantics on the host
  int shift;            // 0..31 (0..63 for EPI_BN64)
};

__device__ __forceinline__ int clip_u8(int x) { return min(max(x, 0), 255); }

template <int MODE>
__device__ __forceinline__ int requant(int acc, int ch, const Epilogue &e)
{
  if (MODE == EPI_BN32) {
    const int k = __ldg(reinterpret_cast<const int *>(e.k) + ch);
    const int l = __ldg(reinterpret_cast<const int *>(e.lambda) + ch);
    const int t = (int)((unsigned)k * (unsigned)acc + (unsigned)l);
    return clip_u8(t >> e.shift);
  } else if (MODE == EPI_BN64) {
    const long long k = __ldg(reinterpret_cast<const long long *>(e.k) + ch);
    const long long l = __ldg(reinterpret_cast<const long long *>(e.lambda) + ch);
    const long long t = (long long)((unsigned long long)k * (unsigned long long)(long long)acc +
                                    (unsigned long long)l);
    return clip_u8((int)(t >> e.shift));
  } else if (MODE == EPI_MULT) {
    const int p = (int)((unsigned)e.out_mult * (unsigned)acc);
    return clip_u8((int)(short)(p >> e.shift));
  } else {
    return clip_u8(acc >> e.shift);
  }
}

// requantisation with the per-channel parameters already in registers / shared memory
template <int MODE>
__device__ __forceinline__ int requant_kl(int acc, long long k, long long l, int out_mult, int shift)
{
  if (MODE == EPI_BN32) {
    const int t = (int)((unsigned)(int)k * (unsigned)acc + (unsigned)(int)l);
    return clip_u8(t >> shift);
  } else if (MODE == EPI_BN64) {
    const long long t = (long long)((unsigned long long)k * (unsigned long long)(long long)acc +
                                    (unsigned long long)l);
    return clip_u8((int)(t >> shift));
  } else if (MODE == EPI_MULT) {
    const int p = (int)((unsigned)out_mult * (unsigned)acc);
    return clip_u8((int)(short)(p >> shift));
  } else {
    return clip_u8(acc >> shift);
  }
}

// 64-bit batch normalisation in 32 bits, where that is the same: with |acc| <= acc_max (255 * 128 per term of
// the sum) k*acc + lambda cannot leave the int32 range, so the 32-bit multiply-add and shift give the very same
// value. A 64-bit product, sum and shift cost about eight instructions a value, and they, not memory, bounded the
// layers with 64-bit parameters (56x56x128 -> 256 at batch 64: 31.3 us against 20.2 with 32-bit ones).
constexpr unsigned ACC_PER_TERM = 255u * 128u;
__host__ __device__ constexpr unsigned acc_bound(int terms) { return terms <= 65535 ? (unsigned)terms * ACC_PER_TERM : 0xffffffffu; }
__device__ __forceinline__ bool bn_fits_32(long long k, long long l, unsigned acc_max, int shift)
{
  const unsigned long long ak = k < 0 ? 0ull - (unsigned long long)k : (unsigned long long)k;
  const unsigned long long al = l < 0 ? 0ull - (unsigned long long)l : (unsigned long long)l;
  return shift <= 31 && ak <= 0x7fffffffull && al <= 0x7fffffffull && ak * acc_max + al <= 0x7fffffffull;
}
// four adjacent channels, k and lambda in shared memory (16-byte aligned); fits: bn_fits_32 holds for all of them
__device__ __forceinline__ void requant4_bn64(const long long *k, const long long *l, unsigned v0, unsigned v1, unsigned v2,
                                              unsigned v3, int shift, bool fits, int (&q)[4])
{
  if (fits) {
    const int4 ka = *reinterpret_cast<const int4 *>(k), kb = *reinterpret_cast<const int4 *>(k + 2);
    const int4 la = *reinterpret_cast<const int4 *>(l), lb = *reinterpret_cast<const int4 *>(l + 2);
    q[0] = (int)((unsigned)ka.x * v0 + (unsigned)la.x) >> shift;
    q[1] = (int)((unsigned)ka.z * v1 + (unsigned)la.z) >> shift;
    q[2] = (int)((unsigned)kb.x * v2 + (unsigned)lb.x) >> shift;
    q[3] = (int)((unsigned)kb.z * v3 + (unsigned)lb.z) >> shift;
  } else {
    const unsigned v[4] = {v0, v1, v2, v3};
#pragma unroll
    for (int t = 0; t < 4; t++)
      q[t] = (int)((long long)((unsigned long long)k[t] * (unsigned long long)(long long)(int)v[t] + (unsigned long long)l[t]) >> shift);
  }
}

// Clamp four int32 values to [0,255] and pack them, a in the lowest byte. cvt.pack.sat converts
// two values per instruction: d[7:0] = sat(second), d[15:8] = sat(first), d[31:16] = third[15:0].
__device__ __forceinline__ unsigned pack4_sat_u8(int a, int b, int c, int d)
{
  unsigned hi, r;
  asm("cvt.pack.sat.u8.s32.b32 %0, %1, %2, %3;" : "=r"(hi) : "r"(d), "r"(c), "r"(0));
  asm("cvt.pack.sat.u8.s32.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(b), "r"(a), "r"(hi));
  return r;
}

// u8 x s8 dot product of four byte lanes
__device__ __forceinline__ int dp4a_us(unsigned a_u8x4, int b_s8x4, int c)
{
  int d;
  asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(a_u8x4), "r"(b_s8x4), "r"(c));
  return d;
}

// Division of 0 .. 2^31-1 by a constant of the launch: a multiply and a shift where the hardware's
// integer division takes some 25 instructions (Granlund and Montgomery, division by invariant integers).
struct FastDiv {
  unsigned d, mul, shift;
  void set(unsigned v)
  {
    d = v; mul = 0; shift = 0;
    if (v <= 1) return;
    unsigned l = 1;
    while ((1ull << l) < v) l++;
    mul = (unsigned)(((1ull << (31 + l)) + v - 1) / v);
    shift = l - 1;
  }
#ifdef __CUDACC__
  __device__ __forceinline__ int div(int n) const { return d == 1 ? n : (int)(__umulhi((unsigned)n, mul) >> shift); }
#endif
};

// ---------------------------------------------------------------------------------------------
// Problem descriptions handed from the entry points to the launchers (all pointers are device
// pointers by then).
// ---------------------------------------------------------------------------------------------
// Block-diagonal copies of a layer's weights (see launch_igemm_tc), made once and kept by whoever
// owns the layer; slot i holds the copy for 2^i pixels per GEMM row. Device memory, freed by the owner.
struct FoldedWeights { int8_t *w[8] = {nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr}; };

struct ConvProblem {
  const uint8_t *in;     // [B][H][W][Cin]
  const int8_t *w;       // [Cout][ky][kx][Cin]
  void *out;             // [B][Ho][Wo][Cout] uint8 (int32 for EPI_RAW32)
  int B, H, W, Cin, Ho, Wo, Cout, ky, kx, pt, pl, sy, sx;
  Epilogue epi;
  FoldedWeights *folded = nullptr;   // optional: where constant weights keep their folded copies
};

struct DepthwiseProblem {
  const uint8_t *in;     // [B][C][H][W] (chw) or [B][H][W][C]
  const int8_t *w;       // [C][ky][kx]
  uint8_t *out;          // [B][Ho][Wo][C]
  int B, H, W, C, Ho, Wo, ky, kx, pt, pl, sy, sx;
  bool in_is_hwc;
  Epilogue epi;
};

struct PoolProblem {
  const uint8_t *in;     // [B][H][W][C]
  uint8_t *out;          // [B][Ho][Wo][C]
  int B, H, W, C, Ho, Wo, ky, kx, pt, pb, pl, pr, sy, sx;
  // avgpool only
  int bn_bits, requant, shift;
  long long lambda, out_add;
};

// ---------------------------------------------------------------------------------------------
// Per-thread context
// ---------------------------------------------------------------------------------------------
struct StageSlot { void *dev = nullptr; size_t cap = 0; };

// Memory for the partial sums of the longest reductions, and when their latest reader was through with them; given back
// when its thread ends.
struct Partials {
  void *mem = nullptr; size_t cap = 0;
  cudaEvent_t done = nullptr;
  ~Partials();
};

struct Context {
  int device = -1;
  cudaStream_t stream = nullptr;
  int batch = 1;
  int err = PULPNN_OK;
  char msg[512] = {0};
  int opt_force_generic = 0;
  int opt_maxpool_clobber = 0;
  int opt_split_k = 0;
  int opt_tune = 0;               // experiment switch: alternative kernel configurations (bit mask)
  int opt_fuse_dwpw = 1;          // the network runner pairs depthwise + pointwise layers into one kernel
  StageSlot slots[8];
  // device scratch owned by the context (split-K partial sums, status word)
  void *scratch = nullptr; size_t scratch_cap = 0;
  Partials partials;
  int *status_word = nullptr;     // device int, 0 = fine
  int sm_count = 0;
};

Context &ctx();
bool ensure_device(Context &c);
void set_error(int code, const char *fmt, ...);
bool cuda_ok(cudaError_t e, const char *what);
void count_launch(unsigned n = 1);
void count_launch(const char *kernel_name);     // one launch, and remembers which kernel family it was
unsigned long long thread_launch_count();       // launches made by the calling thread so far
const char *thread_last_kernel();               // the kernel family of the calling thread's latest named launch

// Programmatic dependent launch. A kernel launched this way may become resident and run its
// prologue while the previous kernel of the stream is still draining; it must execute pdl_wait()
// before it reads anything an earlier kernel wrote or writes anything an earlier kernel may still
// read (the wait returns once the earlier grids have completed and their writes are visible).
// pdl_launch_dependents() lets the NEXT kernel of the stream do the same with respect to this one.
// Both are no-ops in a kernel launched the ordinary way.
template <typename... KArgs, typename... Args>
inline cudaError_t launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                              Args &&...args)
{
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr; cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}
#ifdef __CUDACC__
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
#endif
void *ctx_scratch(Context &c, size_t bytes);    // grow-only device scratch, nullptr on failure
// Memory for partial sums that the context's stream may write from now on, whichever stream used it before; nullptr, and
// no error, under a stream capture and where there is none to be had. ctx_partials_done() after the last kernel that reads them.
void *ctx_partials(Context &c, size_t bytes);
bool ctx_partials_done(Context &c);

// A per-kernel setting that belongs to a device (cudaFuncSetAttribute, an occupancy figure) is
// cached per device, not per process or per thread: one process may drive several GPUs, from one
// thread that rebinds its context or from a thread per GPU.
constexpr int MAX_DEVICES = 64;
struct PerDeviceInt {
  std::atomic<int> v[MAX_DEVICES];
  PerDeviceInt() { for (auto &x : v) x.store(0, std::memory_order_relaxed); }
  int get(int dev) const { return (dev >= 0 && dev < MAX_DEVICES) ? v[dev].load(std::memory_order_acquire) : 0; }
  void set(int dev, int val) { if (dev >= 0 && dev < MAX_DEVICES) v[dev].store(val, std::memory_order_release); }
};

// Stages host buffers through device memory. Device pointers pass through untouched.
class Stager {
 public:
  explicit Stager(Context &c) : c_(c) {}
  const void *in(const void *p, size_t bytes);
  void *out(void *p, size_t bytes);
  void *inout(void *p, size_t bytes);
  bool ok() const { return ok_; }
  // copies results back and waits if any buffer was staged; returns false on a CUDA error
  bool finish();
 private:
  void *stage(const void *p, size_t bytes, bool copy_in, bool copy_out);
  Context &c_;
  struct Pending { void *host; void *dev; size_t bytes; } pend_[8];
  int n_pend_ = 0, n_slot_ = 0;
  bool ok_ = true, staged_ = false;
};

// ---------------------------------------------------------------------------------------------
// Launchers (each returns false and records an error when the launch could not be made)
// ---------------------------------------------------------------------------------------------
bool launch_conv(Context &c, const ConvProblem &p);             // picks tensor-core or generic
bool launch_conv_generic(Context &c, const ConvProblem &p);
// spatial kernels with every input pixel fetched once per tile (estimated ns, -1 where that kernel does not take it)
double conv_halo_tc_estimate(const Context &c, const ConvProblem &p);
bool launch_conv_halo_tc(Context &c, const ConvProblem &p);
// any channel count and alignment on the tensor cores, the im2col rows gathered by the warps
bool conv_gather_tc_supported(const ConvProblem &p);
// ns, or a lower bound that is not below `worth`; -1 where it does not take the problem
double conv_gather_tc_estimate(const Context &c, const ConvProblem &p, double worth);
bool launch_conv_gather_tc(Context &c, const ConvProblem &p);
bool conv_smallcin_tc_supported(const ConvProblem &p);
bool launch_conv_smallcin_tc(Context &c, const ConvProblem &p);
bool conv_smallcin_supported(const ConvProblem &p);
double conv_smallcin_estimate(const Context &c, const ConvProblem &p);        // ns of a problem it takes
bool launch_conv_smallcin(Context &c, const ConvProblem &p);
bool igemm_tc_supported(const Context &c, const ConvProblem &p);
// `slices`: K split over so many CTAs, whose sums go through memory that igemm_tc_partials() got just before
bool launch_igemm_tc(Context &c, const ConvProblem &p, int slices = 1);
int igemm_tc_slices(const Context &c, const ConvProblem &p);    // for a long reduction of few tiles
bool igemm_tc_partials(Context &c, const ConvProblem &p, int slices);     // false (no error) where there is none to be had
// whether its output rows are whole 16-byte pieces; otherwise it stores byte by byte
bool igemm_tc_whole_rows(const Context &c, const ConvProblem &p);
// whether a tile has so few values, behind so short a reduction, that storing them byte by byte does not matter
bool igemm_tc_few_values(const ConvProblem &p);
// m-tiles x n-tiles that kernel cuts the problem into, and whether these are so few that it leaves the GPU idle over a
// reduction of eight slabs or more
int igemm_tc_tiles(const Context &c, const ConvProblem &p, bool *few);
double igemm_tc_spatial_estimate(const Context &c, const ConvProblem &p);     // ns of a spatial kernel with whole rows; -1 where it does not take the problem
// the same GEMM computed by pairs of SMs (tcgen05 cta_group::2), for wide layers with a long reduction
bool igemm_tc2_supported(const Context &c, const ConvProblem &p);
bool launch_igemm_tc2(Context &c, const ConvProblem &p);
// the same GEMM for few tiles, the reduction shared by the CTAs of a cluster
// (estimated ns, or -1 where that kernel does not take the problem)
double igemm_split_estimate(const Context &c, const ConvProblem &p);
bool launch_igemm_split(Context &c, const ConvProblem &p);
// the same contraction for few rows (a fully connected layer at a small batch), on dp4a
bool gemm_fewrows_supported(const ConvProblem &p);
bool launch_gemm_fewrows(Context &c, const ConvProblem &p);
bool launch_depthwise(Context &c, const DepthwiseProblem &p);
bool depthwise_hwc3x3_supported(const DepthwiseProblem &p);
bool launch_depthwise_hwc3x3(Context &c, const DepthwiseProblem &p);
bool depthwise_hwc3x3_tma_supported(const DepthwiseProblem &p);
bool launch_depthwise_hwc3x3_tma(Context &c, const DepthwiseProblem &p);
bool depthwise_chw3x3_tma_supported(const DepthwiseProblem &p);
bool launch_depthwise_chw3x3_tma(Context &c, const DepthwiseProblem &p);
// a 3x3 stride-1 depthwise layer and the pointwise layer behind it in one kernel (dwpw_fused.cu)
bool dwpw_fused_supported(const DepthwiseProblem &dw, const ConvProblem &pw);
bool launch_dwpw_fused(Context &c, const DepthwiseProblem &dw, const ConvProblem &pw);
// the 32 -> 64 channel pair with the depthwise layer on the tensor cores too (dwpw_tcdw.cu)
bool dwpw_tcdw_supported(const DepthwiseProblem &dw, const ConvProblem &pw);
bool launch_dwpw_tcdw(Context &c, const DepthwiseProblem &dw, const ConvProblem &pw);
// 3x3 / 5x5 at any channel count and alignment, HWC or CHW input, from planes in shared memory
bool depthwise_planes_supported(const DepthwiseProblem &p);
bool launch_depthwise_planes(Context &c, const DepthwiseProblem &p);
int *ctx_status_word(Context &c);               // allocated on first use; nullptr on failure
// the same for calls that may come first under a stream capture, where nothing can be allocated: *word stays nullptr
// then, and a bounded wait that runs out still ends its kernel, unrecorded. false: the allocation failed
bool ctx_status_word_unless_capturing(Context &c, int **word);
int static_scratch_status_take(Context &c);     // status of the no-allocation entry point (0: unused or fine)
bool launch_maxpool(Context &c, const PoolProblem &p, uint8_t *clobber_in);
bool launch_avgpool(Context &c, const PoolProblem &p);
bool launch_add(Context &c, const uint8_t *a, const uint8_t *b, uint8_t *out, size_t n, int m1,
                int m2, int shift);

}  // namespace pulpnn
