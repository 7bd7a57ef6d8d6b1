// packed_calls.cu -- the entry points called with their arguments as one block of bytes. Callers from an
// interpreter pay per argument for building a C value and handing it over (api.py: 25 arguments of a convolution,
// some 4 us, as long as the smallest kernels run); packing them into one block is a single call for each of the
// two steps. The blocks hold the arguments in declaration order, pointers first; api.py packs them with the format
// given beside each struct. Returns the calling thread's error code.
#include "internal.cuh"

namespace pulpnn_packed {

#pragma pack(push, 1)
struct ConvArgs { const void *p[7]; uint16_t v[16]; int32_t flags[2]; };                     // =7Q16H2i
struct DwArgs { const void *p[8]; uint16_t v[16]; int8_t flags[2]; };                        // =8Q16H2b
struct LinearArgs { const void *p[6]; uint16_t mult; int8_t shift; uint16_t dims[2]; int32_t flags[2]; };   // =6QHb2H2i
struct Linear32Args { const void *p[4]; uint16_t dims[2]; };                                 // =4Q2H
struct MaxpoolArgs { const void *p[2]; uint16_t v[13]; };                                    // =2Q13H
struct AvgpoolArgs { const void *p[2]; int64_t lambda; uint16_t shift; int64_t out_add; uint16_t v[13]; int32_t requant; };   // =2QqHq13Hi
struct AddArgs { const void *p[3]; uint16_t v[6]; };                                         // =3Q6H
#pragma pack(pop)

template <typename T> T *at(const void *p) { return static_cast<T *>(const_cast<void *>(p)); }

// the entry points of one family share their parameter list: which one it is comes as its address
template <typename BN_T>
void conv(void (*f)(PULPNN_CONV_PARAMS(BN_T)), const ConvArgs &a)
{
  f(at<uint8_t>(a.p[0]), at<uint8_t>(a.p[1]), at<int8_t>(a.p[2]), at<uint8_t>(a.p[3]), at<int8_t>(a.p[4]), at<BN_T>(a.p[5]),
    at<BN_T>(a.p[6]), a.v[0], a.v[1], a.v[2], a.v[3], a.v[4], a.v[5], a.v[6], a.v[7], a.v[8], a.v[9], a.v[10], a.v[11],
    a.v[12], a.v[13], a.v[14], a.v[15], a.flags[0], a.flags[1]);
}
template <typename BN_T>
void depthwise(void (*f)(PULPNN_DW_PARAMS(BN_T)), const DwArgs &a)
{
  f(at<uint8_t>(a.p[0]), at<uint8_t>(a.p[1]), at<int8_t>(a.p[2]), at<uint8_t>(a.p[3]), at<int8_t>(a.p[4]), at<uint8_t>(a.p[5]),
    at<BN_T>(a.p[6]), at<BN_T>(a.p[7]), a.v[0], a.v[1], a.v[2], a.v[3], a.v[4], a.v[5], a.v[6], a.v[7], a.v[8], a.v[9],
    a.v[10], a.v[11], a.v[12], a.v[13], a.v[14], a.v[15], a.flags[0], a.flags[1]);
}

}  // namespace pulpnn_packed

using namespace pulpnn_packed;

#define PULPNN_PACKED_TREE(SFX, BN_T)                                                                            \
  extern "C" int pulpnn_packed_conv##SFX(void (*f)(PULPNN_CONV_PARAMS(BN_T)), const ConvArgs *a)                 \
  {                                                                                                              \
    conv<BN_T>(f, *a);                                                                                           \
    return pulpnn_last_error();                                                                                  \
  }                                                                                                              \
  extern "C" int pulpnn_packed_depthwise##SFX(void (*f)(PULPNN_DW_PARAMS(BN_T)), const DwArgs *a)                \
  {                                                                                                              \
    depthwise<BN_T>(f, *a);                                                                                      \
    return pulpnn_last_error();                                                                                  \
  }                                                                                                              \
  extern "C" int pulpnn_packed_linear##SFX(const LinearArgs *a)                                                  \
  {                                                                                                              \
    pulp_nn_linear##SFX(at<uint8_t>(a->p[0]), at<int8_t>(a->p[1]), at<uint8_t>(a->p[2]), at<int8_t>(a->p[3]),    \
                        at<BN_T>(a->p[4]), at<BN_T>(a->p[5]), a->mult, a->shift, a->dims[0], a->dims[1],         \
                        a->flags[0], a->flags[1]);                                                               \
    return pulpnn_last_error();                                                                                  \
  }                                                                                                              \
  extern "C" int pulpnn_packed_linear_out_32##SFX(const Linear32Args *a)                                         \
  {                                                                                                              \
    pulp_nn_linear_out_32##SFX(at<uint8_t>(a->p[0]), at<int8_t>(a->p[1]), at<int32_t>(a->p[2]),                  \
                               at<int8_t>(a->p[3]), a->dims[0], a->dims[1]);                                     \
    return pulpnn_last_error();                                                                                  \
  }                                                                                                              \
  extern "C" int pulpnn_packed_maxpool##SFX(const MaxpoolArgs *a)                                                \
  {                                                                                                              \
    const uint16_t *v = a->v;                                                                                    \
    pulp_nn_maxpool##SFX(at<uint8_t>(a->p[0]), at<uint8_t>(a->p[1]), v[0], v[1], v[2], v[3], v[4], v[5], v[6],   \
                         v[7], v[8], v[9], v[10], v[11], v[12]);                                                 \
    return pulpnn_last_error();                                                                                  \
  }                                                                                                              \
  extern "C" int pulpnn_packed_avgpool##SFX(const AvgpoolArgs *a)                                                \
  {                                                                                                              \
    const uint16_t *v = a->v;                                                                                    \
    pulp_nn_avgpool##SFX(at<uint8_t>(a->p[0]), at<uint8_t>(a->p[1]), (BN_T)a->lambda, a->shift,                  \
                         (BN_T)a->out_add, v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7], v[8], v[9], v[10],    \
                         v[11], v[12], a->requant);                                                              \
    return pulpnn_last_error();                                                                                  \
  }                                                                                                              \
  extern "C" int pulpnn_packed_add##SFX(const AddArgs *a)                                                        \
  {                                                                                                              \
    const uint16_t *v = a->v;                                                                                    \
    pulp_nn_add##SFX(at<uint8_t>(a->p[0]), at<uint8_t>(a->p[1]), at<uint8_t>(a->p[2]), v[0], v[1], v[2], v[3],   \
                     v[4], v[5]);                                                                                \
    return pulpnn_last_error();                                                                                  \
  }

PULPNN_PACKED_TREE(_bn32, int32_t)
PULPNN_PACKED_TREE(_bn64, int64_t)
