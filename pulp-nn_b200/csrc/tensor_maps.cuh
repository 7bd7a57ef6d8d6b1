// tensor_maps.cuh -- tensor maps of the GEMM operands and the cut of a convolution's output into patches,
// shared by the kernels that load them with TMA.
#pragma once

#include "internal.cuh"
#include "sm100_primitives.cuh"

namespace pulpnn {

// [rows][K] byte matrix, K contiguous; box = bkb bytes of K x box_rows rows, bkb-byte swizzle.
// Elements outside the matrix read as zero.
inline bool make_map(CUtensorMap *map, const void *base, int rows, int K, int box_rows, int bkb)
{
  sm100::EncodeTiledFn enc = sm100::encode_tiled_fn();
  if (!enc) { set_error(PULPNN_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver"); return false; }
  cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)K};
  cuuint32_t box[2] = {(cuuint32_t)bkb, (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  const CUtensorMapSwizzle sw = bkb == 128 ? CU_TENSOR_MAP_SWIZZLE_128B
                              : (bkb == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B);
  CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void *>(base), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) { set_error(PULPNN_ERR_CUDA, "cuTensorMapEncodeTiled failed with code %d", (int)r); return false; }
  return true;
}

// [B][H][W][C] image, boxes of box_c bytes x box_w x box_h pixels of one image, every sx-th (sy-th)
// pixel of the box taken: the pixels one filter tap reads for a patch of outputs
inline bool make_map_4d(CUtensorMap *map, const void *base, int C, int Wd, int Hd, int B, int box_c, int box_w, int box_h,
                 int sx, int sy)
{
  sm100::EncodeTiledFn enc = sm100::encode_tiled_fn();
  if (!enc) { set_error(PULPNN_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver"); return false; }
  cuuint64_t dims[4] = {(cuuint64_t)C, (cuuint64_t)Wd, (cuuint64_t)Hd, (cuuint64_t)B};
  cuuint64_t strides[3] = {(cuuint64_t)C, (cuuint64_t)Wd * C, (cuuint64_t)Hd * Wd * C};
  cuuint32_t box[4] = {(cuuint32_t)box_c, (cuuint32_t)((box_w - 1) * sx + 1), (cuuint32_t)((box_h - 1) * sy + 1), 1};
  cuuint32_t estr[4] = {1, (cuuint32_t)sx, (cuuint32_t)sy, 1};
  const CUtensorMapSwizzle sw = box_c == 128 ? CU_TENSOR_MAP_SWIZZLE_128B
                              : (box_c == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B);
  CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, const_cast<void *>(base), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) { set_error(PULPNN_ERR_CUDA, "cuTensorMapEncodeTiled (4-D) failed with code %d", (int)r); return false; }
  return true;
}

// patch width (a power of two, the patch has 128 pixels) that covers the output with the fewest
// wasted pixels; the wider one on a tie
inline int pick_patch_width_log2(int Ho, int Wo, int sx, int sy)
{
  int best = -1;
  long long best_cost = 0;
  for (int l = 3; l <= 7; l++) {
    const int tw = 1 << l, th = 128 >> l;
    if ((tw - 1) * sx + 1 > 256 || (th - 1) * sy + 1 > 256) continue;
    const long long cost = (long long)((Wo + tw - 1) / tw) * ((Ho + th - 1) / th);
    if (best < 0 || cost <= best_cost) { best = l; best_cost = cost; }
  }
  return best;
}

// a pointwise convolution or a fully connected layer: A is the plain [M][K] matrix
inline bool igemm_is_plain(const ConvProblem &p)
{
  return p.ky == 1 && p.kx == 1 && p.sy == 1 && p.sx == 1 && p.pt == 0 && p.pl == 0 && p.H == p.Ho && p.W == p.Wo;
}

}  // namespace pulpnn
