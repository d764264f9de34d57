// swe_maps.cuh -- host side of the tiled stage kernels' tensor maps.
#pragma once

#include <cudaTypedefs.h>        // PFN_cuTensorMapEncodeTiled (fetched through the runtime, no -lcuda)
#include <cstdlib>
#include <cstring>

#include "swe_split.cuh"

namespace swe {
namespace {

// The driver's tensor-map encoder, or null; null too where SWE_B200_TMA=0 turns
// the tile copies off.
inline PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
  const char* env = std::getenv("SWE_B200_TMA");
  if (env && std::strcmp(env, "0") == 0) return nullptr;
  static PFN_cuTensorMapEncodeTiled_v12000 encode = nullptr;
  if (!encode) {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess || !fn)
      return nullptr;
    encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
  }
  return encode;
}
// A 2-D map over one W x H field of doubles, rows of `pitch` (even), with the
// given box; zeros outside.
inline bool encode_field(PFN_cuTensorMapEncodeTiled_v12000 encode, CUtensorMap* m, const double* base, int W, int H,
                         int pitch, int bx, int by) {
  const cuuint64_t dims[2] = {(cuuint64_t)W, (cuuint64_t)H};
  const cuuint64_t strides[1] = {(cuuint64_t)pitch * sizeof(double)};
  const cuuint32_t box[2] = {(cuuint32_t)bx, (cuuint32_t)by};
  const cuuint32_t estr[2] = {1, 1};
  return encode(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 2, const_cast<double*>(base), dims, strides, box, estr,
                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// The cell kernel's maps: the face fields, whose rows are aligned (an even
// pitch), and the stage input's depth h where W is even (else the kernel copies
// it element by element).
inline bool make_cell_maps(CellMaps& c, const SplitBufs& sb, const double* h, int W, int H) {
  PFN_cuTensorMapEncodeTiled_v12000 encode = tensor_map_encoder();
  const int P = sb.P;
  if (!encode || P % 2 != 0) return false;
  bool ok = encode_field(encode, &c.m[CM_XM], sb.fx[F_M], W, H, P, SPX + 4, SPY + 2) &&
            encode_field(encode, &c.m[CM_YM], sb.fy[F_M], W, H, P, SPX + 4, SPY + 3);
  if (W % 2 == 0) ok = ok && encode_field(encode, &c.m[CM_H], h, W, H, W, SPX + 4, SPY + 2);
  for (int q = 0; q < 3 && ok; q++)
    ok = encode_field(encode, &c.m[CM_XT + q], sb.fx[q + 1], W, H, P, SPX + 2, SPY) &&
         encode_field(encode, &c.m[CM_YT + q], sb.fy[q + 1], W, H, P, SPX, SPY + 1) &&
         encode_field(encode, &c.m[CM_TB + q], sb.tb[q], W, H, P, SPX, SPY);
  return ok;
}

// The face kernel's maps: b and the state (h, hu, hv), each a W x H array, box
// SSXT x SSY.  Without them (an odd W, whose rows are not 16-byte aligned) the
// kernel copies element by element; the same bits.
inline bool make_tile_maps(TileMaps& t, const double* b, double* const* state, int W, int H) {
  PFN_cuTensorMapEncodeTiled_v12000 encode = tensor_map_encoder();
  if (!encode || W % 2 != 0) return false;
  for (int f = 0; f < 4; f++)
    if (!encode_field(encode, &t.m[f], f == 0 ? b : state[f - 1], W, H, W, SSXT, SSY)) return false;
  return true;
}

}  // namespace
}  // namespace swe
