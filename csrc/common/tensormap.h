// Host-side helper: build CUtensorMap objects without linking libcuda (the encode entry point is
// fetched through the runtime, so the library also links on a machine without a driver).
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>

namespace fi {

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline EncodeTiledFn get_encode_tiled() {
  static EncodeTiledFn fn = nullptr;
  if (fn == nullptr) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) !=
            cudaSuccess ||
        q != cudaDriverEntryPointSuccess) {
      return nullptr;
    }
    fn = reinterpret_cast<EncodeTiledFn>(p);
  }
  return fn;
}

// Row-major 2-D tensor [rows, cols] of 16-bit elements with row pitch `ld` elements.
// Box = [box_rows, 64 columns] (128 bytes wide) with the 128-byte swizzle; out-of-range reads give 0.
// Requirements (checked): base 16-byte aligned, pitch a multiple of 16 bytes.
inline int make_tmap_2d_16bit_sw128(CUtensorMap* out, const void* base, uint64_t rows,
                                    uint64_t cols, uint64_t ld, uint32_t box_rows) {
  EncodeTiledFn enc = get_encode_tiled();
  if (enc == nullptr) return -1;
  if ((reinterpret_cast<uintptr_t>(base) & 15) != 0 || ((ld * 2) & 15) != 0) return -2;
  cuuint64_t dims[2] = {cols, rows};
  cuuint64_t strides[1] = {ld * 2};
  cuuint32_t box[2] = {64, box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = enc(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims,
                   strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -3;
}

// The same over rows that are split into equal parts: element (row, part, col) at row * ld + part * part_ld + col.
// Box = [box_rows, box_parts, 64 columns]; in shared memory the parts of a row follow one another.
inline int make_tmap_3d_16bit_sw128(CUtensorMap* out, const void* base, uint64_t rows, uint64_t parts, uint64_t cols,
                                    uint64_t ld, uint64_t part_ld, uint32_t box_rows, uint32_t box_parts) {
  EncodeTiledFn enc = get_encode_tiled();
  if (enc == nullptr) return -1;
  if ((reinterpret_cast<uintptr_t>(base) & 15) != 0 || ((ld * 2) & 15) != 0 || ((part_ld * 2) & 15) != 0) return -2;
  cuuint64_t dims[3] = {cols, parts, rows};
  cuuint64_t strides[2] = {part_ld * 2, ld * 2};
  cuuint32_t box[3] = {64, box_parts, box_rows};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = enc(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims,
                   strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -3;
}

// Gated weights [2 * half, cols] (gate rows, then up rows) as tiles of eight gate rows, their eight up rows, the next eight gate rows and so
// on: box = 128 rows of 64 columns.  half is a multiple of 8.
inline int make_tmap_gate_up_16bit_sw128(CUtensorMap* out, const void* base, uint64_t half, uint64_t cols, uint64_t ld) {
  EncodeTiledFn enc = get_encode_tiled();
  if (enc == nullptr) return -1;
  if ((reinterpret_cast<uintptr_t>(base) & 15) != 0 || ((ld * 2) & 15) != 0 || half % 8 != 0) return -2;
  cuuint64_t dims[4] = {cols, 8, 2, half / 8};
  cuuint64_t strides[3] = {ld * 2, half * ld * 2, 8 * ld * 2};
  cuuint32_t box[4] = {64, 8, 2, 8};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  CUresult r = enc(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(base), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -3;
}

// Packed weights as a 2-D int32 tensor [rows, K/8]; box = 8 * subs words x 128 rows with the swizzle of its width.
inline int make_tmap_packed(CUtensorMap* out, const void* base, uint64_t rows, uint64_t k_words, int subs) {
  EncodeTiledFn enc = get_encode_tiled();
  if (enc == nullptr) return -1;
  if ((reinterpret_cast<uintptr_t>(base) & 15) != 0 || ((k_words * 4) & 15) != 0) return -2;
  cuuint64_t dims[2] = {k_words, rows};
  cuuint64_t strides[1] = {k_words * 4};
  cuuint32_t box[2] = {static_cast<cuuint32_t>(8 * subs), 128};
  cuuint32_t estr[2] = {1, 1};
  const CUtensorMapSwizzle swz = subs == 4 ? CU_TENSOR_MAP_SWIZZLE_128B
                                           : (subs == 2 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_NONE);
  CUresult r = enc(out, CU_TENSOR_MAP_DATA_TYPE_INT32, 2, const_cast<void*>(base), dims, strides, box,
                   estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swz,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -3;
}

// Rows of plain 8- or 16-bit elements [rows, cols], pitch = cols: box = box_cols x box_rows, no swizzle (group scales and zero points,
// whose neighbouring columns are neighbouring weight rows).
inline int make_tmap_plain(CUtensorMap* out, const void* base, uint64_t rows, uint64_t cols, int elem_bytes, uint32_t box_cols,
                           uint32_t box_rows) {
  EncodeTiledFn enc = get_encode_tiled();
  if (enc == nullptr) return -1;
  if ((reinterpret_cast<uintptr_t>(base) & 15) != 0 || ((cols * elem_bytes) & 15) != 0) return -2;
  cuuint64_t dims[2] = {cols, rows};
  cuuint64_t strides[1] = {cols * elem_bytes};
  cuuint32_t box[2] = {box_cols, box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = enc(out, elem_bytes == 1 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, const_cast<void*>(base), dims,
                   strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -3;
}

}  // namespace fi
