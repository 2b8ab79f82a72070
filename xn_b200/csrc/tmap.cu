// Host-side tensor maps of the tensor-memory kernels.  The encoder is resolved from the driver at run time: the library
// links only the CUDA runtime.
#include "tc05.cuh"

namespace xn {
namespace {

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            p = nullptr;
        return (EncodeTiledFn)p;
    }();
    return fn;
}

}  // namespace

// 2-D row-major [rows, k] tensor with `elem` bytes per element and a row pitch of ld elements;
// box = 128 bytes of k by box_rows rows, 128-byte swizzle, out-of-range reads give zeros.
// 3-D form of the same map: `batch` matrices `batch_stride` elements apart (box covers one of them).
// Dimensions are ordered by increasing stride: when the batch stride is smaller than the row pitch (a
// transposed view such as [groups, rows, k] over storage [rows, groups, k]) the map is (k, batch, rows) and
// *batch_inner is set; the shared-memory image of a box is the same either way.
int make_map3(CUtensorMap *map, const void *base, int elem, size_t rows, size_t k, size_t ld, int box_rows,
              size_t batch, size_t batch_stride, int *batch_inner) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return fail(XN_ERR_CUDA, "cuTensorMapEncodeTiled is not available from this driver");
    if (batch <= 1) { batch = 1; batch_stride = rows * ld; }
    const bool inner = batch_stride < ld;
    *batch_inner = inner ? 1 : 0;
    cuuint64_t dims[3] = {(cuuint64_t)k, (cuuint64_t)(inner ? batch : rows), (cuuint64_t)(inner ? rows : batch)};
    cuuint64_t strides[2] = {(cuuint64_t)(inner ? batch_stride : ld) * elem, (cuuint64_t)(inner ? ld : batch_stride) * elem};
    cuuint32_t box[3] = {(cuuint32_t)(BKB / elem), (cuuint32_t)(inner ? 1 : box_rows), (cuuint32_t)(inner ? box_rows : 1)};
    cuuint32_t estr[3] = {1, 1, 1};
    CUtensorMapDataType dt = elem == 1 ? CU_TENSOR_MAP_DATA_TYPE_UINT8
                                       : (elem == 4 ? CU_TENSOR_MAP_DATA_TYPE_UINT32 : CU_TENSOR_MAP_DATA_TYPE_UINT16);
    CUresult r = fn(map, dt, 3, const_cast<void *>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(XN_ERR_CUDA, "cuTensorMapEncodeTiled (3-D) failed with code %d", (int)r);
    return XN_OK;
}

int make_map(CUtensorMap *map, const void *base, int elem, size_t rows, size_t k, size_t ld, int box_rows) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return fail(XN_ERR_CUDA, "cuTensorMapEncodeTiled is not available from this driver");
    cuuint64_t dims[2] = {(cuuint64_t)k, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)ld * elem};
    cuuint32_t box[2] = {(cuuint32_t)(BKB / elem), (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUtensorMapDataType dt = elem == 1 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_UINT16;
    CUresult r = fn(map, dt, 2, const_cast<void *>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(XN_ERR_CUDA, "cuTensorMapEncodeTiled failed with code %d", (int)r);
    return XN_OK;
}

// [K, N] operand with n contiguous, k-rows `ld` elements apart, `batch` matrices batch_stride elements apart:
// dimensions (n, k, batch), box 64 n x 64 k (128-byte rows, 128-byte swizzle).  16-bit elements only.
// As in make_map3 the dimensions are ordered by increasing stride: when the matrices interleave (batch stride
// smaller than the k-row pitch, e.g. the per-head value slices of a fused qkv projection) the map is (n, batch, k)
// and *batch_inner is set.
int make_map_mn(CUtensorMap *map, const void *base, size_t n, size_t k, size_t ld, size_t batch, size_t batch_stride,
                int *batch_inner) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return fail(XN_ERR_CUDA, "cuTensorMapEncodeTiled is not available from this driver");
    if (batch <= 1) { batch = 1; batch_stride = k * ld; }
    const bool inner = batch_stride < ld;
    *batch_inner = inner ? 1 : 0;
    cuuint64_t dims[3] = {(cuuint64_t)n, (cuuint64_t)(inner ? batch : k), (cuuint64_t)(inner ? k : batch)};
    cuuint64_t strides[2] = {(cuuint64_t)(inner ? batch_stride : ld) * 2, (cuuint64_t)(inner ? ld : batch_stride) * 2};
    cuuint32_t box[3] = {64, (cuuint32_t)(inner ? 1 : BKB / 2), (cuuint32_t)(inner ? BKB / 2 : 1)};
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT16, 3, const_cast<void *>(base), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(XN_ERR_CUDA, "cuTensorMapEncodeTiled (n-contiguous operand) failed with code %d", (int)r);
    return XN_OK;
}

}  // namespace xn
