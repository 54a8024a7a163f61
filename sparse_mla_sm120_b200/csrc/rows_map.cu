#include "rows_map.cuh"

#include <atomic>

namespace smla {

namespace {
typedef CUresult (*EncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                             const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
}  // namespace

int rows_tensor_map(const uint8_t* kv, CUtensorMap* map) {
    static std::atomic<EncodeFn> encode{nullptr};
    if (encode.load() == nullptr) {
        cudaDriverEntryPointQueryResult qres;
        void* fn = nullptr;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres) != cudaSuccess || fn == nullptr)
            return set_error(SMLA_E_DEVICE, "the driver has no cuTensorMapEncodeTiled");
        encode = (EncodeFn)fn;
    }
    const cuuint64_t dims[2] = {ROW_BYTES / 4, (cuuint64_t)NO_ROW}, strides[1] = {ROW_BYTES};
    const cuuint32_t box[2] = {32, 1}, estr[2] = {1, 1};
    const CUresult r = encode.load()(map, CU_TENSOR_MAP_DATA_TYPE_INT32, 2, const_cast<uint8_t*>(kv), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                     CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : set_error(SMLA_E_DEVICE, "cuTensorMapEncodeTiled failed (%d)", (int)r);
}

}  // namespace smla
