// Library-wide pieces of the C ABI: the per-thread error message, the device status word and the
// version string.
#include <cstdarg>
#include <cstdio>
#include <map>
#include <mutex>
#include <utility>

#include "tc5.cuh"

__device__ int g_cn_status = 0;

static thread_local char t_err[512] = "";

void cn_set_error(const char* fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(t_err, sizeof t_err, fmt, ap);
    va_end(ap);
}

// The book behind cn_allow_smem: the largest dynamic shared-memory size already allowed per (kernel, device). Returns 1
// when `bytes` is not covered yet (and records it when commit is set), 0 when it is. No CUDA call: testable without a GPU.
extern "C" int cn_smem_book(const void* kernel, int device, int bytes, int commit) {
    static std::mutex mu;
    static std::map<std::pair<const void*, int>, int> done;
    std::lock_guard<std::mutex> lock(mu);
    int& have = done[std::make_pair(kernel, device)];
    if (have >= bytes) return 0;
    if (commit) have = bytes;
    return 1;
}

cudaError_t cn_allow_smem(const void* kernel, int bytes) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (!cn_smem_book(kernel, dev, bytes, 0)) return cudaSuccess;
    // the attribute belongs to the device that is current: every GPU of a process gets its own call
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess) cn_smem_book(kernel, dev, bytes, 1);
    return e;
}

static int encode_map(CUtensorMap* map, CUtensorMapDataType type, unsigned rank, const void* base, const cuuint64_t* dims, const cuuint64_t* strides, const cuuint32_t* box,
                      CUtensorMapSwizzle swizzle) {
    typedef CUresult (*Encode)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                               const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static Encode encode = nullptr;
    if (!encode) {  // the driver's entry point, looked up once (two threads may both look: the same answer)
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult q;
        CN_CUDA(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q));
        if (!fn) CN_FAIL(CN_ERR_CUDA, "cuTensorMapEncodeTiled is not in this driver");
        encode = (Encode)fn;
    }
    const cuuint32_t es[3] = {1, 1, 1};
    const CUresult r = encode(map, type, rank, const_cast<void*>(base), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) CN_FAIL(CN_ERR_CUDA, "tensor map of [%llu x %llu]: driver error %d", (unsigned long long)dims[1], (unsigned long long)dims[0], (int)r);
    return CN_OK;
}

int cn_tmap_words(CUtensorMap* map, const void* base, unsigned long long words, unsigned long long rows, unsigned box_words, unsigned box_rows) {
    const cuuint64_t dims[2] = {words, rows}, strides[1] = {words * 4};
    const cuuint32_t box[2] = {box_words, box_rows};
    return encode_map(map, CU_TENSOR_MAP_DATA_TYPE_UINT32, 2, base, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_NONE);
}

int cn_tmap_blocks(CUtensorMap* map, const void* base, bool bf16, unsigned long long blocks, unsigned long long rows, unsigned long long row_bytes, unsigned box_rows,
                   unsigned box_blocks) {
    const cuuint64_t dims[3] = {64, rows, blocks}, strides[2] = {row_bytes, 128};
    const cuuint32_t box[3] = {64, box_rows, box_blocks};
    return encode_map(map, bf16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, base, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
}

extern "C" const char* cn_last_error_string(void) { return t_err; }

extern "C" const char* cn_version(void) { return "crownest_b200 sm_100a"; }

extern "C" int cn_device_status(int* code_out) {
    int code = 0, zero = 0;
    CN_CUDA(cudaDeviceSynchronize());
    CN_CUDA(cudaMemcpyFromSymbol(&code, g_cn_status, sizeof(int)));
    if (code) CN_CUDA(cudaMemcpyToSymbol(g_cn_status, &zero, sizeof(int)));
    if (code_out) *code_out = code;
    if (code) CN_FAIL(CN_ERR_DEVICE, "a kernel gave up a bounded wait (device code %d)", code);
    return CN_OK;
}
