// The prefill attention kernel (csrc/attention_prefill.cu) with a fake of its bounded wait: in every second CTA one warp's wait for one phase of one
// barrier reports that it ran out.  Nothing else is changed; the other waits are the real ones with a limit of 2e7 cycles.
#include "common.cuh"
#include "tc_stream.cuh"

namespace sbvr {

__device__ int g_fake_warp, g_fake_bar, g_fake_parity;

__device__ __forceinline__ bool wait_that_runs_out(uint64_t* bar, uint32_t parity) {
    if ((blockIdx.x & 1) == 0 && (int)(threadIdx.x >> 5) == g_fake_warp && (int)(smem_u32(bar) & 1023) == g_fake_bar * 8 &&
        (int)parity == g_fake_parity)
        return false;
    const long long t0 = clock64();
    while (!mbar_test(bar, parity))
        if (clock64() - t0 > 20000000LL) return false;
    return true;
}

thread_local int g_last_cuda_error = 0;
bool pdl_enabled() { return true; }
int ts_map_2d(CUtensorMap* out, CUtensorMapDataType type, CUtensorMapSwizzle swizzle, const void* base, size_t rows, size_t cols, size_t pitch,
              int box_rows, int box_cols) {
    typedef CUresult (*Encode)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                               const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult found;
    SBVR_CUDA_TRY(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &found));
    const cuuint64_t dims[2] = {cols, rows}, strides[1] = {pitch};
    const cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows}, ones[2] = {1u, 1u};
    return reinterpret_cast<Encode>(fn)(out, type, 2, const_cast<void*>(base), dims, strides, box, ones, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle,
                                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
}

}  // namespace sbvr

#define mbar_wait_timed wait_that_runs_out
#include "attention_prefill.cu"

extern "C" __attribute__((visibility("default"))) int attention_with_a_wait_that_runs_out(
    const void* qkv, const void* K, const void* V, const int* positions, void* out, int tokens, int tokens_per_seq, int n_heads, int n_kv, int max_ctx,
    float scale, int warp, int bar, int parity, void* stream) {
    using namespace sbvr;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    SBVR_CUDA_TRY(cudaMemcpyToSymbol(g_fake_warp, &warp, sizeof(int)));
    SBVR_CUDA_TRY(cudaMemcpyToSymbol(g_fake_bar, &bar, sizeof(int)));
    SBVR_CUDA_TRY(cudaMemcpyToSymbol(g_fake_parity, &parity, sizeof(int)));
    const int rc = launch_attention_tc(reinterpret_cast<const __half*>(qkv), reinterpret_cast<const __half*>(K), reinterpret_cast<const __half*>(V), positions,
                                       reinterpret_cast<__half*>(out), tokens, tokens_per_seq, n_heads, n_kv, max_ctx, scale, st);
    if (rc) return rc;
    SBVR_CUDA_TRY(cudaStreamSynchronize(st));
    return 0;
}
