// C ABI of sbvr_b200: argument validation, workspace management and dispatch.  Nothing here
// computes; see decode.cu, linear_simt.cu, linear_tcs.cu, linear_gemm.cu.
#include <cstdlib>
#include <mutex>

#include "common.cuh"

namespace sbvr {

thread_local int g_last_cuda_error = 0;

int xop_check(const XOp* xop, const __half* x, int M, int K, int* op, const __half** delta, const __half** norm_w, __half** h_out,
              float* eps) {
    *op = xop ? xop->op : SBVR_XOP_NONE;
    *delta = xop ? xop->delta : nullptr, *norm_w = xop ? xop->norm_w : nullptr, *h_out = xop ? xop->h_out : nullptr;
    *eps = xop ? xop->eps : 0.0f;
    if (*op != SBVR_XOP_ADD_RMSNORM) return SBVR_OK;
    if (!*norm_w) return SBVR_ERR_BAD_ARG;
    if (*h_out) {                                  // h_out is written while other blocks still read x and delta for the row's mean square
        const uintptr_t n = (uintptr_t)M * K * 2, ho = reinterpret_cast<uintptr_t>(*h_out);
        auto overlaps = [&](const void* q) {
            const uintptr_t a = reinterpret_cast<uintptr_t>(q);
            return q && ho < a + n && a < ho + n;
        };
        if (overlaps(x) || overlaps(*delta)) return SBVR_ERR_BAD_ARG;
    }
    if ((reinterpret_cast<uintptr_t>(*delta) | reinterpret_cast<uintptr_t>(*norm_w) | reinterpret_cast<uintptr_t>(*h_out)) & 15)
        return SBVR_ERR_ALIGN;
    return SBVR_OK;
}

bool pdl_enabled() {
    static const bool on = [] {
        const char* e = getenv("SBVR_NO_PDL");
        return !(e && e[0] == '1');
    }();
    return on;
}

int device_info(int device, DeviceInfo* out) {
    static std::mutex mu;
    static DeviceInfo cache[64];
    static bool have[64] = {false};
    if (device < 0 || device >= 64) return SBVR_ERR_BAD_ARG;
    std::lock_guard<std::mutex> lock(mu);
    if (!have[device]) {
        DeviceInfo d;
        SBVR_CUDA_TRY(cudaDeviceGetAttribute(&d.sm_count, cudaDevAttrMultiProcessorCount, device));
        SBVR_CUDA_TRY(cudaDeviceGetAttribute(&d.smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device));
        SBVR_CUDA_TRY(cudaDeviceGetAttribute(&d.l2_bytes, cudaDevAttrL2CacheSize, device));
        SBVR_CUDA_TRY(cudaDeviceGetAttribute(&d.cc_major, cudaDevAttrComputeCapabilityMajor, device));
        SBVR_CUDA_TRY(cudaDeviceGetAttribute(&d.cc_minor, cudaDevAttrComputeCapabilityMinor, device));
        cache[device] = d;
        have[device] = true;
    }
    *out = cache[device];
    return SBVR_OK;
}

static int make_packed(PackedW* w, const uint32_t* bvr, const void* coeff_idx, int idx_bytes, const void* coeff, int C,
                       int N, int K, int S, int G) {
    if (!bvr || !coeff) return SBVR_ERR_BAD_ARG;
    if (idx_bytes != 0 && idx_bytes != 1 && idx_bytes != 2) return SBVR_ERR_BAD_ARG;
    if (idx_bytes != 0 && (!coeff_idx || C < 1 || C > 65536 || (idx_bytes == 1 && C > 256))) return SBVR_ERR_BAD_ARG;
    if (N < 1 || K < 1 || S < 1 || S > 8) return SBVR_ERR_BAD_ARG;
    if (G < 32 || G % 32) return SBVR_ERR_BAD_ARG;
    if (K % G) return SBVR_ERR_SHAPE;
    if (reinterpret_cast<uintptr_t>(bvr) & 3) return SBVR_ERR_ALIGN;
    if (reinterpret_cast<uintptr_t>(coeff) & 1) return SBVR_ERR_ALIGN;
    if (idx_bytes == 2 && (reinterpret_cast<uintptr_t>(coeff_idx) & 1)) return SBVR_ERR_ALIGN;
    w->bvr = bvr, w->idx = coeff_idx, w->coeff = reinterpret_cast<const __half*>(coeff);
    w->idx_bytes = idx_bytes, w->C = C, w->N = N, w->K = K, w->S = S, w->G = G;
    return SBVR_OK;
}

}  // namespace sbvr

using namespace sbvr;

extern "C" {

const char* sbvr_strerror(int status) {
    switch (status) {
        case SBVR_OK: return "ok";
        case SBVR_ERR_BAD_ARG: return "bad argument (null pointer, non-positive size, or unsupported S / G / idx_bytes / C)";
        case SBVR_ERR_SHAPE: return "shape not supported (K must be a multiple of G)";
        case SBVR_ERR_ALIGN: return "pointer alignment too small";
        case SBVR_ERR_CUDA: return "a CUDA runtime call failed (see sbvr_last_cuda_error)";
        case SBVR_ERR_WORKSPACE: return "workspace missing or too small";
        case SBVR_ERR_TIMEOUT: return "a bounded device-side wait ran out";
        case SBVR_ERR_UNSUPPORTED: return "no kernel covers this combination of arguments";
        case SBVR_ERR_NOALLOC_LIMIT:
            return "the problem needs more scratch than the fixed 4 MiB array of sbvr_linear_f16_noalloc; use "
                   "sbvr_linear_f16 with a workspace";
        default: return "unknown status";
    }
}

int sbvr_last_cuda_error(void) { return g_last_cuda_error; }
static unsigned int g_last_timeout_where = 0, g_last_timeout_info[2] = {0, 0};
unsigned int sbvr_last_timeout_where(void) { return g_last_timeout_where; }
unsigned int sbvr_last_timeout_info(int i) { return (i == 0 || i == 1) ? g_last_timeout_info[i] : 0u; }

int sbvr_query(int device, int* sm_count, int* smem_per_block_optin, int* l2_bytes, int* cc_major, int* cc_minor) {
    DeviceInfo d;
    int rc = device_info(device, &d);
    if (rc) return rc;
    if (sm_count) *sm_count = d.sm_count;
    if (smem_per_block_optin) *smem_per_block_optin = d.smem_optin;
    if (l2_bytes) *l2_bytes = d.l2_bytes;
    if (cc_major) *cc_major = d.cc_major;
    if (cc_minor) *cc_minor = d.cc_minor;
    return SBVR_OK;
}

int sbvr_workspace_create(sbvr_workspace_t** out, int device, size_t bytes) {
    if (!out) return SBVR_ERR_BAD_ARG;
    *out = nullptr;
    if (bytes == 0) bytes = (size_t)32 << 20;
    const size_t fixed = SBVR_WS_FIXED_BYTES;
    if (bytes < fixed + 4096) return SBVR_ERR_BAD_ARG;
    int prev = 0;
    SBVR_CUDA_TRY(cudaGetDevice(&prev));
    SBVR_CUDA_TRY(cudaSetDevice(device));
    sbvr_workspace* ws = new (std::nothrow) sbvr_workspace();
    if (!ws) return SBVR_ERR_BAD_ARG;
    ws->mu = new (std::nothrow) std::recursive_mutex();
    if (!ws->mu) {
        delete ws;
        return SBVR_ERR_BAD_ARG;
    }
    ws->device = device;
    ws->bytes = bytes;
    ws->base = nullptr;
    ws->pinned_status = nullptr;
    cudaError_t e = cudaMalloc(reinterpret_cast<void**>(&ws->base), bytes);
    // The clearing runs on the legacy default stream, which streams created as non-blocking do not wait for: without the
    // synchronisation a first kernel on such a stream could leave tags and counts that the clearing then erased, and its
    // waits ran out.
    if (e == cudaSuccess) e = cudaMemset(ws->base, 0, fixed);
    if (e == cudaSuccess) e = cudaStreamSynchronize(cudaStreamLegacy);
    if (e == cudaSuccess) e = cudaMallocHost(&ws->pinned_status, 16);
    if (e != cudaSuccess) {
        g_last_cuda_error = (int)e;
        (void)cudaGetLastError();
        if (ws->base) cudaFree(ws->base);
        delete ws->mu;
        delete ws;
        cudaSetDevice(prev);
        return SBVR_ERR_CUDA;
    }
    ws->status = reinterpret_cast<unsigned int*>(ws->base);
    ws->counters = reinterpret_cast<unsigned int*>(ws->base + 256);
    ws->xchg = reinterpret_cast<unsigned long long*>(ws->base + 256 + (size_t)SBVR_WS_COUNTERS * 4);
    ws->dyn = ws->base + fixed;
    ws->dyn_bytes = bytes - fixed;
    *out = ws;                                     // the workspace exists whatever happens to the device switch below
    SBVR_CUDA_TRY(cudaSetDevice(prev));
    return SBVR_OK;
}

int sbvr_workspace_bytes(int device, int M, int N, int K, size_t* bytes) {
    if (!bytes || M < 1 || N < 1 || K < 1) return SBVR_ERR_BAD_ARG;
    DeviceInfo di;
    int rc = device_info(device, &di);
    if (rc) return rc;
    PackedW w;
    w.bvr = nullptr, w.idx = nullptr, w.coeff = nullptr, w.idx_bytes = 0, w.C = 0;
    w.N = N, w.K = K, w.S = 4, w.G = 256;
    const size_t fixed = SBVR_WS_FIXED_BYTES;
    const size_t stage = (((size_t)M * K * 2 + 255) / 256 + ((size_t)M * N * 2 + 255) / 256) * 256;   // host-pointer staging
    size_t kern = linear_gemm_workspace_bytes(w, M, di.sm_count);
    if (M >= 2 && M <= 16 && K % 256 == 0) {       // the small-batch kernel's digits and partial sums, whatever the encoding
        for (int s = 2; s <= 4; ++s)
            for (int g = 128; g <= 256; g += 128) {
                w.S = s, w.G = g;
                const size_t sb = linear_sb_workspace_bytes(w, di);
                if (sb > kern) kern = sb;
            }
    }
    *bytes = fixed + kern + stage + ((size_t)8 << 20);
    if (*bytes < ((size_t)32 << 20)) *bytes = (size_t)32 << 20;
    return SBVR_OK;
}

int sbvr_linear_folds(int device, int M, int N, int K, int S, int G, int idx_bytes, int* folds) {
    if (!folds || M < 1 || N < 1 || K < 1) return SBVR_ERR_BAD_ARG;
    DeviceInfo di;
    const int rc = device_info(device, &di);
    if (rc) return rc;
    PackedW w;
    w.bvr = nullptr, w.idx = nullptr, w.coeff = nullptr, w.idx_bytes = idx_bytes, w.C = 0;
    w.N = N, w.K = K, w.S = S, w.G = G;
    *folds = M <= 4 || (M <= 16 && S >= 2 && S <= 4 && (G == 128 || G == 256) && K % 256 == 0 && linear_sb_preferred(w, M, di));
    return SBVR_OK;
}

int sbvr_linear_workspace_bytes(int device, const uint32_t* bvr, const void* coeff_idx, int idx_bytes, const void* coeff, int C,
                                int M, int N, int K, int S, int G, size_t* bytes) {
    PackedW w;
    const int rc = make_packed(&w, bvr, coeff_idx, idx_bytes, coeff, C, N, K, S, G);
    if (rc) return rc;
    if (!bytes || M < 1) return SBVR_ERR_BAD_ARG;
    *bytes = 0;
    return linear_tcs_supported(w, M) ? SBVR_OK : sbvr_workspace_bytes(device, M, N, K, bytes);
}

int sbvr_workspace_destroy(sbvr_workspace_t* ws) {
    if (!ws) return SBVR_OK;
    int prev = 0;
    cudaGetDevice(&prev);
    cudaSetDevice(ws->device);
    if (ws->base) cudaFree(ws->base);
    if (ws->pinned_status) cudaFreeHost(ws->pinned_status);
    cudaSetDevice(prev);
    delete ws->mu;
    delete ws;
    return SBVR_OK;
}

int sbvr_workspace_patience(sbvr_workspace_t* ws, unsigned int cycles) {
    if (!ws) return SBVR_ERR_BAD_ARG;
    WsLock lock(ws);
    ws->patience = cycles;
    return SBVR_OK;
}

int sbvr_workspace_status(sbvr_workspace_t* ws, sbvr_stream_t stream) {
    if (!ws) return SBVR_ERR_BAD_ARG;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    unsigned int* h = reinterpret_cast<unsigned int*>(ws->pinned_status);
    SBVR_CUDA_TRY(cudaMemcpyAsync(h, ws->status, 16, cudaMemcpyDeviceToHost, st));
    SBVR_CUDA_TRY(cudaStreamSynchronize(st));
    if (h[0] != 0) {
        g_last_timeout_where = h[1];
        g_last_timeout_info[0] = h[2], g_last_timeout_info[1] = h[3];
        // a kernel gave up: its arrival counters may be half-way; clear everything for the next call
        SBVR_CUDA_TRY(cudaMemsetAsync(ws->base, 0, SBVR_WS_FIXED_BYTES, st));
        SBVR_CUDA_TRY(cudaStreamSynchronize(st));
        return SBVR_ERR_TIMEOUT;
    }
    return SBVR_OK;
}

int sbvr_decode_f16(const uint32_t* bvr, const void* coeff_idx, int idx_bytes, const void* coeff, int C, void* W,
                    int ldw, int N, int K, int K_out, int S, int G, sbvr_stream_t stream) {
    PackedW w;
    int rc = make_packed(&w, bvr, coeff_idx, idx_bytes, coeff, C, N, K, S, G);
    if (rc) return rc;
    if (!W || K_out < 1 || K_out > K || ldw < K_out) return SBVR_ERR_BAD_ARG;
    if (reinterpret_cast<uintptr_t>(W) & 1) return SBVR_ERR_ALIGN;
    return launch_decode(w, reinterpret_cast<__half*>(W), ldw, K_out, reinterpret_cast<cudaStream_t>(stream));
}

// Rows of Kin <= K elements; see sbvr_linear_padded_f16.
static int linear_any(const void* x, int Kin, const uint32_t* bvr, const void* coeff_idx, int idx_bytes, const void* coeff, int C,
                      const void* bias, void* y, int M, int N, int K, int S, int G, int algo, const sbvr_workspace* ws,
                      sbvr_stream_t stream) {
    PackedW w;
    int rc = make_packed(&w, bvr, coeff_idx, idx_bytes, coeff, C, N, K, S, G);
    if (rc) return rc;
    if (!x || !y || M < 1 || Kin < 1 || Kin > K) return SBVR_ERR_BAD_ARG;
    if ((reinterpret_cast<uintptr_t>(x) & (Kin == K ? 3 : 1)) || (reinterpret_cast<uintptr_t>(y) & 1)) return SBVR_ERR_ALIGN;
    if (algo < 0 || algo > 4) return SBVR_ERR_BAD_ARG;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const __half* xh = reinterpret_cast<const __half*>(x);
    const __half* bh = reinterpret_cast<const __half*>(bias);
    __half* yh = reinterpret_cast<__half*>(y);
    WsLock lock(ws);
    // padded rows, where a kernel needs them, live at the end of the workspace, away from the kernels' scratch
    sbvr_workspace shrunk;
    size_t padded = 0;
    if (Kin != K) {
        if (!ws) return SBVR_ERR_WORKSPACE;
        padded = ((size_t)M * K * 2 + 255) / 256 * 256;
        if (padded > ws->dyn_bytes) return SBVR_ERR_WORKSPACE;
        shrunk = *ws;
        shrunk.dyn_bytes = (ws->dyn_bytes - padded) / 256 * 256;
        ws = &shrunk;
    }
    const bool chosen = algo == 0;
    if (algo == 0) {
        DeviceInfo di;
        algo = 1;
        if (ws && device_info(ws->device, &di) == SBVR_OK && di.cc_major == 10) {
            if (linear_tcs_supported(w, M) && (Kin != K || !(reinterpret_cast<uintptr_t>(x) & 15)) &&
                linear_tcs_workspace_bytes(w, M, di.sm_count) <= ws->dyn_bytes) algo = 2;
            else if (M <= 16 && linear_sb_supported(w, M) && linear_sb_preferred(w, M, di) && linear_sb_workspace_bytes(w, di) <= ws->dyn_bytes)
                algo = 4;
            // A small problem is done by the SIMT kernel's one launch before the GEMM's second has started: measured 2.8 against
            // 5.7 us at 64 x 128 (M = 1), 5.2 against 9.8 at 300 x 512 (M = 8), 7.0 against 8.2 at 3000 x 1024 (M = 4), but 22
            // against 12 at 3000 x 3072.  Its time is that of K x (blocks of four rows) as long as all blocks run at once.
            else if ((long long)K * ((M + 3) / 4) <= 1024 && (long long)((N + 31) / 32) * ((M + 3) / 4) <= 4LL * di.sm_count) algo = 1;
            else if (linear_gemm_supported(w, M) &&
                     linear_gemm_workspace_bytes(w, M, di.sm_count) <= ws->dyn_bytes) algo = 3;
        }
    }
    // Algo 4 takes up to 32 rows (16 with groups of 128); beyond sixteen the GEMM does the work, on the weights the kernel takes.  The
    // form that the kernel once had for them (six digits) took 37 us at 14336 x 4096, M = 32, S = 4, 51 at 4096 x 14336 and 17.4 at 4096 x
    // 4096; the GEMM takes 28, 27 and 15.
    if (algo == 4 && M > 16) {
        if (M > 32 || w.G != 256 || !linear_sb_supported(w, 16)) return SBVR_ERR_UNSUPPORTED;
        algo = 3;
    }
    if (Kin != K && algo != 3) {                   // the GEMM pads where it has to
        __half* xd = reinterpret_cast<__half*>(ws->dyn + ws->dyn_bytes);
        rc = launch_pad_rows(xh, xd, M, Kin, K, st);
        if (rc) return rc;
        xh = xd;
    }
    if (algo == 2) {
        if (!ws) return SBVR_ERR_WORKSPACE;
        return launch_linear_tcs(xh, w, bh, yh, M, ws->device, ws->status, ws->xchg, ws->dyn, ws->dyn_bytes, st);
    }
    if (algo == 3) return launch_linear_gemm(xh, Kin, w, bh, yh, M, ws, st);
    if (algo == 4) {
        if (!ws) return SBVR_ERR_WORKSPACE;
        return launch_linear_sb(xh, w, bh, yh, M, ws->device, ws->status, reinterpret_cast<float*>(ws->xchg),
                                reinterpret_cast<unsigned long long*>(ws->counters), ws->patience, ws->dyn, ws->dyn_bytes, chosen, st);
    }
    return launch_linear_simt(xh, w, bh, yh, M, st);
}

int sbvr_linear_f16(const void* x, const uint32_t* bvr, const void* coeff_idx, int idx_bytes, const void* coeff, int C,
                    const void* bias, void* y, int M, int N, int K, int S, int G, int algo, sbvr_workspace_t* ws,
                    sbvr_stream_t stream) {
    return linear_any(x, K, bvr, coeff_idx, idx_bytes, coeff, C, bias, y, M, N, K, S, G, algo, ws, stream);
}

int sbvr_linear_padded_f16(const void* x, int K_in, const uint32_t* bvr, const void* coeff_idx, int idx_bytes, const void* coeff,
                           int C, const void* bias, void* y, int M, int N, int K, int S, int G, int algo, sbvr_workspace_t* ws,
                           sbvr_stream_t stream) {
    return linear_any(x, K_in, bvr, coeff_idx, idx_bytes, coeff, C, bias, y, M, N, K, S, G, algo, ws, stream);
}

int sbvr_linear_fused_f16(int x_op, const void* x, const void* delta, const void* norm_weight, void* h_out, float eps,
                          const uint32_t* bvr, const void* coeff_idx, int idx_bytes, const void* coeff, int C,
                          const void* bias, void* y, int M, int N, int K, int S, int G, sbvr_workspace_t* ws,
                          sbvr_stream_t stream) {
    PackedW w;
    int rc = make_packed(&w, bvr, coeff_idx, idx_bytes, coeff, C, N, K, S, G);
    if (rc) return rc;
    if (!x || !y || M < 1) return SBVR_ERR_BAD_ARG;
    if (x_op != SBVR_XOP_SILU_MUL && x_op != SBVR_XOP_ADD_RMSNORM && x_op != SBVR_XOP_DIGITS) return SBVR_ERR_BAD_ARG;
    if ((reinterpret_cast<uintptr_t>(x) & 15) || (reinterpret_cast<uintptr_t>(y) & 1)) return SBVR_ERR_ALIGN;
    DeviceInfo di;
    if (!ws) return SBVR_ERR_WORKSPACE;
    rc = device_info(ws->device, &di);
    if (rc) return rc;
    if (di.cc_major != 10) return SBVR_ERR_UNSUPPORTED;
    XOp xop;
    xop.op = x_op;
    xop.delta = reinterpret_cast<const __half*>(delta), xop.norm_w = reinterpret_cast<const __half*>(norm_weight);
    xop.h_out = reinterpret_cast<__half*>(h_out), xop.eps = eps;
    WsLock lock(ws);
    if (!linear_tcs_supported(w, M)) {             // more rows (or digits that do not fit the GEMV): the small-batch kernel
        if (x_op == SBVR_XOP_DIGITS || M > 16 || !linear_sb_supported(w, M)) return SBVR_ERR_UNSUPPORTED;
        if (linear_sb_workspace_bytes(w, di) > ws->dyn_bytes) return SBVR_ERR_WORKSPACE;
        return launch_linear_sb(reinterpret_cast<const __half*>(x), w, reinterpret_cast<const __half*>(bias),
                                reinterpret_cast<__half*>(y), M, ws->device, ws->status, reinterpret_cast<float*>(ws->xchg),
                                reinterpret_cast<unsigned long long*>(ws->counters), ws->patience, ws->dyn, ws->dyn_bytes, true, reinterpret_cast<cudaStream_t>(stream), &xop);
    }
    if (linear_tcs_workspace_bytes(w, M, di.sm_count) > ws->dyn_bytes) return SBVR_ERR_WORKSPACE;
    return launch_linear_tcs(reinterpret_cast<const __half*>(x), w, reinterpret_cast<const __half*>(bias),
                             reinterpret_cast<__half*>(y), M, ws->device, ws->status, ws->xchg, ws->dyn,
                             ws->dyn_bytes, reinterpret_cast<cudaStream_t>(stream), &xop);
}

int sbvr_linear_push_f16(int x_op, const void* x, const void* delta, const void* norm_weight, void* h_out, float eps,
                         const uint32_t* bvr, const void* coeff_idx, int idx_bytes, const void* coeff, int C,
                         const void* bias, const sbvr_push_desc_t* push_desc_dev, int M, int N, int K, int S, int G,
                         sbvr_workspace_t* ws, sbvr_stream_t stream) {
    PackedW w;
    int rc = make_packed(&w, bvr, coeff_idx, idx_bytes, coeff, C, N, K, S, G);
    if (rc) return rc;
    if (!x || !push_desc_dev || M < 1) return SBVR_ERR_BAD_ARG;
    if (x_op != SBVR_XOP_NONE && x_op != SBVR_XOP_SILU_MUL && x_op != SBVR_XOP_ADD_RMSNORM) return SBVR_ERR_BAD_ARG;
    if ((reinterpret_cast<uintptr_t>(x) & 15) || (reinterpret_cast<uintptr_t>(push_desc_dev) & 7)) return SBVR_ERR_ALIGN;
    DeviceInfo di;
    if (!ws) return SBVR_ERR_WORKSPACE;
    rc = device_info(ws->device, &di);
    if (rc) return rc;
    if (di.cc_major != 10) return SBVR_ERR_UNSUPPORTED;
    if (G != 256 || !linear_tcs_supported(w, M)) return SBVR_ERR_UNSUPPORTED;
    WsLock lock(ws);
    if (linear_tcs_workspace_bytes(w, M, di.sm_count) > ws->dyn_bytes) return SBVR_ERR_WORKSPACE;
    XOp xop;
    xop.op = x_op;
    xop.delta = reinterpret_cast<const __half*>(delta), xop.norm_w = reinterpret_cast<const __half*>(norm_weight);
    xop.h_out = reinterpret_cast<__half*>(h_out), xop.eps = eps;
    return launch_linear_tcs(reinterpret_cast<const __half*>(x), w, reinterpret_cast<const __half*>(bias), nullptr, M,
                             ws->device, ws->status, ws->xchg, ws->dyn, ws->dyn_bytes, reinterpret_cast<cudaStream_t>(stream),
                             x_op == SBVR_XOP_NONE ? nullptr : &xop, push_desc_dev);
}

int sbvr_linear_f16_host(const void* x_host, const uint32_t* bvr, const void* coeff_idx, int idx_bytes,
                         const void* coeff, int C, const void* bias, void* y_host, int M, int N, int K, int S, int G,
                         int algo, sbvr_workspace_t* ws, sbvr_stream_t stream) {
    if (!ws || !x_host || !y_host || M < 1 || N < 1 || K < 1) return SBVR_ERR_BAD_ARG;
    // staging buffers for x and y live at the end of the workspace
    const size_t xb = ((size_t)M * K * 2 + 255) / 256 * 256, yb = ((size_t)M * N * 2 + 255) / 256 * 256;
    if (xb + yb + ((size_t)8 << 20) > ws->dyn_bytes) return SBVR_ERR_WORKSPACE;
    char* xd = ws->dyn + ws->dyn_bytes - xb - yb;
    char* yd = xd + xb;
    WsLock lock(ws);
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    SBVR_CUDA_TRY(cudaMemcpyAsync(xd, x_host, (size_t)M * K * 2, cudaMemcpyHostToDevice, st));
    sbvr_workspace shrunk = *ws;                 // keep the kernels' scratch away from the staging buffers
    shrunk.dyn_bytes = ws->dyn_bytes - xb - yb;
    int rc = sbvr_linear_f16(xd, bvr, coeff_idx, idx_bytes, coeff, C, bias, yd, M, N, K, S, G, algo, &shrunk, stream);
    if (rc) return rc;
    SBVR_CUDA_TRY(cudaMemcpyAsync(y_host, yd, (size_t)M * N * 2, cudaMemcpyDeviceToHost, st));
    return SBVR_OK;
}

}  // extern "C"
