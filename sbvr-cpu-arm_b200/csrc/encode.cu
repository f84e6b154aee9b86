// The arithmetic core of the SBVR encoder: for groups of 256 fp16 values and candidate coefficient lines, the mean
// squared error of representing every value by the nearest of the 2^S sums a line can form, the selector of that
// nearest sum, and the packing of selectors into bit-planes.
//
// The reference evaluates a candidate set by materialising diff[c, e, j] = (data[e] - point[c, j])^2 as an fp16 tensor,
// taking the minimum over j and the fp32 mean over e (sbvr/core.py:485-500, `_data_diff_min_mse`; points =
// search_matrix @ bin_combs^T, :520-521), one group at a time in a Python loop.  Here one thread owns one (group,
// candidate) pair, keeps the 2^S points in registers and streams the group from shared memory: nothing of size
// candidates x 256 x 2^S ever exists, and many groups are evaluated against the codebook in one launch.
//
// Arithmetic, step for step as the reference's tensor ops round:
//   point[j] = fp16( fp32 sum over s, in order, of line[s] * bit_s(j) ),  bit_s(j) = (j >> (S-1-s)) & 1  (bin_combs, :345-351)
//   diff     = fp16( fp16(d - point)^2 )                                  (fp16 subtraction, fp16 square)
//   m[e]     = min over j of diff (the first j on ties)                   (fp16 min)
//   mse      = (fp32 sum over e of m[e]) / 256                            (`.to(float32).mean`)
#include "common.cuh"

namespace sbvr {

constexpr int ENC_G = 256;            // group length (the reference enforces 256, sbvr/core.py:222)
constexpr int ENC_THREADS = 128;

template <int S>
__device__ __forceinline__ void enc_points(const __half* line, __half2 (&pt)[1 << S]) {
    float c[S];
#pragma unroll
    for (int s = 0; s < S; ++s) c[s] = __half2float(line[s]);
#pragma unroll
    for (int j = 0; j < (1 << S); ++j) {
        float v = 0.0f;
#pragma unroll
        for (int s = 0; s < S; ++s)
            if ((j >> (S - 1 - s)) & 1) v += c[s];
        pt[j] = __half2half2(__float2half_rn(v));
    }
}

// mse[b, c] for b < B groups and c < L lines.  grid = (ceil(L / 128), B).
template <int S>
__global__ void __launch_bounds__(ENC_THREADS) encode_mse_kernel(const __half* __restrict__ data,
                                                                 const __half* __restrict__ lines, int L,
                                                                 float* __restrict__ mse) {
    __shared__ __align__(16) __half2 ds[ENC_G / 2];
    const int b = blockIdx.y;
    for (int i = threadIdx.x; i < ENC_G / 2; i += ENC_THREADS)
        ds[i] = reinterpret_cast<const __half2*>(data + (size_t)b * ENC_G)[i];
    __syncthreads();
    const int c = blockIdx.x * ENC_THREADS + threadIdx.x;
    if (c >= L) return;
    __half2 pt[1 << S];
    enc_points<S>(lines + (size_t)c * S, pt);
    float s0 = 0.0f, s1 = 0.0f;
#pragma unroll 4
    for (int i = 0; i < ENC_G / 2; ++i) {
        const __half2 d = ds[i];
        __half2 t = __hsub2(d, pt[0]);
        __half2 m = __hmul2(t, t);
#pragma unroll
        for (int j = 1; j < (1 << S); ++j) {
            t = __hsub2(d, pt[j]);
            m = __hmin2(m, __hmul2(t, t));
        }
        const float2 f = __half22float2(m);
        s0 += f.x, s1 += f.y;
    }
    mse[(size_t)b * L + c] = (s0 + s1) * (1.0f / ENC_G);
}

// sel[b, e] = first j minimising fp16((d - point_j)^2) for the line `which[b]` of `lines`.  grid = B, block = 256.
template <int S>
__global__ void __launch_bounds__(ENC_G) encode_select_kernel(const __half* __restrict__ data,
                                                              const __half* __restrict__ lines,
                                                              const int* __restrict__ which, uint8_t* __restrict__ sel) {
    const int b = blockIdx.x, e = threadIdx.x;
    __half2 pt[1 << S];
    enc_points<S>(lines + (size_t)which[b] * S, pt);
    const __half d = data[(size_t)b * ENC_G + e];
    int best = 0;
    __half t = __hsub(d, __low2half(pt[0]));
    __half bm = __hmul(t, t);
#pragma unroll
    for (int j = 1; j < (1 << S); ++j) {
        t = __hsub(d, __low2half(pt[j]));
        const __half v = __hmul(t, t);
        if (__hlt(v, bm)) bm = v, best = j;
    }
    sel[(size_t)b * ENC_G + e] = (uint8_t)best;
}

// ---------------------------------------------------------------------------------------------
// The walk over the groups (sbvr/core.py:555-653), one launch sequence per group that misses the codebook.
//
// Which group misses next depends on the codebook as its predecessors left it, but what a group's best stored line is does
// not depend on how it is found: best_mse / best_at hold it for every undecided group, a new line is compared with the
// undecided groups only, and the first group whose best is not below the cut-off is the next miss.  Its own search space
// (sbvr/core.py:368-483) is generated and evaluated in the search kernel, one thread per candidate line, and only the winner
// comes back: a step of the walk is three launches and one synchronisation, where the same step in tensor operations was
// some sixty launches and a dozen synchronisations (1.2 ms).
//
// The roundings of the candidates are those of the tensor operations they replace, on the GPU: `arange` in fp16 is
// fp16(start + step * i) with one fp32 rounding in between, `linspace` in fp16 rounds its step, the product and the sum to
// fp16 and counts the second half from the end, a division by a Python number is a product with its fp32 reciprocal.
//
// Exactness of what is left out.  The nearest sum of a value has the smallest fp16((d - p)^2) because both roundings are
// monotone: the minimum is taken over |d - p| and squared once.  An mse is a sum of non-negative terms added in a fixed
// order, and fp32 addition is monotone: a candidate whose partial sum exceeds the best mse so far cannot win (an equal one
// may, by its index, and is kept).
// ---------------------------------------------------------------------------------------------
struct EncStats {
    float d_max, d_min, d_95, d_avg;
};

__device__ __forceinline__ float enc_h(float v) { return __half2float(__float2half_rn(v)); }

// The least |d - p| of a pair of values over the 2^S points, squared, as fp16 pair
template <int S>
__device__ __forceinline__ float2 enc_err(__half2 d, const __half2 (&pt)[1 << S]) {
    __half2 m = __habs2(__hsub2(d, pt[0]));
#pragma unroll
    for (int j = 1; j < (1 << S); ++j) m = __hmin2(m, __habs2(__hsub2(d, pt[j])));
    return __half22float2(__hmul2(m, m));
}

// Maximum, minimum, 95 % quantile (between the 14th and the 13th largest of 256, sorted position 242.25) and mean of every
// group: one warp per group.
__global__ void __launch_bounds__(256) encode_stats_kernel(const __half* __restrict__ data, int NG, EncStats* __restrict__ st) {
    const int g = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (g >= NG) return;
    const uint4 v = reinterpret_cast<const uint4*>(data + (size_t)g * ENC_G)[lane];
    const __half* h = reinterpret_cast<const __half*>(&v);
    uint32_t key[8];                               // order-preserving 16 bits | a number of its own per element
    float sum = 0.0f, lo = INFINITY;
    bool finite = true;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        const uint32_t b = __half_as_ushort(h[e]);
        key[e] = (((b & 0x8000u) ? ~b : (b | 0x8000u)) << 16) | (uint32_t)(lane * 8 + e);
        const float f = __half2float(h[e]);
        finite = finite && fabsf(f) < INFINITY;
        sum += f;
        lo = fminf(lo, f);
    }
    float q[2] = {0.0f, 0.0f}, hi = 0.0f;
#pragma unroll 1
    for (int r = 0; r < 14; ++r) {
        uint32_t m = 0;
#pragma unroll
        for (int e = 0; e < 8; ++e) m = max(m, key[e]);
        m = __reduce_max_sync(0xffffffffu, m);
#pragma unroll
        for (int e = 0; e < 8; ++e)
            if (key[e] == m) key[e] = 0;
        const uint32_t b = m >> 16;
        const float f = __half2float(__ushort_as_half((unsigned short)((b & 0x8000u) ? (b & 0x7FFFu) : ~b)));
        if (r == 0) hi = f;
        if (r >= 12) q[r - 12] = f;
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        sum += __shfl_xor_sync(0xffffffffu, sum, o);
        lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    }
    finite = __all_sync(0xffffffffu, finite);
    if (lane == 0) {
        EncStats s;
        s.d_max = hi, s.d_min = lo, s.d_95 = q[1] + 0.25f * (q[0] - q[1]);
        s.d_avg = finite ? sum * (1.0f / ENC_G) : INFINITY;
        st[g] = s;
    }
}

// Lines [line0, line1) against the groups from `from` on; then the first of them whose best is not below the cut-off.
template <int S>
__global__ void __launch_bounds__(32) encode_update_kernel(const __half* __restrict__ data, int NG, int from,
                                                           const __half* __restrict__ lines, int line0, int line1,
                                                           float* __restrict__ best_mse, int* __restrict__ best_at, double cutoff,
                                                           int* __restrict__ miss) {
    const int g = from + blockIdx.x * 32 + threadIdx.x;
    bool missing = false;
    if (g < NG) {
        float best = best_mse[g];
        int at = -1;
        const uint4* row = reinterpret_cast<const uint4*>(data + (size_t)g * ENC_G);
        for (int n = line0; n < line1; ++n) {
            __half2 pt[1 << S];
            enc_points<S>(lines + (size_t)n * S, pt);
            float s0 = 0.0f, s1 = 0.0f;
#pragma unroll 1
            for (int i = 0; i < ENC_G / 8; ++i) {
                const uint4 v = __ldg(row + i);
                const __half2* d = reinterpret_cast<const __half2*>(&v);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float2 f = enc_err<S>(d[e], pt);
                    s0 += f.x, s1 += f.y;
                }
                if ((s0 + s1) * (1.0f / ENC_G) > best) break;
            }
            const float mse = (s0 + s1) * (1.0f / ENC_G);
            if (mse < best) best = mse, at = n;
        }
        if (at >= 0) best_mse[g] = best, best_at[g] = at;
        missing = !((double)best < cutoff);
    }
    const unsigned int m = __ballot_sync(0xffffffffu, missing);
    if (m && threadIdx.x == 0) atomicMin(miss, from + (int)blockIdx.x * 32 + __ffs((int)m) - 1);
}

// One set of search-space constants (plain, extended): scaled power lines and biases as fp16 tables, steps.
struct EncSpace {
    const __half* unit;      // [R][S]: (1, r, r^2, ..) / span of their sums
    const __half* bias;      // [B]
    int R, B, per_dim;       // per_dim: intervals per axis of the grid
    float inv_s, inv_ext;    // 1 / s_search_num, 1 / extend_ratio (1 where not extended)
};
struct EncSearch {
    const __half* data;
    const EncStats* stats;
    const float* best_mse;
    const int* best_at;
    const int* miss;               // the group to search
    unsigned long long* best;      // (mse bits << 32 | candidate), reset by the kernel in front
    unsigned int* done;            // blocks that have finished
    sbvr_encode_result_t* result;
    EncSpace space[2];
    int NG, warm, misses;
};

__device__ __forceinline__ float enc_linspace(float start, float end, int steps, int i) {
    const float step = enc_h(enc_h(end - start) / enc_h((float)(steps - 1)));
    return (i < steps / 2) ? enc_h(start + enc_h(step * enc_h((float)i))) : enc_h(end - enc_h(step * enc_h((float)(steps - i - 1))));
}

// Candidate `c` of the group's space, in the order the reference lists them; not sorted.
template <int S>
__device__ __forceinline__ void enc_candidate(const EncSpace& sp, int c, int ns, float s_start, float s_step, const float (&a0)[S],
                                              const float (&a1)[S], float (&line)[S]) {
    const int nline = sp.B * ns * sp.R;
    if (c < nline) {
        const int r = c % sp.R, bs = c / sp.R, si = bs % ns, b = bs / ns;
        const float sv = enc_h(fmaf(s_step, (float)si, s_start));
        const float bv = __half2float(sp.bias[b]);
#pragma unroll
        for (int s = 0; s < S; ++s) line[s] = enc_h(bv + enc_h(sv * __half2float(sp.unit[r * S + s])));
    } else {
        int q = c - nline;
#pragma unroll
        for (int s = S - 1; s >= 0; --s) {
            line[s] = enc_linspace(a0[s], a1[s], sp.per_dim + 1, q % (sp.per_dim + 1));
            q /= sp.per_dim + 1;
        }
    }
}

template <int S>
__global__ void __launch_bounds__(ENC_THREADS) encode_search_kernel(const EncSearch p) {
    __shared__ __align__(16) __half2 ds[ENC_G / 2];
    __shared__ unsigned int last_s;
    const int g = *p.miss;
    if (g >= p.NG) {                               // every group is decided
        if (blockIdx.x == 0 && threadIdx.x == 0) p.result->group = p.NG, p.result->status = 0;
        return;
    }
    const EncStats st = p.stats[g];
    const float cached = p.warm ? INFINITY : p.best_mse[g];
    // extended search while the codebook serves well: hits / seen > 0.6
    const bool ext = p.warm || (double)(g - p.misses) / (double)(g + 1) > 0.6;
    const EncSpace& sp = p.space[ext ? 1 : 0];
    const float s_hi = enc_h(enc_h(st.d_max - st.d_min) * 1.1f), s_lo = 2.0f * st.d_95;
    float s_step = __fmul_rn(s_hi - s_lo, sp.inv_s);           // products and sums rounded separately
    if (ext) s_step = __fmul_rn(s_step, sp.inv_ext);
    const float s_start = __fadd_rn(s_lo, s_step), s_end = __fadd_rn(s_hi, s_step);
    const double count = ceil(((double)s_end - (double)s_start) / (double)s_step);
    // what the tables do not cover (a mean that widens the biases, values that are not finite, an empty range) is the caller's
    if (!(fabsf(st.d_avg) * 2.0f / S < 0.295f) || !(s_step > 0.0f) || !(count >= 1.0 && count <= 1024.0)) {
        if (blockIdx.x == 0 && threadIdx.x == 0)
            p.result->group = g, p.result->status = 2, p.result->cached_mse = cached, p.result->cached_at = p.warm ? -1 : p.best_at[g];
        return;
    }
    const int ns = (int)count;
    float a0[S], a1[S];
#pragma unroll
    for (int s = 0; s < S; ++s) {
        const float e0 = enc_linspace(st.d_min, st.d_max, S + 1, s), e1 = enc_linspace(st.d_min, st.d_max, S + 1, s + 1);
        const float slack = enc_h(fabsf(e0) * 0.8f);
        a0[s] = enc_h(e0 - slack), a1[s] = enc_h(e1 + slack);
    }
    int total = 1;
#pragma unroll
    for (int s = 0; s < S; ++s) total *= sp.per_dim + 1;
    total += sp.B * ns * sp.R;
    for (int i = threadIdx.x; i < ENC_G / 2; i += ENC_THREADS) ds[i] = reinterpret_cast<const __half2*>(p.data + (size_t)g * ENC_G)[i];
    __syncthreads();
    const unsigned long long start_key = (unsigned long long)__float_as_uint(cached) << 32;
    for (int c = blockIdx.x * ENC_THREADS + threadIdx.x; c - (int)threadIdx.x < total; c += gridDim.x * ENC_THREADS) {
        float line[S];
        enc_candidate<S>(sp, min(c, total - 1), ns, s_start, s_step, a0, a1, line);
        // sums are formed in the order of the sorted line
#pragma unroll
        for (int i = 0; i < S; ++i)
#pragma unroll
            for (int j = 0; j + 1 < S - i; ++j)
                if (fabsf(line[j]) > fabsf(line[j + 1])) {
                    const float t = line[j];
                    line[j] = line[j + 1], line[j + 1] = t;
                }
        __half2 pt[1 << S];
#pragma unroll
        for (int j = 0; j < (1 << S); ++j) {
            float v = 0.0f;
#pragma unroll
            for (int s = 0; s < S; ++s)
                if ((j >> (S - 1 - s)) & 1) v += line[s];
            pt[j] = __half2half2(__float2half_rn(v));
        }
        float s0 = 0.0f, s1 = 0.0f;
        bool alive = c < total;
        for (int i = 0; i < ENC_G / 2; i += 8) {
            const float bound = __uint_as_float((unsigned int)(__ldcg(p.best) >> 32));
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const float2 f = enc_err<S>(ds[i + e], pt);
                s0 += f.x, s1 += f.y;
            }
            if ((s0 + s1) * (1.0f / ENC_G) > fminf(bound, cached)) alive = false;
            if (!__any_sync(0xffffffffu, alive)) break;
        }
        if (alive) {
            const unsigned long long key = ((unsigned long long)__float_as_uint((s0 + s1) * (1.0f / ENC_G)) << 32) | (unsigned int)c;
            if (key < start_key && key < __ldcg(p.best)) atomicMin(p.best, key);
        }
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last_s = (atomicAdd(p.done, 1u) == gridDim.x - 1) ? 1u : 0u;
    __syncthreads();
    if (last_s && threadIdx.x == 0) {
        __threadfence();
        const unsigned long long key = __ldcg(p.best);
        sbvr_encode_result_t* r = p.result;
        r->group = g;
        r->cached_mse = cached, r->cached_at = p.warm ? -1 : p.best_at[g];
        r->status = (key < start_key) ? 1 : 0;
        r->mse = __uint_as_float((unsigned int)(key >> 32));
        float line[S];
        enc_candidate<S>(sp, (key < start_key) ? (int)(key & 0xffffffffu) : 0, ns, s_start, s_step, a0, a1, line);
#pragma unroll
        for (int s = 0; s < S; ++s) r->line[s] = __half_as_ushort(__float2half_rn(line[s]));
    }
}

// device scratch of a walk: [0] next miss, [1] finished blocks, [2..3] best key
__global__ void encode_reset_kernel(int* scratch, int miss, __half* line, uint2 bits, int S) {
    for (int i = 0; i < S; ++i)                    // the line the caller appends to the codebook (S = 0: none)
        line[i] = __ushort_as_half((unsigned short)(((i & 2) ? bits.y : bits.x) >> (16 * (i & 1))));
    scratch[0] = miss;
    scratch[1] = 0;
    reinterpret_cast<unsigned long long*>(scratch)[1] = ~0ull;
}
// the group the scan found, for a caller that searches it himself
__global__ void encode_report_kernel(const int* scratch, const float* best_mse, const int* best_at, int NG, int warm,
                                     sbvr_encode_result_t* r) {
    const int g = scratch[0];
    r->group = g < NG ? g : NG;
    r->status = g < NG ? 2 : 0;
    r->cached_mse = (g < NG && !warm) ? best_mse[g] : INFINITY;
    r->cached_at = (g < NG && !warm) ? best_at[g] : -1;
}

template <int S>
static int encode_advance(const sbvr_encode_walk_t& w, int sm_count, cudaStream_t st) {
    int* scratch = reinterpret_cast<int*>(w.scratch);
    const int from = w.from;
    const bool app = w.append_at >= 0;
    const uint2 bits = make_uint2(w.append[0] | ((unsigned int)w.append[1] << 16), w.append[2] | ((unsigned int)w.append[3] << 16));
    encode_reset_kernel<<<1, 1, 0, st>>>(scratch, w.warm ? from : w.groups,
                                         reinterpret_cast<__half*>(const_cast<void*>(w.lines)) + (app ? (size_t)w.append_at * S : 0), bits,
                                         app ? S : 0);
    if (!w.warm && from < w.groups)
        encode_update_kernel<S><<<(w.groups - from + 31) / 32, 32, 0, st>>>(
            reinterpret_cast<const __half*>(w.data), w.groups, from, reinterpret_cast<const __half*>(w.lines), w.line0, w.line1,
            w.best_mse, w.best_at, w.cutoff, scratch);
    if (w.search) {
        EncSearch p;
        p.data = reinterpret_cast<const __half*>(w.data), p.stats = reinterpret_cast<const EncStats*>(w.stats);
        p.best_mse = w.best_mse, p.best_at = w.best_at, p.miss = scratch;
        p.best = reinterpret_cast<unsigned long long*>(scratch) + 1, p.done = reinterpret_cast<unsigned int*>(scratch) + 1;
        p.result = w.result, p.NG = w.groups, p.warm = w.warm, p.misses = w.misses;
        for (int e = 0; e < 2; ++e) {
            p.space[e].unit = reinterpret_cast<const __half*>(w.unit[e]), p.space[e].bias = reinterpret_cast<const __half*>(w.bias[e]);
            p.space[e].R = w.R[e], p.space[e].B = w.B[e], p.space[e].per_dim = w.per_dim[e];
            p.space[e].inv_s = 1.0f / (float)w.s_search_num, p.space[e].inv_ext = 1.0f / (float)w.extend_ratio;
        }
        encode_search_kernel<S><<<sm_count * 8, ENC_THREADS, 0, st>>>(p);
    } else {
        encode_report_kernel<<<1, 1, 0, st>>>(scratch, w.best_mse, w.best_at, w.groups, w.warm, w.result);
    }
    SBVR_CUDA_TRY(cudaGetLastError());
    SBVR_CUDA_TRY(cudaStreamSynchronize(st));
    return SBVR_OK;
}

// Selectors [N, Kp] -> bit-planes bvr[Kp/32, N, S]: bit i of word (kw, n, s) = bit (S-1-s) of sel[n, 32 kw + i]
// (`_change_coeff_sel_to_bvr` + layout change, sbvr/core.py:842-876, :783).  One warp per word position.
__global__ void encode_pack_kernel(const uint8_t* __restrict__ sel, int N, int KW, int S, uint32_t* __restrict__ bvr) {
    const int lane = threadIdx.x & 31;
    const size_t word = (size_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);     // kw * N + n
    if (word >= (size_t)KW * N) return;
    const int kw = (int)(word / N), n = (int)(word % N);
    const uint32_t v = sel[((size_t)n * KW + kw) * 32 + lane];
    uint32_t mine = 0;
    for (int s = 0; s < S; ++s) {
        const uint32_t w = __ballot_sync(0xffffffffu, (v >> (S - 1 - s)) & 1u);
        if (lane == s) mine = w;
    }
    if (lane < S) bvr[word * S + lane] = mine;
}

}  // namespace sbvr

using namespace sbvr;

extern "C" int sbvr_encode_mse_f16(const void* data, int groups, const void* lines, int L, int S, float* mse,
                                    sbvr_stream_t stream) {
    if (!data || !lines || !mse || groups < 1 || L < 1) return SBVR_ERR_BAD_ARG;
    if (groups > 65535) return SBVR_ERR_SHAPE;
    if (reinterpret_cast<uintptr_t>(data) & 3) return SBVR_ERR_ALIGN;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const dim3 grid((L + ENC_THREADS - 1) / ENC_THREADS, groups);
    const __half* d = reinterpret_cast<const __half*>(data);
    const __half* l = reinterpret_cast<const __half*>(lines);
    switch (S) {
        case 1: encode_mse_kernel<1><<<grid, ENC_THREADS, 0, st>>>(d, l, L, mse); break;
        case 2: encode_mse_kernel<2><<<grid, ENC_THREADS, 0, st>>>(d, l, L, mse); break;
        case 3: encode_mse_kernel<3><<<grid, ENC_THREADS, 0, st>>>(d, l, L, mse); break;
        case 4: encode_mse_kernel<4><<<grid, ENC_THREADS, 0, st>>>(d, l, L, mse); break;
        default: return SBVR_ERR_UNSUPPORTED;
    }
    SBVR_CUDA_TRY(cudaGetLastError());
    return SBVR_OK;
}

extern "C" int sbvr_encode_select_f16(const void* data, int groups, const void* lines, const int* which, int S,
                                       uint8_t* sel, sbvr_stream_t stream) {
    if (!data || !lines || !which || !sel || groups < 1) return SBVR_ERR_BAD_ARG;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const __half* d = reinterpret_cast<const __half*>(data);
    const __half* l = reinterpret_cast<const __half*>(lines);
    switch (S) {
        case 1: encode_select_kernel<1><<<groups, ENC_G, 0, st>>>(d, l, which, sel); break;
        case 2: encode_select_kernel<2><<<groups, ENC_G, 0, st>>>(d, l, which, sel); break;
        case 3: encode_select_kernel<3><<<groups, ENC_G, 0, st>>>(d, l, which, sel); break;
        case 4: encode_select_kernel<4><<<groups, ENC_G, 0, st>>>(d, l, which, sel); break;
        default: return SBVR_ERR_UNSUPPORTED;
    }
    SBVR_CUDA_TRY(cudaGetLastError());
    return SBVR_OK;
}

extern "C" int sbvr_encode_pack(const uint8_t* sel, int N, int Kp, int S, uint32_t* bvr, sbvr_stream_t stream) {
    if (!sel || !bvr || N < 1 || Kp < 32 || S < 1 || S > 8) return SBVR_ERR_BAD_ARG;
    if (Kp % 32) return SBVR_ERR_SHAPE;
    const int KW = Kp / 32;
    const size_t words = (size_t)KW * N;
    const size_t blocks = (words + 7) / 8;
    if (blocks > 0x7fffffffu) return SBVR_ERR_SHAPE;
    encode_pack_kernel<<<(unsigned int)blocks, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(sel, N, KW, S, bvr);
    SBVR_CUDA_TRY(cudaGetLastError());
    return SBVR_OK;
}

extern "C" int sbvr_encode_stats_f16(const void* data, int groups, float* stats, sbvr_stream_t stream) {
    if (!data || !stats || groups < 1) return SBVR_ERR_BAD_ARG;
    if ((reinterpret_cast<uintptr_t>(data) | reinterpret_cast<uintptr_t>(stats)) & 15) return SBVR_ERR_ALIGN;
    encode_stats_kernel<<<(groups + 7) / 8, 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
        reinterpret_cast<const __half*>(data), groups, reinterpret_cast<EncStats*>(stats));
    SBVR_CUDA_TRY(cudaGetLastError());
    return SBVR_OK;
}

extern "C" int sbvr_encode_advance(const sbvr_encode_walk_t* w, sbvr_stream_t stream) {
    if (!w || !w->data || !w->lines || !w->best_mse || !w->best_at || !w->scratch || !w->result) return SBVR_ERR_BAD_ARG;
    if (w->groups < 1 || w->from < 0 || w->from > w->groups || w->line0 < 0 || w->line1 < w->line0) return SBVR_ERR_BAD_ARG;
    if ((reinterpret_cast<uintptr_t>(w->data) & 15) || (reinterpret_cast<uintptr_t>(w->scratch) & 15)) return SBVR_ERR_ALIGN;
    if (w->search) {
        if (!w->stats || w->s_search_num < 1 || !(w->extend_ratio > 0.0)) return SBVR_ERR_BAD_ARG;
        for (int e = 0; e < 2; ++e) {
            if (!w->unit[e] || !w->bias[e] || w->R[e] < 1 || w->B[e] < 1 || w->per_dim[e] < 1) return SBVR_ERR_BAD_ARG;
            double n = (double)w->B[e] * 1024.0 * w->R[e], gd = 1.0;        // candidate numbers stay below 2^31
            for (int s = 0; s < w->S; ++s) gd *= (double)w->per_dim[e] + 1.0;
            if (n + gd >= 2.0e9 || w->per_dim[e] > 2000) return SBVR_ERR_UNSUPPORTED;
        }
    }
    int dev = 0;
    SBVR_CUDA_TRY(cudaGetDevice(&dev));
    DeviceInfo di;
    const int rc = device_info(dev, &di);
    if (rc) return rc;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    switch (w->S) {
        case 1: return encode_advance<1>(*w, di.sm_count, st);
        case 2: return encode_advance<2>(*w, di.sm_count, st);
        case 3: return encode_advance<3>(*w, di.sm_count, st);
        case 4: return encode_advance<4>(*w, di.sm_count, st);
        default: return SBVR_ERR_UNSUPPORTED;
    }
}
