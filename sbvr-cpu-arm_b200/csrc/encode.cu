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
// The walk over the groups (sbvr/core.py:555-653), a step per group that misses the codebook.
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

// Lines [line0, line1) against group g; true if its best is not below the cut-off.
template <int S>
__device__ __forceinline__ bool enc_update(const __half* data, int g, const __half* lines, int line0, int line1, float* best_mse,
                                           int* best_at, double cutoff) {
    float best = __ldcg(best_mse + g);
    int at = -1;
    const uint4* row = reinterpret_cast<const uint4*>(data + (size_t)g * ENC_G);
    for (int n = line0; n < line1; ++n) {
        __half2 pt[1 << S];
        __half line[S];
#pragma unroll
        for (int s = 0; s < S; ++s) line[s] = __ushort_as_half(__ldcg(reinterpret_cast<const unsigned short*>(lines) + (size_t)n * S + s));
        enc_points<S>(line, pt);
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
    if (at >= 0) {
        __stcg(best_mse + g, best);
        __stcg(best_at + g, at);
    }
    return !((double)best < cutoff);
}

// ... against the groups from `from` on; then the first of them that misses.
template <int S>
__global__ void __launch_bounds__(32) encode_update_kernel(const __half* __restrict__ data, int NG, int from,
                                                           const __half* __restrict__ lines, int line0, int line1,
                                                           float* __restrict__ best_mse, int* __restrict__ best_at, double cutoff,
                                                           int* __restrict__ miss) {
    const int g = from + blockIdx.x * 32 + threadIdx.x;
    const bool missing = g < NG && enc_update<S>(data, g, lines, line0, line1, best_mse, best_at, cutoff);
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

// What a group's statistics make of its search space.
template <int S>
struct EncGroup {
    int ns, total;                                 // scales; candidates
    float s_start, s_step, a0[S], a1[S];
    // false: not covered by the tables (a mean that widens the biases, values that are not finite, an empty range)
    __device__ __forceinline__ bool init(const EncStats& st, const EncSpace& sp, bool ext) {
        const float s_hi = enc_h(enc_h(st.d_max - st.d_min) * 1.1f), s_lo = 2.0f * st.d_95;
        s_step = __fmul_rn(s_hi - s_lo, sp.inv_s);             // products and sums rounded separately
        if (ext) s_step = __fmul_rn(s_step, sp.inv_ext);
        s_start = __fadd_rn(s_lo, s_step);
        const float s_end = __fadd_rn(s_hi, s_step);
        const double count = ceil(((double)s_end - (double)s_start) / (double)s_step);
        if (!(fabsf(st.d_avg) * 2.0f / S < 0.295f) || !(s_step > 0.0f) || !(count >= 1.0 && count <= 1024.0)) return false;
        ns = (int)count;
#pragma unroll
        for (int s = 0; s < S; ++s) {
            const float e0 = enc_linspace(st.d_min, st.d_max, S + 1, s), e1 = enc_linspace(st.d_min, st.d_max, S + 1, s + 1);
            const float slack = enc_h(fabsf(e0) * 0.8f);
            a0[s] = enc_h(e0 - slack), a1[s] = enc_h(e1 + slack);
        }
        total = 1;
#pragma unroll
        for (int s = 0; s < S; ++s) total *= sp.per_dim + 1;
        total += sp.B * ns * sp.R;
        return true;
    }
};

// This block's share of a group's candidates, the group's values in shared memory; the least key (mse bits << 32 | candidate) below
// that of `cached` goes to *best.
template <int S>
__device__ __forceinline__ void enc_search(const EncGroup<S>& q, const EncSpace& sp, const __half2* ds, float cached, unsigned long long* best) {
    const unsigned long long start_key = (unsigned long long)__float_as_uint(cached) << 32;
    float bound = cached;
    for (int c = blockIdx.x * ENC_THREADS + threadIdx.x; c - (int)threadIdx.x < q.total; c += gridDim.x * ENC_THREADS) {
        float line[S];
        enc_candidate<S>(sp, min(c, q.total - 1), q.ns, q.s_start, q.s_step, q.a0, q.a1, line);
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
        bool alive = c < q.total;
        for (int i = 0; i < ENC_G / 2; i += 8) {
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const float2 f = enc_err<S>(ds[i + e], pt);
                s0 += f.x, s1 += f.y;
            }
            if ((s0 + s1) * (1.0f / ENC_G) > bound) alive = false;
            if (!__any_sync(0xffffffffu, alive)) break;
            if (i % 32 == 24) bound = fminf(bound, __uint_as_float((unsigned int)(__ldcg(best) >> 32)));      // (a round trip to L2)
        }
        if (alive) {
            const unsigned long long key = ((unsigned long long)__float_as_uint((s0 + s1) * (1.0f / ENC_G)) << 32) | (unsigned int)c;
            if (key < start_key && key < __ldcg(best)) atomicMin(best, key);
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
    const float cached = p.warm ? INFINITY : p.best_mse[g];
    // extended search while the codebook serves well: hits / seen > 0.6
    const bool ext = p.warm || (double)(g - p.misses) / (double)(g + 1) > 0.6;
    const EncSpace& sp = p.space[ext ? 1 : 0];
    EncGroup<S> q;
    if (!q.init(p.stats[g], sp, ext)) {            // the caller's
        if (blockIdx.x == 0 && threadIdx.x == 0)
            p.result->group = g, p.result->status = 2, p.result->cached_mse = cached, p.result->cached_at = p.warm ? -1 : p.best_at[g];
        return;
    }
    for (int i = threadIdx.x; i < ENC_G / 2; i += ENC_THREADS) ds[i] = reinterpret_cast<const __half2*>(p.data + (size_t)g * ENC_G)[i];
    __syncthreads();
    enc_search<S>(q, sp, ds, cached, p.best);
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last_s = (atomicAdd(p.done, 1u) == gridDim.x - 1) ? 1u : 0u;
    __syncthreads();
    if (last_s && threadIdx.x == 0) {
        __threadfence();
        const unsigned long long key = __ldcg(p.best), start_key = (unsigned long long)__float_as_uint(cached) << 32;
        sbvr_encode_result_t* r = p.result;
        r->group = g;
        r->cached_mse = cached, r->cached_at = p.warm ? -1 : p.best_at[g];
        r->status = (key < start_key) ? 1 : 0;
        r->mse = __uint_as_float((unsigned int)(key >> 32));
        float line[S];
        enc_candidate<S>(sp, (key < start_key) ? (int)(key & 0xffffffffu) : 0, q.ns, q.s_start, q.s_step, q.a0, q.a1, line);
#pragma unroll
        for (int s = 0; s < S; ++s) r->line[s] = __half_as_ushort(__float2half_rn(line[s]));
    }
}

// ---------------------------------------------------------------------------------------------
// Many steps of the walk in one launch.  All blocks are resident (a cooperative launch) and go through a step together: new lines against
// the undecided groups, the first miss's candidates, and then block 0 alone decides -- it files the winner under a line within 0.01 %
// of it or a new one, and moves the cut-off -- while the others wait; three meetings of the grid.  1024 x 4096, S = 4: a step takes 54 us, 36
// of them the search (459 000 candidates, 16 half-rate differences and minima per pair of values, about half of them before the
// warp's last candidate is out), 13 the update, 4 the decision; with three launches, a synchronisation and the decision in Python
// per step it took 87.  Whole encoding: 11.3 -> 8.5 ms.
//
// The arithmetic of the decisions is the host's: a line's magnitude is the fp32 sum of its |c| in order, rounded to fp16; a difference
// of lines is rounded to fp32 and then to fp16; the mean of the accepted errors is a sum in double with Neumaier's
// compensation (what Python's `sum` does).  What the kernel cannot decide like the host (a group the tables do not cover, a winner with
// two coefficients of one magnitude, whose order is the tensor sort's) it leaves to the caller with the walk as it stands.
// ---------------------------------------------------------------------------------------------
constexpr int ENC_WINDOW = SBVR_ENCODE_WINDOW;                     // accepted errors the cut-off looks back on at most

struct EncCtl {                                    // device memory, all zero before the launch
    unsigned int arrived;
    int miss, from, n, line0, misses, steps, accepted, stop;
    int pad;
    double cutoff;
    unsigned long long best;
};
struct EncRun {
    EncSearch q;                                   // data, stats, best_mse, best_at, space, NG (the rest is the kernel's own)
    float* best_mse;
    int* best_at;
    __half* lines;
    EncCtl* ctl;
    sbvr_encode_record_t* records;
    int* outcome;
    int from, n, line0, misses, capacity, warmup, window, hist_n, limit;
    double acceptable;
    double hist[ENC_WINDOW];
};

// All blocks meet; false: they did not within about a second of SM clock.
__device__ __forceinline__ bool enc_meet(EncCtl* c, unsigned int& round) {
    __shared__ int ok_s;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(&c->arrived, 1u);
        const unsigned int want = ++round * gridDim.x;
        const long long t0 = clock64();
        unsigned int v;
        int ok = 1;
        for (;;) {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(&c->arrived) : "memory");
            if ((int)(v - want) >= 0) break;
            if (clock64() - t0 > 2000000000LL) {
                ok = 0;
                break;
            }
        }
        __threadfence();
        ok_s = ok;
    }
    __syncthreads();
    return ok_s != 0;
}

// Block 0: what becomes of group g.  Returns why the walk stops here (0: it does not).
template <int S>
__device__ __forceinline__ int enc_decide(const EncRun& p, const EncGroup<S>& q, const EncSpace& sp, int g, float cached, int& n, int& accepted,
                                          double* hist, int& hist_n) {
    __shared__ __half line_s[S];
    __shared__ float near_s;
    __shared__ int at_s, state_s;
    __shared__ float mse_s;
    if (threadIdx.x == 0) {
        const unsigned long long key = __ldcg(&p.ctl->best), start_key = (unsigned long long)__float_as_uint(cached) << 32;
        state_s = key < start_key ? 1 : 0;
        at_s = 0x7fffffff;
        if (state_s) {
            mse_s = __uint_as_float((unsigned int)(key >> 32));
            float line[S];
            enc_candidate<S>(sp, (int)(key & 0xffffffffu), q.ns, q.s_start, q.s_step, q.a0, q.a1, line);
#pragma unroll
            for (int i = 0; i < S; ++i)
#pragma unroll
                for (int j = 0; j + 1 < S - i; ++j)
                    if (fabsf(line[j]) > fabsf(line[j + 1])) {
                        const float t = line[j];
                        line[j] = line[j + 1], line[j + 1] = t;
                    }
            float mag = 0.0f;
#pragma unroll
            for (int s = 0; s < S; ++s) {
                if (s && !(fabsf(line[s]) > fabsf(line[s - 1]))) state_s = 2;
                line_s[s] = __float2half_rn(line[s]);          // (exact: candidates are fp16 values)
                mag = __fadd_rn(mag, fabsf(line[s]));
            }
            near_s = enc_h(__fmul_rn(enc_h(mag), 0.0001f));
        }
    }
    __syncthreads();
    const int state = state_s;
    if (state != 1) return state ? 2 : 0;          // 0: the codebook already has something at least as good
    for (int i = threadIdx.x; i < n; i += ENC_THREADS) {
        float mag = 0.0f;
#pragma unroll
        for (int s = 0; s < S; ++s) {
            const float a = __half2float(__ushort_as_half(__ldcg(reinterpret_cast<const unsigned short*>(p.lines) + (size_t)i * S + s)));
            mag = __fadd_rn(mag, fabsf(enc_h(__fsub_rn(a, __half2float(line_s[s])))));
        }
        if (enc_h(mag) < near_s) atomicMin(&at_s, i);
    }
    __syncthreads();
    int at = at_s;
    const bool append = at == 0x7fffffff;
    if (append && n >= p.capacity) return 2;
    if (append) at = n;
    if (threadIdx.x == 0) {
        sbvr_encode_record_t r;
        r.group = g, r.at = at, r.mse = mse_s;
#pragma unroll
        for (int s = 0; s < 4; ++s) r.line[s] = s < S ? __half_as_ushort(line_s[s < S ? s : 0]) : (unsigned short)0;
        p.records[accepted] = r;
        if (append)
#pragma unroll
            for (int s = 0; s < S; ++s) __stcg(reinterpret_cast<unsigned short*>(p.lines) + (size_t)n * S + s, __half_as_ushort(line_s[s]));
        // the last `window` accepted errors, the newest behind
        if (hist_n == p.window) {
            for (int i = 1; i < hist_n; ++i) hist[i - 1] = hist[i];
            hist[hist_n - 1] = (double)mse_s;
        } else {
            hist[hist_n] = (double)mse_s;
        }
    }
    if (hist_n < p.window) ++hist_n;
    if (append) ++n;
    ++accepted;
    __syncthreads();
    return 0;
}

__device__ __forceinline__ double enc_cutoff(const double* hist, int n, double acceptable) {
    double sum = 0.0, c = 0.0;
    for (int i = 0; i < n; ++i) {
        const double x = hist[i], t = __dadd_rn(sum, x);
        if (fabs(sum) >= fabs(x)) c = __dadd_rn(c, __dadd_rn(__dadd_rn(sum, -t), x));
        else c = __dadd_rn(c, __dadd_rn(__dadd_rn(x, -t), sum));
        sum = t;
    }
    if (c != 0.0 && isfinite(c)) sum = __dadd_rn(sum, c);
    const double m = __dmul_rn(__ddiv_rn(sum, (double)n), 0.99);
    return acceptable > m ? acceptable : m;        // Python's max(m, acceptable): the first unless the second is greater
}

// Lines [line0, line1) against the undecided groups from `from` on, sixteen groups of a block at a time: a warp makes a group's 256 errors
// (one 512-byte row per load), then a thread per group adds them in the order of `enc_update`.  With a thread per group throughout
// -- a row each, a round trip to L2 per sixteen values -- this took 28 us a step for 16 384 groups.
constexpr int ENC_UG = 16;
template <int S>
__device__ __forceinline__ void enc_update_all(const EncRun& p, int from, int line0, int line1, double cutoff) {
    __shared__ __align__(16) float2 err[ENC_UG][ENC_G / 2 + 1];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int g0 = from + blockIdx.x * ENC_UG; g0 < p.q.NG; g0 += gridDim.x * ENC_UG) {
        const int g = g0 + (int)threadIdx.x;
        const bool mine = threadIdx.x < ENC_UG && g < p.q.NG;
        float best = mine ? __ldcg(p.best_mse + g) : 0.0f;
        int at = -1;
        for (int n = line0; n < line1; ++n) {
            __half line[S];
            __half2 pt[1 << S];
#pragma unroll
            for (int s = 0; s < S; ++s) line[s] = __ushort_as_half(__ldcg(reinterpret_cast<const unsigned short*>(p.lines) + (size_t)n * S + s));
            enc_points<S>(line, pt);
#pragma unroll
            for (int k = 0; k < ENC_UG / (ENC_THREADS / 32); ++k) {
                const int j = warp * (ENC_UG / (ENC_THREADS / 32)) + k;
                if (g0 + j < p.q.NG) {
                    const uint4 v = __ldg(reinterpret_cast<const uint4*>(p.q.data + (size_t)(g0 + j) * ENC_G) + lane);
                    const __half2* d = reinterpret_cast<const __half2*>(&v);
#pragma unroll
                    for (int e = 0; e < 4; ++e) err[j][lane * 4 + e] = enc_err<S>(d[e], pt);
                }
            }
            __syncthreads();
            if (mine) {
                float s0 = 0.0f, s1 = 0.0f;
#pragma unroll 16
                for (int i = 0; i < ENC_G / 2; ++i) {
                    const float2 f = err[threadIdx.x][i];
                    s0 += f.x, s1 += f.y;
                }
                const float mse = (s0 + s1) * (1.0f / ENC_G);
                if (mse < best) best = mse, at = n;
            }
            __syncthreads();
        }
        if (at >= 0) {
            __stcg(p.best_mse + g, best);
            __stcg(p.best_at + g, at);
        }
        if (warp == 0) {
            const unsigned int m = __ballot_sync(0xffffffffu, mine && !((double)best < cutoff));
            if (m && lane == 0) atomicMin(&p.ctl->miss, g0 + __ffs((int)m) - 1);
        }
    }
}

template <int S>
__global__ void __launch_bounds__(ENC_THREADS) encode_walk_kernel(const __grid_constant__ EncRun p) {
    __shared__ __align__(16) __half2 ds[ENC_G / 2];
    __shared__ double hist[ENC_WINDOW];
    EncCtl* c = p.ctl;
    unsigned int round = 0;
    int n = p.n, misses = p.misses, accepted = 0, steps = 0, hist_n = p.hist_n, from = p.from, line0 = p.line0;      // block 0's are the truth
    auto publish = [&](int stop) {                 // block 0, one thread
        const bool warm = n < p.warmup;
        if (!stop && from >= p.q.NG) stop = SBVR_ENCODE_DONE;
        if (!stop && !warm && n >= p.capacity) stop = SBVR_ENCODE_FULL;
        if (!stop && !warm && hist_n == 0) stop = SBVR_ENCODE_CALLER;
        if (!stop && steps >= p.limit) stop = SBVR_ENCODE_LIMIT;
        c->from = from, c->n = n, c->line0 = line0, c->misses = misses, c->accepted = accepted;
        c->cutoff = warm ? 0.0 : (hist_n ? enc_cutoff(hist, hist_n, p.acceptable) : 0.0);
        c->miss = warm ? from : p.q.NG;
        c->best = ~0ull;
        c->stop = stop;
    };
    if (blockIdx.x == 0) {
        for (int i = threadIdx.x; i < hist_n; i += ENC_THREADS) hist[i] = p.hist[i];
        __syncthreads();
        if (threadIdx.x == 0) publish(0);
    }
    bool met = enc_meet(c, round);
    while (met) {
        if (__ldcg(&c->stop)) break;
        from = __ldcg(&c->from), n = __ldcg(&c->n), line0 = __ldcg(&c->line0), misses = __ldcg(&c->misses);
        const double cutoff = __ldcg(&c->cutoff);
        const bool warm = n < p.warmup;
        const int met_from = line0;                // (should the blocks not meet: lines that not every group has met)
        if (!warm) {
            enc_update_all<S>(p, from, line0, n, cutoff);
            line0 = n;
        }
        if (!(met = enc_meet(c, round))) {
            line0 = met_from;
            break;
        }
        const int g = __ldcg(&c->miss);
        float cached = INFINITY;
        bool covered = true;
        EncGroup<S> q;
        bool ext = warm;
        if (g < p.q.NG) {
            if (!warm) cached = __ldcg(p.best_mse + g);
            ext = warm || (double)(g - misses) / (double)(g + 1) > 0.6;
            covered = q.init(p.q.stats[g], p.q.space[ext ? 1 : 0], ext);
            if (covered) {
                for (int i = threadIdx.x; i < ENC_G / 2; i += ENC_THREADS) ds[i] = reinterpret_cast<const __half2*>(p.q.data + (size_t)g * ENC_G)[i];
                __syncthreads();
                enc_search<S>(q, p.q.space[ext ? 1 : 0], ds, cached, &c->best);
            }
        }
        if (!(met = enc_meet(c, round))) {
            line0 = met_from;
            break;
        }
        if (blockIdx.x == 0) {
            int stop = 0;
            if (g >= p.q.NG) stop = SBVR_ENCODE_DONE;
            else if (!covered) stop = SBVR_ENCODE_CALLER;
            else if (enc_decide<S>(p, q, p.q.space[ext ? 1 : 0], g, cached, n, accepted, hist, hist_n)) stop = SBVR_ENCODE_CALLER;
            else ++misses, ++steps, from = g + 1;
            if (stop == SBVR_ENCODE_CALLER) from = g;          // (every group in front of it is served)
            if (threadIdx.x == 0) publish(stop);
        }
        met = enc_meet(c, round);
    }
    // Blocks that have not met -- another stream's kernel keeps some from running -- leave the walk at the last decision: block 0 decides only
    // when all have searched, and a line that a group meets a second time changes nothing.
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        p.outcome[0] = met ? __ldcg(&c->stop) : SBVR_ENCODE_TIMEOUT;
        p.outcome[1] = from, p.outcome[2] = n, p.outcome[3] = line0, p.outcome[4] = misses, p.outcome[5] = accepted;
    }
}

template <int S>
static int encode_run(const EncRun& r, int sm_count, cudaStream_t st) {
    int per_sm = 0;
    SBVR_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, encode_walk_kernel<S>, ENC_THREADS, 0));
    if (per_sm < 1) return SBVR_ERR_UNSUPPORTED;
    if (per_sm > 8) per_sm = 8;
    EncRun copy = r;
    void* args[] = {&copy};
    SBVR_CUDA_TRY(cudaMemsetAsync(r.ctl, 0, sizeof(EncCtl), st));
    SBVR_CUDA_TRY(cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(encode_walk_kernel<S>), dim3(per_sm * sm_count), dim3(ENC_THREADS),
                                              args, 0, st));
    SBVR_CUDA_TRY(cudaStreamSynchronize(st));
    return SBVR_OK;
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

static EncSearch enc_search_params(const sbvr_encode_walk_t& w) {
    EncSearch p = {};
    p.data = reinterpret_cast<const __half*>(w.data), p.stats = reinterpret_cast<const EncStats*>(w.stats);
    p.best_mse = w.best_mse, p.best_at = w.best_at;
    p.result = w.result, p.NG = w.groups, p.warm = w.warm, p.misses = w.misses;
    for (int e = 0; e < 2; ++e) {
        p.space[e].unit = reinterpret_cast<const __half*>(w.unit[e]), p.space[e].bias = reinterpret_cast<const __half*>(w.bias[e]);
        p.space[e].R = w.R[e], p.space[e].B = w.B[e], p.space[e].per_dim = w.per_dim[e];
        p.space[e].inv_s = 1.0f / (float)w.s_search_num, p.space[e].inv_ext = 1.0f / (float)w.extend_ratio;
    }
    return p;
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
        EncSearch p = enc_search_params(w);
        p.miss = scratch;
        p.best = reinterpret_cast<unsigned long long*>(scratch) + 1, p.done = reinterpret_cast<unsigned int*>(scratch) + 1;
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

static int enc_check(const sbvr_encode_walk_t* w) {
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
    return SBVR_OK;
}

extern "C" int sbvr_encode_run(const sbvr_encode_walk_t* w, const sbvr_encode_run_t* run, sbvr_stream_t stream) {
    int rc = enc_check(w);
    if (rc) return rc;
    if (!w->search || !run || !run->ctl || !run->records || !run->outcome || run->n < 0 || run->capacity < 1 || run->limit < 1 ||
        run->window < 1 || run->hist_n < 0 || run->hist_n > run->window || w->append_at >= 0 || w->line0 > run->n)
        return SBVR_ERR_BAD_ARG;
    if (run->window > SBVR_ENCODE_WINDOW || run->limit > (1 << 20)) return SBVR_ERR_UNSUPPORTED;
    if (reinterpret_cast<uintptr_t>(run->ctl) & 15) return SBVR_ERR_ALIGN;
    int dev = 0;
    SBVR_CUDA_TRY(cudaGetDevice(&dev));
    DeviceInfo di;
    rc = device_info(dev, &di);
    if (rc) return rc;
    EncRun r = {};
    r.q = enc_search_params(*w);
    r.best_mse = w->best_mse, r.best_at = w->best_at, r.lines = reinterpret_cast<__half*>(const_cast<void*>(w->lines));
    r.ctl = reinterpret_cast<EncCtl*>(run->ctl), r.records = run->records, r.outcome = run->outcome;
    r.from = w->from, r.n = run->n, r.line0 = w->line0, r.misses = w->misses, r.capacity = run->capacity, r.warmup = run->warmup;
    r.window = run->window, r.hist_n = run->hist_n, r.limit = run->limit, r.acceptable = run->acceptable;
    for (int i = 0; i < run->hist_n; ++i) r.hist[i] = run->hist[i];
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    switch (w->S) {
        case 1: return encode_run<1>(r, di.sm_count, st);
        case 2: return encode_run<2>(r, di.sm_count, st);
        case 3: return encode_run<3>(r, di.sm_count, st);
        case 4: return encode_run<4>(r, di.sm_count, st);
        default: return SBVR_ERR_UNSUPPORTED;
    }
}

extern "C" int sbvr_encode_advance(const sbvr_encode_walk_t* w, sbvr_stream_t stream) {
    const int bad = enc_check(w);
    if (bad) return bad;
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
