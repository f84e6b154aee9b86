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
template <int S, int THREADS>
__device__ __forceinline__ void enc_search(const EncGroup<S>& q, const EncSpace& sp, const __half2* ds, float cached, unsigned long long* best) {
    const unsigned long long start_key = (unsigned long long)__float_as_uint(cached) << 32;
    float bound = cached;
    for (int c = blockIdx.x * THREADS + threadIdx.x; c - (int)threadIdx.x < q.total; c += gridDim.x * THREADS) {
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
    enc_search<S, ENC_THREADS>(q, sp, ds, cached, p.best);
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
// Many steps of the walk in one launch.  All blocks are resident (a cooperative launch) and go through a step together, two meetings of the
// grid each: new lines against the undecided groups; the first miss's candidates.  What becomes of the winner -- it is filed under a line
// within 0.01 % of it or a new one, and moves the cut-off -- every block decides for itself from the same words; block 0 alone writes it
// down.  1024 x 4096, S = 4, 16 384 groups, 201 misses of 459 000 candidates each: 11.1 -> 6.2 ms, 50 -> 24 us a step, of them 10 the bounds
// of the candidates, 5 the two meetings, 4 a group's tables, 2 the first look at it, 1.5 the decision, 1 the new line against the window.
//
// The arithmetic of the decisions is the host's: a line's magnitude is the fp32 sum of its |c| in order, rounded to fp16; a difference
// of lines is rounded to fp32 and then to fp16; the mean of the accepted errors is a sum in double with Neumaier's
// compensation (what Python's `sum` does).  What the kernel cannot decide like the host (a group the tables do not cover, a winner with
// two coefficients of one magnitude, whose order is the tensor sort's) it leaves to the caller with the walk as it stands.
// ---------------------------------------------------------------------------------------------
constexpr int ENC_WINDOW = SBVR_ENCODE_WINDOW;                     // accepted errors the cut-off looks back on at most

struct EncCtl {                                    // device memory, all zero before the launch
    unsigned int arrived;
    unsigned int go;                               // steps that block 0 has seen everyone search: their decisions may be acted on
    int miss[3];                                   // of step t in slot t % 3: first group that misses
    float ub[3];                                   // an upper bound of the best candidate's mse
    unsigned long long best[3];                    // (mse bits << 32 | candidate)
};
static_assert(sizeof(EncCtl) <= 64, "sbvr_encode_run_t::ctl");
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

// Waits until *word, an always growing counter, has reached `want`; false: it has not within about a second of SM clock.
__device__ __forceinline__ bool enc_reached(const unsigned int* word, unsigned int want) {
    const long long t0 = clock64();
    for (;;) {
        unsigned int v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(word) : "memory");
        if ((int)(v - want) >= 0) return true;
        if (clock64() - t0 > 2000000000LL) return false;
    }
}

// All blocks meet; false: they did not.
__device__ __forceinline__ bool enc_meet(EncCtl* c, unsigned int& round) {
    __shared__ int ok_s;
    __syncthreads();
    if (threadIdx.x == 0) {
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&c->arrived) : "memory");
        ok_s = enc_reached(&c->arrived, ++round * gridDim.x) ? 1 : 0;
    }
    __syncthreads();
    return ok_s != 0;
}

// ---- the search of one group by all blocks -----------------------------------------------------------------------------
// Evaluated value by value a candidate is 2^S fp16 differences and minima per pair of 256 values, and half of its values were
// needed on average before it was out: 36 us of a step's 50 (459 000 candidates, S = 4; with bounds 10).  Its squared error is much cheaper
// to BOUND.
// With the candidate's sums sorted, q_0 <= .. <= q_J, every value v belongs to the sum on its side of the midpoints b_j, and
//   sum (v - nearest)^2 = sum (v - q_J)^2 - 2 sum_j (q_j+1 - q_j) F(b_j),   F(b) = sum over v of max(b - v, 0),
// since moving the values below b_j from q_j+1 to q_j gains (v - q_j+1)^2 - (v - q_j)^2 = 2 (q_j+1 - q_j) (b_j - v).  F is convex
// and piecewise linear: chords over ENC_NB equal intervals lie above it, by count * width / 4 of an interval at most.  So a table of
// chords gives a lower bound of the error in 2^S - 1 look-ups, and an upper bound with the largest gap of a chord: about 0.8 % below
// and 6 % above on 256 normal values.  Candidates whose lower bound is above the least upper bound (of the whole grid, as far as known)
// or above the group's best stored line cannot win; what is left, a handful per block, is evaluated as ever, a warp per candidate.
//
// The bounds hold for the evaluated error, not only for the real one.  An evaluated value is fp16(fp16(|v - q|)^2): off by three relative
// roundings of 2^-11, or by 2^-25 where the square is subnormal; their fp32 sum by 128 roundings of 2^-24.  ENC_REL and ENC_ABS
// cover them.  The bound's own arithmetic is fp32 on values centred in their range [-R, R], with Rq = max(R, |q|): F is off by at most
// 4.5e-4 Rq (the prefix sums of 256 values, slope and offset of a chord, the interval's index by 6e-5 of a width), so that twice
// the sum of gap * F is off by 1.8e-3 Rq^2, its additions by 1.8e-3, the sums in front of it by 6e-4: 4.2e-3 Rq^2 in all, below ENC_EPS.
constexpr int ENC_WT = 640;                        // threads of the walk's blocks, one per SM (512 and 768: 7.6 ms where 640 take 7.1)
constexpr int ENC_WARPS = ENC_WT / 32;
constexpr int ENC_NB = 512;
constexpr int ENC_SMALL = 64;
constexpr int ENC_ROUNDS = 5;                      // candidates of a thread between two evaluations
constexpr int ENC_LIST = ENC_ROUNDS * ENC_WT;
constexpr int ENC_SCALES = 1024, ENC_AXIS = 2001, ENC_RATIOS = 256, ENC_BIASES = 256;      // most that the tables in shared memory hold
constexpr float ENC_REL = 1.6e-3f, ENC_ABS = 256.0f / 33554432.0f, ENC_EPS = 1.0f / 128.0f;

template <int S>
struct EncFast {                                   // shared memory of a block
    float2 chord[ENC_NB + 2];                      // half the slope, offset; [0] below the values, [ENC_NB + 1] above
    union {
        struct {
            int count[ENC_NB];
            float sum[ENC_NB];
        } b;
        float2 err[ENC_WARPS][ENC_G / 2];
        float2 own[ENC_WARPS][ENC_G / 2];          // chords of a warp's own group: ENC_OWN + 2 of them
    };
    float red[ENC_WARPS][4];
    float small[ENC_SMALL + 1];                    // sum of v^2 over the values below k / ENC_SMALL of the largest magnitude
    uint2 list[ENC_LIST];                          // candidate, lower bound
    int alive[ENC_LIST];
    int n_list, n_alive;
    float unit[2][ENC_RATIOS][S], bias[2][ENC_BIASES];         // plain and extended lists
    float scale[ENC_SCALES], axis[S][ENC_AXIS];    // a group's scales and axes
};

// Sums of all subsets of line[0 .. S) (magnitudes ascending), ascending, as fp16 values centred at `mid`.  A list L of sums without
// coefficient c becomes L + min(c, 0) followed by L + max(c, 0); as |c| is at least every magnitude before it, only the ends of the two
// halves can overlap: one comparison at the third coefficient, a merge of four and four at the fourth.  (Sums are rounded: two that
// are equal but for that may come out an fp16 step in the wrong order, which is far below what the bounds allow for.)
__device__ __forceinline__ void enc_cmp(float& a, float& b) {
    const float lo = fminf(a, b), hi = fmaxf(a, b);
    a = lo, b = hi;
}
template <int S>
__device__ __forceinline__ void enc_sorted_sums(const float (&line)[S], float mid, float (&v)[1 << S]) {
    v[0] = 0.0f;
#pragma unroll
    for (int s = 0; s < S; ++s) {
        const float lo = fminf(line[s], 0.0f), hi = fmaxf(line[s], 0.0f);
#pragma unroll
        for (int j = (1 << s) - 1; j >= 0; --j) v[j + (1 << s)] = v[j] + hi, v[j] += lo;
        if (s == 2) enc_cmp(v[3], v[4]);
        if (s == 3) {                              // Batcher's merge of v[4 .. 7] and v[8 .. 11]
            enc_cmp(v[4], v[8]), enc_cmp(v[5], v[9]), enc_cmp(v[6], v[10]), enc_cmp(v[7], v[11]);
            enc_cmp(v[6], v[8]), enc_cmp(v[7], v[9]);
            enc_cmp(v[5], v[6]), enc_cmp(v[7], v[8]), enc_cmp(v[9], v[10]);
        }
    }
#pragma unroll
    for (int j = 0; j < (1 << S); j += 2) {
        const float2 f = __half22float2(__floats2half2_rn(v[j], v[j + 1]));
        v[j] = f.x - mid, v[j + 1] = f.y - mid;
    }
}
template <int S>
__device__ __forceinline__ void enc_sort_line(float (&line)[S]) {
#pragma unroll
    for (int i = 0; i < S; ++i)
#pragma unroll
        for (int j = 0; j + 1 < S - i; ++j)
            if (fabsf(line[j]) > fabsf(line[j + 1])) {
                const float t = line[j];
                line[j] = line[j + 1], line[j + 1] = t;
            }
}
template <int S>
__device__ __forceinline__ void enc_line_points(const float (&line)[S], __half2 (&pt)[1 << S]) {
    __half h[S];
#pragma unroll
    for (int s = 0; s < S; ++s) h[s] = __float2half_rn(line[s]);       // (exact: candidates are fp16 values)
    enc_points<S>(h, pt);
}
__device__ __forceinline__ float enc_warp_sum(float v) {
#pragma unroll
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
// The errors of a warp's 256 values (pairs lane, lane + 32, ..), added in the order of an evaluation: even and odd values apart, first to last.
__device__ __forceinline__ float enc_ordered_mse(const float2 (&f)[4], float2* err, int lane) {
#pragma unroll
    for (int e = 0; e < 4; ++e) err[lane + 32 * e] = f[e];
    __syncwarp();
    float s = 0.0f;
    if (lane < 2) {
        const float* x = reinterpret_cast<const float*>(err) + lane;
#pragma unroll 16
        for (int i = 0; i < ENC_G / 2; ++i) s += x[2 * i];
    }
    __syncwarp();
    return (__shfl_sync(0xffffffffu, s, 0) + __shfl_sync(0xffffffffu, s, 1)) * (1.0f / ENC_G);
}

// What enc_candidate makes of a number, from tables in shared memory: scales, axes (a division and five roundings a value) and the lists
// that all groups share.  Quotients by the lists' lengths are products with the rounded-up reciprocal, exact for numbers below
// 2^32 / length.
struct EncLines {
    int nline, ns;
    unsigned int by_r, by_ns, by_axis, R, axis;
    const float *unit, *bias;
};
__device__ __forceinline__ unsigned int enc_reciprocal(int d) { return d == 1 ? 0u : 0xffffffffu / (unsigned int)d + 1u; }
__device__ __forceinline__ unsigned int enc_quotient(unsigned int n, unsigned int reciprocal) { return reciprocal ? __umulhi(n, reciprocal) : n; }
template <int S>
__device__ __forceinline__ bool enc_lines_fit(const EncGroup<S>& q, const EncSpace& sp) {
    return q.total <= (1 << 21) && q.ns <= ENC_SCALES && sp.R <= ENC_RATIOS && sp.B <= ENC_BIASES && sp.per_dim + 1 <= ENC_AXIS;
}
template <int S>
__device__ __forceinline__ void enc_lists_init(EncFast<S>& sm, const EncSpace (&space)[2]) {
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        for (int i = threadIdx.x; i < min(space[e].R, ENC_RATIOS) * S; i += ENC_WT) sm.unit[e][i / S][i % S] = __half2float(space[e].unit[i]);
        for (int i = threadIdx.x; i < min(space[e].B, ENC_BIASES); i += ENC_WT) sm.bias[e][i] = __half2float(space[e].bias[i]);
    }
}
template <int S>
__device__ __forceinline__ EncLines enc_lines_init(EncFast<S>& sm, const EncGroup<S>& q, const EncSpace& sp, bool ext) {
    const int n = sp.per_dim + 1;
    for (int i = ENC_WT - 1 - (int)threadIdx.x; i < n * S; i += ENC_WT) {      // (the last threads: the first have the chords to make)
#pragma unroll
        for (int s = 0; s < S; ++s)
            if (i / n == s) sm.axis[s][i % n] = enc_linspace(q.a0[s], q.a1[s], n, i % n);
    }
    for (int i = (ENC_WT + ENC_G - 1 - (int)threadIdx.x) % ENC_WT; i < q.ns; i += ENC_WT) sm.scale[i] = enc_h(fmaf(q.s_step, (float)i, q.s_start));
    EncLines l;
    l.R = (unsigned int)sp.R, l.ns = q.ns, l.axis = (unsigned int)n, l.nline = sp.B * q.ns * sp.R;
    l.by_r = enc_reciprocal(sp.R), l.by_ns = enc_reciprocal(q.ns), l.by_axis = enc_reciprocal(n);
    l.unit = sm.unit[ext ? 1 : 0][0], l.bias = sm.bias[ext ? 1 : 0];
    return l;
}
template <int S>
__device__ __forceinline__ void enc_line(const EncFast<S>& sm, const EncLines& l, int c, float (&line)[S]) {
    if (c < l.nline) {
        const unsigned int bs = enc_quotient((unsigned int)c, l.by_r), r = (unsigned int)c - bs * l.R;
        const unsigned int b = enc_quotient(bs, l.by_ns), si = bs - b * (unsigned int)l.ns;
        const float sv = sm.scale[si], bv = l.bias[b];
#pragma unroll
        for (int s = 0; s < S; ++s) line[s] = enc_h(bv + enc_h(sv * l.unit[r * S + s]));
    } else {
        unsigned int n = (unsigned int)(c - l.nline);
#pragma unroll
        for (int s = S - 1; s >= 0; --s) {
            const unsigned int m = enc_quotient(n, l.by_axis);
            line[s] = sm.axis[s][n - m * l.axis];
            n = m;
        }
    }
}

// Whether the bounds' roundings are as above: a range that is neither empty nor where fp16 squares overflow.
__device__ __forceinline__ bool enc_boundable(const EncStats& st) {
    return st.d_max - st.d_min > 1e-6f && fmaxf(fabsf(st.d_max), fabsf(st.d_min)) <= 16.0f;
}

// One lower and one upper bound of a line's squared error (sums over the 256 values, the evaluated ones) by a table of NB chords.
struct EncTable {
    float mid, R, inv, total, squares, gap;        // range, sums over the centred values, twice the largest gap between a chord and F
};
// Interval of b = b2 / 2: 1 + floor((b + R) / width), 0 below, NB + 1 above.  x is the place in [0, 1] of the table, by a multiply-add that
// saturates; the nearest whole number to x (NB + 1) is in the lower bits of that plus 2^23.
template <int NB>
__device__ __forceinline__ int enc_interval(float b2, float inv) {
    const float x = __saturatef(fmaf(b2, 0.5f / (NB + 1) * inv, 0.5f));        // (b + R) inv = b inv + NB / 2
    return __float_as_int(fmaf(x, (float)(NB + 1), 8388608.0f)) - 0x4B000000;
}
template <int S, int NB>
__device__ __forceinline__ float2 enc_bounds(const EncTable& t, const float2* chord, const float (&line)[S]) {
    constexpr int J = (1 << S) - 1;
    float v[1 << S];
    enc_sorted_sums<S>(line, t.mid, v);
    float acc = 0.0f;
#pragma unroll
    for (int j = 0; j < J; ++j) {
        const float b2 = v[j] + v[j + 1];
        const float2 ch = chord[enc_interval<NB>(b2, t.inv)];
        acc = fmaf(v[j + 1] - v[j], fmaf(ch.x, b2, ch.y), acc);
    }
    const float raw = fmaf(-2.0f, acc, fmaf(v[J], fmaf((float)ENC_G, v[J], -2.0f * t.total), t.squares));
    const float rq = fmaxf(t.R, fmaxf(fabsf(v[0]), fabsf(v[J]))), eps = ENC_EPS * rq * rq;
    const float high = fmaf(raw + eps + t.gap * (v[J] - v[0]), 1.0f + ENC_REL, ENC_ABS);
    return make_float2(fmaf(raw, 1.0f - ENC_REL, -eps - ENC_ABS), high < INFINITY && rq < 64.0f ? high : INFINITY);
}

// This block's share of a group's candidates; `best` and `ub` are the grid's words.
template <int S>
__device__ __forceinline__ void enc_search_bounded(EncFast<S>& sm, const EncGroup<S>& q, const EncSpace& sp, const EncStats& st, const __half2* ds,
                                                   float cached, bool ext, unsigned long long* best, float* ub, EncLines& lines) {
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    EncTable t;
    t.mid = 0.5f * (st.d_max + st.d_min), t.R = 0.5f * (st.d_max - st.d_min);
    const float width = 2.0f * t.R / ENC_NB;
    t.inv = (float)ENC_NB / (2.0f * t.R);
    // ---- the tables
    for (int i = tid; i < ENC_NB; i += ENC_WT) sm.b.count[i] = 0, sm.b.sum[i] = 0.0f;
    if (tid <= ENC_SMALL) sm.small[tid] = 0.0f;
    if (tid == 0) sm.n_list = 0, sm.n_alive = 0;
    const float vabs = fmaxf(fabsf(st.d_max), fabsf(st.d_min)), per_v = (float)ENC_SMALL / vabs;
    lines = enc_lines_init<S>(sm, q, sp, ext);
    __syncthreads();
    float sq = 0.0f;
    if (tid < ENC_G) {
        const float d = __half2float(reinterpret_cast<const __half*>(ds)[tid]), v = d - t.mid;
        atomicAdd(&sm.small[min((int)(fabsf(d) * per_v) + 1, ENC_SMALL)], d * d);
        const int k = min(max(enc_interval<ENC_NB>(2.0f * v, t.inv) - 1, 0), ENC_NB - 1);
        atomicAdd(&sm.b.count[k], 1);
        atomicAdd(&sm.b.sum[k], v);
        sq = v * v;
    }
    __syncthreads();
    const bool on = tid < ENC_NB;
    const float cn = on ? (float)sm.b.count[tid] : 0.0f, cs = on ? sm.b.sum[tid] : 0.0f;
    float n_in = cn, s_in = cs, top = cn;          // inclusive over the warp's lanes
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const float a = __shfl_up_sync(0xffffffffu, n_in, o), b = __shfl_up_sync(0xffffffffu, s_in, o);
        if (lane >= o) n_in += a, s_in += b;
        top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
    }
    sq = enc_warp_sum(sq);
    if (warp == ENC_WARPS - 1) {                   // running sums of small[1 .. ENC_SMALL]
        float a = sm.small[1 + 2 * lane], b = a + sm.small[2 + 2 * lane], in = b;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float f = __shfl_up_sync(0xffffffffu, in, o);
            if (lane >= o) in += f;
        }
        sm.small[1 + 2 * lane] = in - b + a, sm.small[2 + 2 * lane] = in;
    }
    if (lane == 31) sm.red[warp][0] = n_in, sm.red[warp][1] = s_in, sm.red[warp][2] = top, sm.red[warp][3] = sq;
    __syncthreads();
    float rank = n_in - cn, below = s_in - cs, largest = 0.0f;
    t.total = 0.0f, t.squares = 0.0f;
#pragma unroll
    for (int i = 0; i < ENC_NB / 32; ++i) {
        if (i < warp) rank += sm.red[i][0], below += sm.red[i][1];
        t.total += sm.red[i][1], largest = fmaxf(largest, sm.red[i][2]);
        if (i < ENC_G / 32) t.squares += sm.red[i][3];
    }
    if (on) {
        const float x0 = fmaf(width, (float)tid, -t.R), x1 = fmaf(width, (float)(tid + 1), -t.R);
        const float f0 = fmaf(rank, x0, -below), f1 = fmaf(rank + cn, x1, -(below + cs)), slope = (f1 - f0) * t.inv;
        sm.chord[1 + tid] = make_float2(0.5f * slope, fmaf(-slope, x0, f0));
    }
    if (tid == 0) sm.chord[0] = make_float2(0.0f, 0.0f), sm.chord[ENC_NB + 1] = make_float2(0.5f * ENC_G, -t.total);
    __syncthreads();
    t.gap = 0.51f * largest * width;               // (a little more than twice count * width / 4)

    // ---- bounds of every candidate, survivors into the list; then the survivors
    const unsigned long long start_key = (unsigned long long)__float_as_uint(cached) << 32;
    float bound = cached;                          // mse that a candidate must not exceed
    const int stride = gridDim.x * ENC_WT;
    for (int base = (int)blockIdx.x * 32 + warp * 32 * (int)gridDim.x; __syncthreads_or(base < q.total); base += ENC_ROUNDS * stride) {
        float told = __ldcg(ub);
        bound = fminf(bound, told);
#pragma unroll 1
        for (int i = 0; i < ENC_ROUNDS; ++i) {
            const int c = base + i * stride + lane;
            if (c - lane >= q.total) break;
            float line[S];
            enc_line<S>(sm, lines, min(c, q.total - 1), line);
            // Coefficients of one sign: no sum but 0 is nearer to 0 than the smallest, to which values of at most half of it stay.
            {
                float lo = fabsf(line[0]);
                bool plus = true, minus = true;
#pragma unroll
                for (int s = 0; s < S; ++s) lo = fminf(lo, fabsf(line[s])), plus = plus && line[s] > 0.0f, minus = minus && line[s] < 0.0f;
                const float stay = sm.small[(int)fminf(0.499f * lo * per_v, (float)ENC_SMALL)];
                if (__all_sync(0xffffffffu, (plus || minus) && fmaf(stay, 1.0f - ENC_REL, -ENC_ABS) > bound * (float)ENC_G)) continue;
            }
            enc_sort_line<S>(line);
            const float2 lh = enc_bounds<S, ENC_NB>(t, sm.chord, line);
            float least = lh.y * (1.0f / ENC_G);
#pragma unroll
            for (int o = 16; o; o >>= 1) least = fminf(least, __shfl_xor_sync(0xffffffffu, least, o));
            if (least < bound) bound = least;
            if (lane == 0 && least < told) atomicMin(reinterpret_cast<int*>(ub), __float_as_int(least)), told = least;     // (not negative: ordered like ints)
            // (a bound that is not a number leaves the candidate to its evaluation)
            if (c < q.total && !(lh.x > bound * (float)ENC_G)) sm.list[atomicAdd(&sm.n_list, 1)] = make_uint2((unsigned int)c, __float_as_uint(lh.x));
        }
        const float told2 = __ldcg(ub);
        const unsigned long long have = __ldcg(best);
        __syncthreads();
        bound = fminf(bound, fminf(told2, __uint_as_float((unsigned int)(have >> 32))));       // (no candidate yet: not a number, which fminf leaves out)
        const int n_list = sm.n_list;
        for (int e = tid; e < n_list; e += ENC_WT)
            if (!(__uint_as_float(sm.list[e].y) > bound * (float)ENC_G)) sm.alive[atomicAdd(&sm.n_alive, 1)] = (int)sm.list[e].x;
        __syncthreads();
        const int n_alive = sm.n_alive;
        if (n_alive <= 8 * ENC_WARPS) {
            for (int e = warp; e < n_alive; e += ENC_WARPS) {
                const int c = sm.alive[e];
                float line[S];
                __half2 pt[1 << S];
                enc_line<S>(sm, lines, c, line);
                enc_sort_line<S>(line);
                enc_line_points<S>(line, pt);
                float2 f[4];
                float sum = 0.0f;
#pragma unroll
                for (int k = 0; k < 4; ++k) f[k] = enc_err<S>(ds[lane + 32 * k], pt), sum += f[k].x + f[k].y;
                sum = enc_warp_sum(sum) * (1.0f / ENC_G);
                if (sum * (1.0f - 2e-5f) > bound) continue;    // (the sum in another order is off by some 2^-17 at most)
                const float mse = enc_ordered_mse(f, sm.err[warp], lane);
                bound = fminf(bound, mse);
                const unsigned long long key = ((unsigned long long)__float_as_uint(mse) << 32) | (unsigned int)c;
                if (lane == 0 && key < start_key && key < __ldcg(best)) atomicMin(best, key);
            }
        } else {                                   // values so small that the bounds say little: a thread per survivor
            for (int e0 = warp * 32; e0 < n_alive; e0 += ENC_WT) {
                const int c = sm.alive[min(e0 + lane, n_alive - 1)];
                float line[S];
                __half2 pt[1 << S];
                enc_line<S>(sm, lines, c, line);
                enc_sort_line<S>(line);
                enc_line_points<S>(line, pt);
                float s0 = 0.0f, s1 = 0.0f;
                bool alive = e0 + lane < n_alive;
                for (int i = 0; i < ENC_G / 2; i += 8) {
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        const float2 f = enc_err<S>(ds[i + e], pt);
                        s0 += f.x, s1 += f.y;
                    }
                    if ((s0 + s1) * (1.0f / ENC_G) > bound) alive = false;
                    if (!__any_sync(0xffffffffu, alive)) break;
                    if (i % 32 == 24) bound = fminf(bound, __uint_as_float((unsigned int)(__ldcg(best) >> 32)));
                }
                if (alive) {
                    const float mse = (s0 + s1) * (1.0f / ENC_G);
                    const unsigned long long key = ((unsigned long long)__float_as_uint(mse) << 32) | (unsigned int)c;
                    if (key < start_key && key < __ldcg(best)) atomicMin(best, key);
                    bound = fminf(bound, mse);
                }
            }
        }
        __syncthreads();
        if (tid == 0) sm.n_list = 0, sm.n_alive = 0;
    }
}

// ---- new lines against undecided groups ----------------------------------------------------------------------------------
// The groups are met in windows of one group per warp (all but one of a block's), which keep their group's values and best line in
// registers from step to step: only the first group that misses matters, so that the groups behind the window may wait for their
// lines until the window gets there.  A step compares one line with some 2 800 groups in registers; with every undecided group it read
// 16 384 rows and took 13 us.  The errors' sum in the order of an evaluation, two chains of 128 additions, is formed only where the
// sum in another order says that the line may be better.  A new window meets all lines since the walk's start: a warp makes a table of
// ENC_OWN chords of its group and bounds 32 lines at a time, a lane each (80 us a window of 2 800 groups and 150 lines; 125 one line after
// the other).
constexpr int ENC_UWARPS = ENC_WARPS - 1;
constexpr int ENC_OWN = 126;
constexpr int ENC_MANY = 8;                        // lines from which the table pays
static_assert(ENC_OWN + 2 <= ENC_G / 2, "EncFast::own");

// The chords of the group whose values a warp has in d[].
template <int S>
__device__ __forceinline__ EncTable enc_own_table(float2* chord, const EncStats& st, const __half2 (&d)[4], int lane) {
    constexpr int NB = ENC_OWN, PER = (NB + 31) / 32;
    EncTable t;
    t.mid = 0.5f * (st.d_max + st.d_min), t.R = 0.5f * (st.d_max - st.d_min);
    const float width = 2.0f * t.R / NB;
    t.inv = (float)NB / (2.0f * t.R);
    for (int i = lane; i < NB + 2; i += 32) chord[i] = make_float2(0.0f, 0.0f);
    __syncwarp();
    float sq = 0.0f;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float2 f = __half22float2(d[k]);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const float v = (h ? f.y : f.x) - t.mid;
            float2* b = chord + 1 + min(max(enc_interval<NB>(2.0f * v, t.inv) - 1, 0), NB - 1);
            atomicAdd(&b->x, 1.0f);
            atomicAdd(&b->y, v);
            sq = fmaf(v, v, sq);
        }
    }
    __syncwarp();
    float2 mine[PER];
    float n = 0.0f, sv = 0.0f, top = 0.0f;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        mine[i] = lane * PER + i < NB ? chord[1 + lane * PER + i] : make_float2(0.0f, 0.0f);
        n += mine[i].x, sv += mine[i].y, top = fmaxf(top, mine[i].x);
    }
    float n_in = n, s_in = sv;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const float a = __shfl_up_sync(0xffffffffu, n_in, o), b = __shfl_up_sync(0xffffffffu, s_in, o);
        if (lane >= o) n_in += a, s_in += b;
        top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
    }
    t.total = __shfl_sync(0xffffffffu, s_in, 31), t.squares = enc_warp_sum(sq), t.gap = 0.51f * top * width;
    float rank = n_in - n, below = s_in - sv;
    __syncwarp();
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        const int k = lane * PER + i;
        const float x0 = fmaf(width, (float)k, -t.R), x1 = fmaf(width, (float)(k + 1), -t.R), f0 = fmaf(rank, x0, -below);
        rank += mine[i].x, below += mine[i].y;
        const float f1 = fmaf(rank, x1, -below), slope = (f1 - f0) * t.inv;
        if (k < NB) chord[1 + k] = make_float2(0.5f * slope, fmaf(-slope, x0, f0));
    }
    if (lane == 0) chord[0] = make_float2(0.0f, 0.0f), chord[NB + 1] = make_float2(0.5f * ENC_G, -t.total);
    __syncwarp();
    return t;
}

// All blocks, the same decision: what becomes of group g, whose winner is `line` (ascending magnitudes, the same in every thread).
// Returns why the walk stops here (0: it does not).  `line_s`: the new line, if one is appended; `stored`: line threadIdx.x of the codebook,
// fetched before the winner was known.
template <int S>
__device__ __forceinline__ void enc_stored_line(const __half* lines, int i, unsigned short (&h)[S]) {
#pragma unroll
    for (int s = 0; s < S; ++s) h[s] = __ldcg(reinterpret_cast<const unsigned short*>(lines) + (size_t)i * S + s);
}
template <int S>
__device__ __forceinline__ int enc_decide(const EncRun& p, const float (&line)[S], const unsigned short (&stored)[S], int g, unsigned long long key,
                                          int& n, int& accepted, double* hist, int& hist_n, int& head, __half* line_s, bool& append) {
    __shared__ int at_s;
    float mag = 0.0f;
    bool twice = false;                            // two coefficients of one magnitude
#pragma unroll
    for (int s = 0; s < S; ++s) {
        if (s) twice = twice || !(fabsf(line[s]) > fabsf(line[s ? s - 1 : 0]));
        mag = __fadd_rn(mag, fabsf(line[s]));
    }
    append = false;
    if (twice) return 2;
    const float near = enc_h(__fmul_rn(enc_h(mag), 0.0001f));
    auto close = [&](const unsigned short (&h)[S]) {
        float m = 0.0f;
#pragma unroll
        for (int s = 0; s < S; ++s) m = __fadd_rn(m, fabsf(enc_h(__fsub_rn(__half2float(__ushort_as_half(h[s])), line[s]))));
        return enc_h(m) < near;
    };
    int at = 0x7fffffff;
    if ((int)threadIdx.x < n && close(stored)) at = threadIdx.x;
    for (int i = threadIdx.x + ENC_WT; i < n && at == 0x7fffffff; i += ENC_WT) {
        unsigned short h[S];
        enc_stored_line<S>(p.lines, i, h);
        if (close(h)) at = i;
    }
    if (threadIdx.x == 0) at_s = 0x7fffffff;
    append = !__syncthreads_or(at != 0x7fffffff);
    if (!append) {
        if (at != 0x7fffffff) atomicMin(&at_s, at);
        __syncthreads();
        at = at_s;
    } else {
        if (n >= p.capacity) return 2;
        at = n;
    }
    const float mse = __uint_as_float((unsigned int)(key >> 32));
    if (threadIdx.x == 0) {
#pragma unroll
        for (int s = 0; s < S; ++s) line_s[s] = __float2half_rn(line[s]);      // (exact: candidates are fp16 values)
        if (blockIdx.x == 0) {
            sbvr_encode_record_t r;
            r.group = g, r.at = at, r.mse = mse;
#pragma unroll
            for (int s = 0; s < 4; ++s) r.line[s] = s < S ? __half_as_ushort(__float2half_rn(line[s < S ? s : 0])) : (unsigned short)0;
            p.records[accepted] = r;
            if (append)
#pragma unroll
                for (int s = 0; s < S; ++s) __stcg(reinterpret_cast<unsigned short*>(p.lines) + (size_t)n * S + s, __half_as_ushort(__float2half_rn(line[s])));
        }
    }
    // the last `window` accepted errors, a ring with the oldest at `head`
    const int to = hist_n == p.window ? head : (head + hist_n) % p.window;
    if (threadIdx.x == 0) hist[to] = (double)mse;
    if (hist_n == p.window) head = (head + 1) % p.window;
    else ++hist_n;
    if (append) ++n;
    ++accepted;
    __syncthreads();
    return 0;
}

__device__ __forceinline__ double enc_cutoff(const double* hist, int n, int head, int window, double acceptable) {
    double sum = 0.0, c = 0.0;
    for (int i = 0; i < n; ++i) {
        const double x = hist[head + i < window ? head + i : head + i - window], t = __dadd_rn(sum, x);
        if (fabs(sum) >= fabs(x)) c = __dadd_rn(c, __dadd_rn(__dadd_rn(sum, -t), x));
        else c = __dadd_rn(c, __dadd_rn(__dadd_rn(x, -t), sum));
        sum = t;
    }
    if (c != 0.0 && isfinite(c)) sum = __dadd_rn(sum, c);
    const double m = __dmul_rn(__ddiv_rn(sum, (double)n), 0.99);
    return acceptable > m ? acceptable : m;        // Python's max(m, acceptable): the first unless the second is greater
}

template <int S>
__global__ void __launch_bounds__(ENC_WT, 1) encode_walk_kernel(const __grid_constant__ EncRun p) {
    extern __shared__ __align__(16) unsigned char smem[];
    EncFast<S>& sm = *reinterpret_cast<EncFast<S>*>(smem);
    __shared__ __align__(16) __half2 ds[ENC_G / 2];
    __shared__ double hist[ENC_WINDOW], cutoff_s;
    __shared__ __half line_s[S];
    __shared__ int miss_s, go_s;
    EncCtl* c = p.ctl;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, NG = p.q.NG;
    unsigned int round = 0;
    int n = p.n, misses = p.misses, accepted = 0, steps = 0, hist_n = p.hist_n, head = 0, from = p.from;
    const int rest = p.line0;                      // lines that the groups behind the window have met
    int base = from, end = from, met_lines = rest; // the window and the lines that its groups have met
    int stop = 0;
    unsigned int t = 0;                            // steps, of the slots in *c
    bool appended = false;                         // the last line is in line_s (and may not be in memory yet for all to see)
    float best = 0.0f;                             // this warp's group of the window: best mse, values
    __half2 d[4] = {};
    bool mine = false, loaded = false;

    for (int i = threadIdx.x; i < hist_n; i += ENC_WT) hist[i] = p.hist[i];
    enc_lists_init<S>(sm, p.q.space);
    auto clear = [&](int slot) { c->miss[slot] = NG, c->ub[slot] = INFINITY, c->best[slot] = ~0ull; };
    if (blockIdx.x == 0 && threadIdx.x == 0)
        for (int i = 0; i < 3; ++i) clear(i);
    bool met = enc_meet(c, round);
    while (met) {
        const bool warm = n < p.warmup;
        if (from >= NG) stop = SBVR_ENCODE_DONE;
        else if (!warm && n >= p.capacity) stop = SBVR_ENCODE_FULL;
        else if (!warm && hist_n == 0) stop = SBVR_ENCODE_CALLER;
        else if (steps >= p.limit) stop = SBVR_ENCODE_LIMIT;
        if (stop) break;
        const int slot = (int)(t % 3);
        int g = from;
        if (!warm) {
            if (from >= end) base = from, end = (int)min((long long)NG, (long long)from + (long long)gridDim.x * ENC_UWARPS), met_lines = rest, loaded = false;
            const int mg = base + (int)blockIdx.x * ENC_UWARPS + warp;
            if (!loaded) {
                mine = warp < ENC_UWARPS && mg < end;
                if (mine) {
                    best = __ldcg(p.best_mse + mg);
#pragma unroll
                    for (int k = 0; k < 4; ++k) d[k] = reinterpret_cast<const __half2*>(p.q.data + (size_t)mg * ENC_G)[lane + 32 * k];
                }
                loaded = true;
            }
            if (threadIdx.x == 0) miss_s = NG;
            if (warp == ENC_UWARPS && lane == 0) cutoff_s = enc_cutoff(hist, hist_n, head, p.window, p.acceptable);
            if (mine && mg >= from) {
                int at = -1;
                auto line_of = [&](int l, __half (&line)[S]) {
#pragma unroll
                    for (int s = 0; s < S; ++s)
                        line[s] = appended && l == n - 1 ? line_s[s]
                                                         : __ushort_as_half(__ldcg(reinterpret_cast<const unsigned short*>(p.lines) + (size_t)l * S + s));
                };
                auto meet_line = [&](int l) {
                    __half line[S];
                    __half2 pt[1 << S];
                    line_of(l, line);
                    enc_points<S>(line, pt);
                    float2 f[4];
                    float sum = 0.0f;
#pragma unroll
                    for (int k = 0; k < 4; ++k) f[k] = enc_err<S>(d[k], pt), sum += f[k].x + f[k].y;
                    sum = enc_warp_sum(sum) * (1.0f / ENC_G);
                    if (sum * (1.0f - 2e-5f) > best) return;
                    const float mse = enc_ordered_mse(f, sm.err[warp], lane);
                    if (mse < best) best = mse, at = l;
                };
                const EncStats own = n - met_lines >= ENC_MANY ? p.q.stats[mg] : EncStats{0.0f, 0.0f, 0.0f, 0.0f};
                if (enc_boundable(own)) {
                    // (the table lies where enc_ordered_mse puts its errors: the lines that may be better are noted first)
                    for (int l0 = met_lines; l0 < n; l0 += 32 * 32) {
                        const EncTable table = enc_own_table<S>(sm.own[warp], own, d, lane);
                        unsigned int maybe = 0;        // lane k: of lines l0 + 32 k ..
                        float bound = best;
                        const int last = min(32, (n - l0 + 31) / 32);
#pragma unroll 1
                        for (int k = 0; k < last; ++k) {
                            const int l = l0 + 32 * k + lane;
                            __half line[S];
                            float lf[S];
                            line_of(min(l, n - 1), line);
#pragma unroll
                            for (int s = 0; s < S; ++s) lf[s] = __half2float(line[s]);
                            const float2 lh = enc_bounds<S, ENC_OWN>(table, sm.own[warp], lf);
                            float least = lh.y * (1.0f / ENC_G);
#pragma unroll
                            for (int o = 16; o; o >>= 1) least = fminf(least, __shfl_xor_sync(0xffffffffu, least, o));
                            bound = fminf(bound, least);
                            const unsigned int m = __ballot_sync(0xffffffffu, l < n && !(lh.x > bound * (float)ENC_G));
                            if (lane == k) maybe = m;
                        }
                        __syncwarp();
#pragma unroll 1
                        for (int k = 0; k < last; ++k)
#pragma unroll 1
                            for (unsigned int m = __shfl_sync(0xffffffffu, maybe, k); m; m &= m - 1) meet_line(l0 + 32 * k + __ffs((int)m) - 1);
                    }
                } else {
                    for (int l = met_lines; l < n; ++l) meet_line(l);
                }
                if (at >= 0 && lane == 0) {
                    __stcg(p.best_mse + mg, best);
                    __stcg(p.best_at + mg, at);
                }
            }
            met_lines = n;
            appended = false;
            __syncthreads();
            if (mine && mg >= from && lane == 0 && !((double)best < cutoff_s)) atomicMin(&miss_s, mg);
            __syncthreads();
            if (threadIdx.x == 0 && miss_s < NG) atomicMin(&c->miss[slot], miss_s);
            if (!(met = enc_meet(c, round))) break;
            g = __ldcg(&c->miss[slot]);
            // everyone has read the words of the step before: its slot is that of the step after the next
            if (blockIdx.x == 0 && threadIdx.x == 0) clear((int)((t + 2) % 3));
            if (g >= NG) {                         // every group of the window is served
                from = end;
                ++t;
                continue;
            }
        }
        const float cached = warm ? INFINITY : __ldcg(p.best_mse + g);
        // extended search while the codebook serves well: hits / seen > 0.6
        const bool ext = warm || (double)(g - misses) / (double)(g + 1) > 0.6;
        const EncSpace& sp = p.q.space[ext ? 1 : 0];
        const EncStats st = p.q.stats[g];
        EncGroup<S> q;
        if (!q.init(st, sp, ext)) {
            stop = SBVR_ENCODE_CALLER;
            from = g;                              // (every group in front of it is served)
            break;
        }
        for (int i = threadIdx.x; i < ENC_G / 2; i += ENC_WT) ds[i] = reinterpret_cast<const __half2*>(p.q.data + (size_t)g * ENC_G)[i];
        __syncthreads();
        unsigned short stored[S] = {};
        if ((int)threadIdx.x < n) enc_stored_line<S>(p.lines, threadIdx.x, stored);
        if (appended && (int)threadIdx.x == n - 1)             // (of the decision before, with no meeting since: while warming up)
#pragma unroll
            for (int s = 0; s < S; ++s) stored[s] = __half_as_ushort(line_s[s]);
        const bool bounded = enc_boundable(st) && enc_lines_fit<S>(q, sp);
        EncLines lines;
        if (bounded) enc_search_bounded<S>(sm, q, sp, st, ds, cached, ext, &c->best[slot], &c->ub[slot], lines);
        else enc_search<S, ENC_WT>(q, sp, ds, cached, &c->best[slot]);
        if (!(met = enc_meet(c, round))) break;
        if (blockIdx.x == 0 && threadIdx.x == 32) {
            if (warm) clear((int)((t + 2) % 3));
            asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(&c->go), "r"(t + 1u) : "memory");
        }
        const unsigned long long key = __ldcg(&c->best[slot]);
        appended = false;
        if (key < ((unsigned long long)__float_as_uint(cached) << 32)) {       // (else the codebook already has something at least as good)
            float line[S];
            if (bounded) enc_line<S>(sm, lines, (int)(key & 0xffffffffu), line);
            else enc_candidate<S>(sp, (int)(key & 0xffffffffu), q.ns, q.s_start, q.s_step, q.a0, q.a1, line);
            enc_sort_line<S>(line);
            if (enc_decide<S>(p, line, stored, g, key, n, accepted, hist, hist_n, head, line_s, appended)) {
                stop = SBVR_ENCODE_CALLER;
                from = g;
                break;
            }
        }
        ++misses, ++steps, ++t, from = g + 1;
        // Nobody acts on a decision that block 0, for want of a meeting, has not taken.
        if (threadIdx.x == 0) go_s = blockIdx.x == 0 || enc_reached(&c->go, t) ? 1 : 0;
        __syncthreads();
        met = go_s != 0;
    }
    // Blocks that have not met -- another stream's kernel keeps some from running -- leave the walk at the last decision, with the lines that
    // every group has met: a line that a group meets a second time changes nothing.
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        p.outcome[0] = met ? stop : SBVR_ENCODE_TIMEOUT;
        p.outcome[1] = from, p.outcome[2] = n, p.outcome[3] = met && end >= NG ? met_lines : rest, p.outcome[4] = misses, p.outcome[5] = accepted;
    }
}

template <int S>
static int encode_run(const EncRun& r, int sm_count, cudaStream_t st) {
    int per_sm = 0;
    static SmemOnce once;
    const int smem = (int)sizeof(EncFast<S>), rc = set_max_smem_once(once, encode_walk_kernel<S>, smem);
    if (rc) return rc;
    SBVR_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, encode_walk_kernel<S>, ENC_WT, smem));
    if (per_sm < 1) return SBVR_ERR_UNSUPPORTED;
    EncRun copy = r;
    void* args[] = {&copy};
    SBVR_CUDA_TRY(cudaMemsetAsync(r.ctl, 0, sizeof(EncCtl), st));
    SBVR_CUDA_TRY(cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(encode_walk_kernel<S>), dim3(sm_count), dim3(ENC_WT),
                                              args, (size_t)smem, st));
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
