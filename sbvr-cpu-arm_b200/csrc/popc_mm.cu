// SBVR x SBVR product: both operands are bit-plane encoded.
//
//   y[m][n] = sum_g sum_{a < LS} sum_{b < RS} popc( l_a[m, g] & r_b[n, g] ) * cl[g, m, a] * cr[g, n, b]  (+ bias[n])
//
// l_a[m, g], r_b[n, g] = the 256 bits of plane a / b of row m / n in group g; cl, cr = the fp16 coefficient lines
// the index tensors select.  Replaces `_sbvr_mm_T` / cuda_1xtN_sbvr_mm_T of the reference
// (sbvr/kernels/sbvr_ops.cpp:35-76, sbvr/kernels/sbvr_kernel.cu:464-562, launch :914-1023) on the same layouts:
//   l_bvr u32 [K/32, M, LS], l_idx u8|u16 [K/256, M], l_cache f16 [Cl, LS];   r_* likewise with N, RS.
// Differences from the reference kernel, both on the side of accuracy: counts are kept in 32 bits (the reference's uchar
// counters wrap at 256, sbvr_kernel.cu:486-487) and the coefficient products and sums are fp32 (the reference multiplies in
// half2).
//
// The counts are integer tensor-core products: `w & (0x01010101 << j)` turns bits j, j + 8, j + 16, j + 24 of a packed word
// into four bytes of 0 or 2^j, which is how mma.sync m16n8k32 (u8 x u8 -> s32) wants an operand register; the other operand's
// word is shifted so that the same bits are worth 2^(7 - j), and every product of two set bits is 128.  Both operands go from
// global memory to the MMA without shared memory.  A tile: sixteen (weight row, plane) pairs; B tile: eight
// (activation row, plane) pairs; thread t of a quad holds word t of four, and the four pairs of bit positions of those words
// are four MMAs.  Per group of 256 k the counts (times 128, accumulated on top of 2^23's bit pattern, so that reading them as floats is
// one subtraction) are multiplied by the two coefficients and added in fp32.
//
// Measured (four planes on both sides, us; popcount instructions on CUDA cores, a sixteenth of the lanes each, in brackets):
// 4096 x 4096: M = 1 7.1 (8.3), M = 4 9.4 (15.6), M = 16 24.4 (50); 14336 x 4096: M = 2 22 (25), M = 4 32 (41).  Bound by instruction
// issue at 335 per warp and group of 32 weight-plane rows; 0.8 us of a call is the wait for the kernel in front, which may
// be writing either operand.  With one activation row half of the columns are empty: on large weights popcounts win (popc_few_rows).
#include "common.cuh"

namespace sbvr {

constexpr int PM_WARPS = 4;
constexpr int PM_THREADS = 32 * PM_WARPS;
constexpr int PM_TW = 2;                            // A tiles of a warp
constexpr int PM_MAGIC = 0x4B000000;                // 2^23 as a float

struct PmParams {
    const uint32_t* l_bvr;
    const void* l_idx;
    const __half* l_cache;
    const uint32_t* r_bvr;
    const void* r_idx;
    const __half* r_cache;
    const __half* bias;
    __half* y;
    int l_idx_bytes, r_idx_bytes, M, N, K;
    int ks;                                         // warps of a CTA that share rows and split the groups (1, 2, 4, 8)
};

__device__ __forceinline__ void pm_mma(int (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.u8.u8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

template <int LS, int RS, int NT>
__global__ void __launch_bounds__(PM_THREADS, NT <= 2 ? 4 : 2) popc_mm_kernel(const PmParams p) {
    constexpr int LP = (LS == 3) ? 4 : LS, RP = (RS == 3) ? 4 : RS;     // columns / rows per activation / weight row
    constexpr int CM = 8 / LP, MT = NT * CM;        // activation rows per B tile, of a CTA
    constexpr int WR = PM_TW * 16 / RP;             // weight rows of a warp
    __shared__ float red[PM_WARPS][WR][MT];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, t = lane & 3;
    const int M = p.M, N = p.N, KB = p.K / 256, ks = p.ks;
    const int rb = (int)blockIdx.x * (PM_WARPS / ks) + warp / ks, sl = warp % ks;
    const int g0 = KB * sl / ks, g1 = KB * (sl + 1) / ks;
    const int m0 = (int)blockIdx.y * MT;
    pdl_launch_dependents();

    struct Group {
        uint32_t a[PM_TW][2][2], b[NT][2];          // [tile][row g, g + 8][four words], [tile][four words]
        __half cr[PM_TW][2], cl[NT][2];
    };
    // Rows and columns beyond the operands repeat the first one; their coefficients are zero.  Everything is addressed by 32-bit
    // offsets from the operands' starts (checked by the host), which advance by a constant per group.
    uint32_t ow[PM_TW][2], oc[PM_TW][2], on[PM_TW][2];    // word, coefficient inside a line, line number of this thread's A rows
    bool live_r[PM_TW][2];
#pragma unroll
    for (int i = 0; i < PM_TW; ++i)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int pr = (rb * PM_TW + i) * 16 + h * 8 + g;
            const int n = pr / RP, b = pr % RP;
            live_r[i][h] = n < N && b < RS;
            on[i][h] = live_r[i][h] ? (uint32_t)n : 0u, oc[i][h] = live_r[i][h] ? (uint32_t)b : 0u;
            ow[i][h] = ((uint32_t)t * N + on[i][h]) * RS + oc[i][h];
        }
    uint32_t lw[NT], lc[NT][2], lm[NT][2];
    bool live_l[NT][2];
#pragma unroll
    for (int j = 0; j < NT; ++j) {
        int m = m0 + j * CM + g / LP, a = g % LP;
        if (m >= M || a >= LS) m = 0, a = 0;
        lw[j] = ((uint32_t)t * M + m) * LS + a;
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int me = m0 + j * CM + (2 * t + e) / LP, ae = (2 * t + e) % LP;
            live_l[j][e] = me < M && ae < LS;
            lm[j][e] = live_l[j][e] ? (uint32_t)me : 0u, lc[j][e] = live_l[j][e] ? (uint32_t)ae : 0u;
        }
    }
    const uint32_t rs4 = 4u * N * RS, ls4 = 4u * M * LS;  // four word rows
    // The warp's share of the weight is requested into L2 at once (up to 32 groups of it), a line of line numbers or of words per
    // lane: a group's loads then wait for L2 only.
    {
        const int nr = min(rb * WR, N - 1);
        const int pg = min(g1, g0 + 32);
        if (g0 + lane < pg) {
            const char* a = reinterpret_cast<const char*>(p.r_idx) + ((size_t)(g0 + lane) * N + nr) * p.r_idx_bytes;
            asm volatile("prefetch.global.L2 [%0];" ::"l"(a));
        }
        for (int kw = g0 * 8 + lane; kw < pg * 8; kw += 32) asm volatile("prefetch.global.L2 [%0];" ::"l"(p.r_bvr + ((size_t)kw * N + nr) * RS));
    }
    struct Lines {
        uint32_t r[PM_TW][2], l[NT][2];             // codebook lines of a group
    };
    auto lines_r = [&](int gr, Lines& q) {
        if (gr >= g1) return;
        const uint32_t o = (uint32_t)gr * N;
        if (p.r_idx_bytes == 1) {
#pragma unroll
            for (int i = 0; i < 2 * PM_TW; ++i) q.r[i / 2][i % 2] = __ldg(reinterpret_cast<const uint8_t*>(p.r_idx) + o + on[i / 2][i % 2]);
        } else {
#pragma unroll
            for (int i = 0; i < 2 * PM_TW; ++i) q.r[i / 2][i % 2] = __ldg(reinterpret_cast<const uint16_t*>(p.r_idx) + o + on[i / 2][i % 2]);
        }
    };
    auto lines_l = [&](int gr, Lines& q) {
        if (gr >= g1) return;
        const uint32_t o = (uint32_t)gr * M;
        if (p.l_idx_bytes == 1) {
#pragma unroll
            for (int j = 0; j < 2 * NT; ++j) q.l[j / 2][j % 2] = __ldg(reinterpret_cast<const uint8_t*>(p.l_idx) + o + lm[j / 2][j % 2]);
        } else {
#pragma unroll
            for (int j = 0; j < 2 * NT; ++j) q.l[j / 2][j % 2] = __ldg(reinterpret_cast<const uint16_t*>(p.l_idx) + o + lm[j / 2][j % 2]);
        }
    };
    auto load_r = [&](int gr, const Lines& ln, Group& q) {
        if (gr >= g1) return;
        const uint32_t* w = p.r_bvr + (size_t)gr * 2 * rs4;
#pragma unroll
        for (int i = 0; i < PM_TW; ++i)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                q.a[i][h][0] = __ldcs(w + ow[i][h]), q.a[i][h][1] = __ldcs(w + rs4 + ow[i][h]);
                q.cr[i][h] = __ldg(p.r_cache + ln.r[i][h] * RS + oc[i][h]);
            }
    };
    auto load_l = [&](int gr, const Lines& ln, Group& q) {
        if (gr >= g1) return;
        const uint32_t* w = p.l_bvr + (size_t)gr * 2 * ls4;
#pragma unroll
        for (int j = 0; j < NT; ++j) {
            q.b[j][0] = __ldg(w + lw[j]), q.b[j][1] = __ldg(w + ls4 + lw[j]);
#pragma unroll
            for (int e = 0; e < 2; ++e) q.cl[j][e] = __ldg(p.l_cache + ln.l[j][e] * LS + lc[j][e]);
        }
    };
    float acc[PM_TW][NT][4];
#pragma unroll
    for (int i = 0; i < PM_TW; ++i)
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.0f;
    auto multiply = [&](const Group& q) {
        int d[PM_TW][NT][4];
#pragma unroll
        for (int i = 0; i < PM_TW; ++i)
#pragma unroll
            for (int j = 0; j < NT; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) d[i][j][e] = PM_MAGIC;
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
            for (int b = 0; b < 8; b += 2) {
                uint32_t b0[NT], b1[NT];
#pragma unroll
                for (int j = 0; j < NT; ++j) {     // bit b of a byte moves to 7 - b
                    const uint32_t w = q.b[j][c];
                    const int s0 = 7 - 2 * b, s1 = 5 - 2 * b;
                    b0[j] = (s0 > 0 ? w << s0 : w >> -s0) & (0x80808080u >> b), b1[j] = (s1 > 0 ? w << s1 : w >> -s1) & (0x40404040u >> b);
                }
#pragma unroll
                for (int i = 0; i < PM_TW; ++i) {
                    const uint32_t w0 = q.a[i][0][c], w1 = q.a[i][1][c];
                    const uint32_t a[4] = {w0 & (0x01010101u << b), w1 & (0x01010101u << b), w0 & (0x02020202u << b), w1 & (0x02020202u << b)};
#pragma unroll
                    for (int j = 0; j < NT; ++j) pm_mma(d[i][j], a, b0[j], b1[j]);
                }
            }
        float cr[PM_TW][2], cl[NT][2];
#pragma unroll
        for (int i = 0; i < 2 * PM_TW; ++i) cr[i / 2][i % 2] = live_r[i / 2][i % 2] ? __half2float(q.cr[i / 2][i % 2]) * (1.0f / 128) : 0.0f;
#pragma unroll
        for (int j = 0; j < 2 * NT; ++j) cl[j / 2][j % 2] = live_l[j / 2][j % 2] ? __half2float(q.cl[j / 2][j % 2]) : 0.0f;
#pragma unroll
        for (int i = 0; i < PM_TW; ++i)
#pragma unroll
            for (int j = 0; j < NT; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    acc[i][j][e] = fmaf((__int_as_float(d[i][j][e]) - 8388608.0f) * cl[j][e & 1], cr[i][e >> 1], acc[i][j][e]);
    };
    // Two groups are on their way while one is multiplied, and the line numbers of a third: a group's line number, line and
    // words cost two round trips to memory, several times what its MMAs take.
    Group q[3];
    Lines ln, ln1;
    pdl_wait();                                     // either operand may be an encoding that the kernel in front is writing
    lines_r(g0, ln);
    lines_r(g0 + 1, ln1);
    lines_l(g0, ln);
    lines_l(g0 + 1, ln1);
    load_r(g0, ln, q[0]);
    load_r(g0 + 1, ln1, q[1]);
    load_l(g0, ln, q[0]);
    load_l(g0 + 1, ln1, q[1]);
    lines_r(g0 + 2, ln);
    lines_l(g0 + 2, ln);
#pragma unroll 1
    for (int gr = g0; gr < g1; gr += 3) {
#pragma unroll
        for (int u = 0; u < 3; ++u) {
            if (gr + u >= g1) break;
            load_r(gr + u + 2, ln, q[(u + 2) % 3]);
            load_l(gr + u + 2, ln, q[(u + 2) % 3]);
            lines_r(gr + u + 3, ln);
            lines_l(gr + u + 3, ln);
            multiply(q[u]);
        }
    }
    // planes of an activation row are neighbouring columns, those of a weight row neighbouring rows
#pragma unroll
    for (int i = 0; i < PM_TW; ++i)
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                float v = acc[i][j][2 * h] + acc[i][j][2 * h + 1];
                if (LP == 4) v += __shfl_xor_sync(0xffffffffu, v, 1);
#pragma unroll
                for (int o = 4; o < 4 * RP; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                if (g % RP == 0 && (2 * t) % LP == 0) red[warp][(i * 16 + h * 8 + g) / RP][j * CM + 2 * t / LP] = v;
            }
    __syncthreads();
    // the slices of a row in order
    const int rows = (PM_WARPS / ks) * WR;
    for (int e = threadIdx.x; e < rows * MT; e += PM_THREADS) {
        const int r = e % rows, ml = e / rows, m = m0 + ml, n = (int)blockIdx.x * rows + r;
        if (n >= N || m >= M) continue;
        float v = 0.0f;
        for (int s = 0; s < ks; ++s) v += red[(r / WR) * ks + s][r % WR][ml];
        if (p.bias) v += __half2float(p.bias[n]);
        p.y[(size_t)m * N + n] = __float2half_rn(v);
    }
}

template <int LS, int RS, int NT>
static int popc_launch_nt(PmParams p, int sm_count, cudaStream_t st) {
    constexpr int MT = NT * (8 / (LS == 3 ? 4 : LS)), WR = PM_TW * 16 / (RS == 3 ? 4 : RS);
    // The groups are split over the warps of a CTA as long as all CTAs fit at once (four per SM by their registers, two with four tiles).
    const long long gy = (p.M + MT - 1) / MT, whole = (p.N + PM_WARPS * WR - 1) / (PM_WARPS * WR);
    p.ks = 1;
    while (p.ks * 2 <= PM_WARPS && p.ks * 2 <= p.K / 256 && whole * gy * p.ks * 2 <= (NT <= 2 ? 4 : 2) * sm_count) p.ks *= 2;
    const int rows = (PM_WARPS / p.ks) * WR;
    const dim3 grid((p.N + rows - 1) / rows, (p.M + MT - 1) / MT);
    SBVR_CUDA_TRY(launch_pdl(popc_mm_kernel<LS, RS, NT>, grid, dim3(PM_THREADS), 0, st, p));
    return SBVR_OK;
}
// ---------------------------------------------------------------------------------------------
// One or two activation rows on large weights: popcount instructions.  A warp owns 32 / RP weight rows (RP = planes per row, 4 for
// RS = 3) and a quarter of K; lane = (row, plane) reads one packed word per 32 k, 128 contiguous bytes per warp.  The left operand
// (at most 8 rows per pass) sits in shared memory with its coefficients.
// ---------------------------------------------------------------------------------------------
constexpr int PF_MT = 8;               // left rows per pass
constexpr int PF_KQ = 4;               // K quarters per row block (one warp each)
constexpr int PF_RB = 2;               // row blocks per CTA
constexpr int PF_THREADS = 32 * PF_KQ * PF_RB;

template <int LS, int RS>
__global__ void __launch_bounds__(PF_THREADS) popc_few_kernel(const uint32_t* __restrict__ l_bvr, const void* __restrict__ l_idx,
                                                             int l_idx_bytes, const __half* __restrict__ l_cache,
                                                             const uint32_t* __restrict__ r_bvr, const void* __restrict__ r_idx,
                                                             int r_idx_bytes, const __half* __restrict__ r_cache,
                                                             const __half* __restrict__ bias, __half* __restrict__ y, int M,
                                                             int m0, int N, int K) {
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr int RP = (RS == 3) ? 4 : RS;
    constexpr int ROWS = 32 / RP;                       // weight rows per warp
    const int KW = K / 32, KB = K / 256;
    const int mt = min(PF_MT, M - m0);
    uint32_t* lw = reinterpret_cast<uint32_t*>(smem);                       // [KW][mt][LS]
    float* lc = reinterpret_cast<float*>(smem + (size_t)KW * PF_MT * LS * 4);   // [KB][mt][LS]
    float* red = lc + (size_t)KB * PF_MT * LS;                               // [PF_RB][PF_KQ][PF_MT][ROWS]
    pdl_launch_dependents();
    pdl_wait();
    for (int i = threadIdx.x; i < KW * mt * LS; i += PF_THREADS) {
        const int a = i % LS, m = (i / LS) % mt, kw = i / (LS * mt);
        lw[(kw * PF_MT + m) * LS + a] = l_bvr[((size_t)kw * M + m0 + m) * LS + a];
    }
    for (int i = threadIdx.x; i < KB * mt * LS; i += PF_THREADS) {
        const int a = i % LS, m = (i / LS) % mt, g = i / (LS * mt);
        const size_t e = (size_t)g * M + m0 + m;
        const size_t line = (l_idx_bytes == 1) ? reinterpret_cast<const uint8_t*>(l_idx)[e]
                                               : reinterpret_cast<const uint16_t*>(l_idx)[e];
        lc[(g * PF_MT + m) * LS + a] = __half2float(l_cache[line * LS + a]);
    }
    __syncthreads();

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rb = warp / PF_KQ, kq = warp % PF_KQ;
    const int n = ((int)blockIdx.x * PF_RB + rb) * ROWS + lane / RP, b = lane % RP;
    const bool live = (n < N) && (b < RS);
    const int g0 = (KB * kq) / PF_KQ, g1 = (KB * (kq + 1)) / PF_KQ;
    float acc[PF_MT];
#pragma unroll
    for (int m = 0; m < PF_MT; ++m) acc[m] = 0.0f;
    for (int g = g0; g < g1; ++g) {                     // (two groups in flight cost occupancy here: 17.7 -> 26 us at 14336 x 4096)
        uint32_t rw[8];
        float cr = 0.0f;
#pragma unroll
        for (int kw = 0; kw < 8; ++kw) rw[kw] = live ? __ldcs(r_bvr + ((size_t)(g * 8 + kw) * N + n) * RS + b) : 0u;
        if (live) {
            const size_t e = (size_t)g * N + n;
            const size_t line = (r_idx_bytes == 1) ? reinterpret_cast<const uint8_t*>(r_idx)[e]
                                                   : reinterpret_cast<const uint16_t*>(r_idx)[e];
            cr = __half2float(r_cache[line * RS + b]);
        }
#pragma unroll
        for (int m = 0; m < PF_MT; ++m) {
            if (m < mt) {
                float s = 0.0f;
#pragma unroll
                for (int a = 0; a < LS; ++a) {
                    int cnt = 0;
#pragma unroll
                    for (int kw = 0; kw < 8; ++kw) cnt += __popc(lw[((g * 8 + kw) * PF_MT + m) * LS + a] & rw[kw]);
                    s += lc[(g * PF_MT + m) * LS + a] * (float)cnt;
                }
                acc[m] += cr * s;
            }
        }
    }
    // planes of a row sit in neighbouring lanes; then the K quarters meet in shared memory, in a fixed order
#pragma unroll
    for (int m = 0; m < PF_MT; ++m) {
#pragma unroll
        for (int o = RP / 2; o; o >>= 1) acc[m] += __shfl_xor_sync(0xffffffffu, acc[m], o);
        if (b == 0) red[((rb * PF_KQ + kq) * PF_MT + m) * ROWS + lane / RP] = acc[m];
    }
    __syncthreads();
    for (int i = threadIdx.x; i < PF_RB * mt * ROWS; i += PF_THREADS) {
        const int r = i % ROWS, m = (i / ROWS) % mt, rbb = i / (ROWS * mt);
        const int nn = ((int)blockIdx.x * PF_RB + rbb) * ROWS + r;
        if (nn >= N) continue;
        float v = 0.0f;
#pragma unroll
        for (int q = 0; q < PF_KQ; ++q) v += red[((rbb * PF_KQ + q) * PF_MT + m) * ROWS + r];
        if (bias) v += __half2float(bias[nn]);
        y[(size_t)(m0 + m) * N + nn] = __float2half_rn(v);
    }
}

template <int LS, int RS>
static size_t popc_few_smem(int K) {
    constexpr int ROWS = 32 / ((RS == 3) ? 4 : RS);
    return (size_t)(K / 32) * PF_MT * LS * 4 + (size_t)(K / 256) * PF_MT * LS * 4 + (size_t)PF_RB * PF_KQ * PF_MT * ROWS * 4;
}
template <int LS, int RS>
static int popc_launch_few(const PmParams& p, cudaStream_t st) {
    constexpr int ROWS = 32 / ((RS == 3) ? 4 : RS);
    const size_t smem = popc_few_smem<LS, RS>(p.K);
    if (smem > 200 * 1024) return SBVR_ERR_UNSUPPORTED;
    static SmemOnce once;
    const int rc = set_max_smem_once(once, popc_few_kernel<LS, RS>, 200 * 1024);
    if (rc) return rc;
    const int blocks = (p.N + PF_RB * ROWS - 1) / (PF_RB * ROWS);
    for (int m0 = 0; m0 < p.M; m0 += PF_MT)
        SBVR_CUDA_TRY(launch_pdl(popc_few_kernel<LS, RS>, dim3(blocks), dim3(PF_THREADS), smem, st, p.l_bvr, p.l_idx, p.l_idx_bytes,
                                 p.l_cache, p.r_bvr, p.r_idx, p.r_idx_bytes, p.r_cache, p.bias, p.y, p.M, m0, p.N, p.K));
    return SBVR_OK;
}

// Where popcounts are faster (four planes on the right, us, tensor cores in brackets): M = 1 with four planes on the left 8192 x 4096
// 10.8 (11.1), 14336 x 4096 17.8 (21.3), 16384 x 8192 32 (42), with two 9.1 (11.2), 15 (21), 26 (43); M = 2 with two planes 14336 x 4096
// 17.7 (21.4), 16384 x 8192 32 (43), but 8192 x 4096 12.6 (11.2), and with four 25 (21) at 14336 x 4096; up to 4096 rows
// never: 8.3 (7.1) at 4096 x 4096.
template <int LS, int RS>
static bool popc_few_rows(const PmParams& p, int sm_count) {
    constexpr int ROWS = 32 / ((RS == 3) ? 4 : RS);
    const long long blocks = (p.N + PF_RB * ROWS - 1) / (PF_RB * ROWS);
    if (popc_few_smem<LS, RS>(p.K) > 200 * 1024) return false;
    return (p.M == 1 && blocks > 3LL * sm_count) || (p.M == 2 && LS == 2 && blocks > 5LL * sm_count);
}

template <int LS, int RS>
static int popc_launch(const PmParams& p, cudaStream_t st) {
    constexpr int CM = 8 / (LS == 3 ? 4 : LS);
    int dev = 0;
    SBVR_CUDA_TRY(cudaGetDevice(&dev));
    DeviceInfo di;
    const int rc = device_info(dev, &di);
    if (rc) return rc;
    // the tensor-core kernel addresses by 32-bit offsets and has its passes over M in grid.y
    const bool fits = (long long)p.N * RS * 8 < (1LL << 31) && (long long)p.M * LS * 8 < (1LL << 31) &&
                      (long long)(p.K / 256) * (p.N > p.M ? p.N : p.M) < (1LL << 32) && (p.M + 4 * CM - 1) / (4 * CM) <= 65535;
    if (!fits || popc_few_rows<LS, RS>(p, di.sm_count)) return popc_launch_few<LS, RS>(p, st);
    const int tiles = (p.M + CM - 1) / CM;
    return tiles <= 1 ? popc_launch_nt<LS, RS, 1>(p, di.sm_count, st) : tiles <= 2 ? popc_launch_nt<LS, RS, 2>(p, di.sm_count, st) : popc_launch_nt<LS, RS, 4>(p, di.sm_count, st);
}

}  // namespace sbvr

using namespace sbvr;

extern "C" int sbvr_popc_mm_f16(const uint32_t* l_bvr, const void* l_idx, int l_idx_bytes, const void* l_cache, int Cl, int LS,
                                 const uint32_t* r_bvr, const void* r_idx, int r_idx_bytes, const void* r_cache, int Cr, int RS,
                                 const void* bias, void* y, int M, int N, int K, sbvr_stream_t stream) {
    if (!l_bvr || !l_idx || !l_cache || !r_bvr || !r_idx || !r_cache || !y) return SBVR_ERR_BAD_ARG;
    if (M < 1 || N < 1 || K < 1 || Cl < 1 || Cr < 1) return SBVR_ERR_BAD_ARG;
    if ((l_idx_bytes != 1 && l_idx_bytes != 2) || (r_idx_bytes != 1 && r_idx_bytes != 2)) return SBVR_ERR_BAD_ARG;
    if ((l_idx_bytes == 1 && Cl > 256) || (r_idx_bytes == 1 && Cr > 256) || Cl > 65536 || Cr > 65536) return SBVR_ERR_BAD_ARG;
    if (K % 256) return SBVR_ERR_SHAPE;
    if ((reinterpret_cast<uintptr_t>(l_bvr) | reinterpret_cast<uintptr_t>(r_bvr)) & 3) return SBVR_ERR_ALIGN;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    PmParams p;
    p.l_bvr = l_bvr, p.l_idx = l_idx, p.l_cache = reinterpret_cast<const __half*>(l_cache);
    p.r_bvr = r_bvr, p.r_idx = r_idx, p.r_cache = reinterpret_cast<const __half*>(r_cache);
    p.bias = reinterpret_cast<const __half*>(bias), p.y = reinterpret_cast<__half*>(y);
    p.l_idx_bytes = l_idx_bytes, p.r_idx_bytes = r_idx_bytes, p.M = M, p.N = N, p.K = K, p.ks = 1;
#define SBVR_PM(L_, R_) \
    if (LS == L_ && RS == R_) return popc_launch<L_, R_>(p, st)
    SBVR_PM(2, 2);
    SBVR_PM(2, 3);
    SBVR_PM(2, 4);
    SBVR_PM(3, 2);
    SBVR_PM(3, 3);
    SBVR_PM(3, 4);
    SBVR_PM(4, 2);
    SBVR_PM(4, 3);
    SBVR_PM(4, 4);
#undef SBVR_PM
    return SBVR_ERR_UNSUPPORTED;
}
