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
// 4096 x 4096: M = 1 6.4 (8.3), M = 4 8.4 (15.6), M = 16 24.8 (50); 14336 x 4096: M = 1 21.9 (17.9: half of the columns are
// empty), M = 2 22 (25), M = 4 31 (42).  Bound by instruction issue at 335 per warp and group of 32 weight-plane rows.
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
    lines_r(g0, ln);                                // the weight does not depend on the kernel in front
    lines_r(g0 + 1, ln1);
    load_r(g0, ln, q[0]);
    load_r(g0 + 1, ln1, q[1]);
    pdl_wait();
    lines_l(g0, ln);
    lines_l(g0 + 1, ln1);
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
static int popc_launch_nt(PmParams p, cudaStream_t st) {
    constexpr int MT = NT * (8 / (LS == 3 ? 4 : LS)), WR = PM_TW * 16 / (RS == 3 ? 4 : RS);
    // The groups are split over the warps of a CTA as long as all CTAs fit at once (four per SM by their registers, two with four tiles).
    int dev = 0;
    SBVR_CUDA_TRY(cudaGetDevice(&dev));
    DeviceInfo di;
    const int rc = device_info(dev, &di);
    if (rc) return rc;
    const long long gy = (p.M + MT - 1) / MT, whole = (p.N + PM_WARPS * WR - 1) / (PM_WARPS * WR);
    p.ks = 1;
    while (p.ks * 2 <= PM_WARPS && p.ks * 2 <= p.K / 256 && whole * gy * p.ks * 2 <= (NT <= 2 ? 4 : 2) * di.sm_count) p.ks *= 2;
    const int rows = (PM_WARPS / p.ks) * WR;
    const dim3 grid((p.N + rows - 1) / rows, (p.M + MT - 1) / MT);
    if (grid.y > 65535) return SBVR_ERR_SHAPE;
    SBVR_CUDA_TRY(launch_pdl(popc_mm_kernel<LS, RS, NT>, grid, dim3(PM_THREADS), 0, st, p));
    return SBVR_OK;
}
template <int LS, int RS>
static int popc_launch(const PmParams& p, cudaStream_t st) {
    constexpr int CM = 8 / (LS == 3 ? 4 : LS);
    const int tiles = (p.M + CM - 1) / CM;
    return tiles <= 1 ? popc_launch_nt<LS, RS, 1>(p, st) : tiles <= 2 ? popc_launch_nt<LS, RS, 2>(p, st) : popc_launch_nt<LS, RS, 4>(p, st);
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
    if ((long long)N * RS * 8 >= (1LL << 31) || (long long)M * LS * 8 >= (1LL << 31) || (long long)(K / 256) * (N > M ? N : M) >= (1LL << 32))
        return SBVR_ERR_UNSUPPORTED;                // 32-bit offsets
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
