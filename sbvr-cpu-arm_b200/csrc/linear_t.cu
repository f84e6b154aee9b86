// SBVR linear on the TRANSPOSED ("row-dequant") weight encoding: the weight was encoded as W^T, so a packed word
// holds 32 consecutive OUTPUT columns n of one input k and the groups of G run along n:
//
//     bvr_t  uint32 [N/32, K, S]      bit (n % 32) of word (n / 32, k, s) = plane s of element (k, n)
//     idx_t  u8|u16 [N/G, K]          codebook line of (group of G outputs, k)
//     y[m, n] = fp16( bias[n] + sum_k x[m, k] * sum_s c[idx_t[n / G, k]][s] * bit_s[n, k] )
//
// Replaces cuda_row_deq_mm_T / cuda_row_deq_wo_shfl_mm_T / cuda_1xtN_rd_WP8_TBW4_NS4 (reference
// sbvr/kernels/sbvr_kernel.cu:121-191, :193-254, :284-359; launcher :876-912, binding sbvr/kernels/sbvr_ops.cpp:79-120).
//
// Within a group of outputs the coefficients belong to the input, so the product is one of bits with the vector
// z[m][(k, s)] = x[m, k] * c[k][s] (exact in fp32): y[m, n] = sum over (k, s) of z * bit.  It runs on the 8-bit integer tensor
// path, mma.sync m16n8k32:
//   A  sixteen outputs.  Four contraction entries (for S = 4 the planes of one k, for S = 2 those of two) are four words; a 4 x 4
//      byte transpose puts byte b of the four words into one register P_b, and `P_b & (0x01010101 << i)` is the A register of
//      output 8 b + i: four bytes, each zero or 2^i.  The factor belongs to the row of D and is taken out at the end
//      (i = 7 is the sign: -2^7).  Lane (g, t) of a warp needs the outputs 8 b + g, so the mask is a constant of the lane.
//   B  z as 31-bit fixed point with a power-of-two step per (row m, part of K), cut into four signed bytes: four columns per
//      activation row, made once per CTA in shared memory.  For a largest |z| of 1.f * 2^e in the part the step is 2^(e - 29),
//      every z is off by at most 2^(e - 30): as good as fp32 products, also where one input is far above the others (with three
//      bytes, 2^(e - 22), outputs without a plane bit at an activation 2^13 above the rest were off by 2.7e-3).
//   D  exact 32-bit sums over the whole part (at most 2 048 k).
// A part of K with a product that is not finite is multiplied out instead (lt_multiply_out).
// A warp takes a word row (32 outputs) and streams it 32 entries of 16 bytes at a time, four such loads ahead, through a small
// buffer of its own in shared memory (every load instruction is 512 contiguous bytes; lanes of a quad column read the same
// entry back).  K is split over CTAs while less than two per SM exist, and so that two fit an SM; the parts are added in part order
// by the CTA that arrives last at the word rows' counter, so results do not depend on timing.
// Measured (S = 4, us; the CUDA-core kernel below in brackets): 14336 x 4096: M = 1 17.7 (21.1), M = 4 25 (70), M = 8 41 (128);
// 4096 x 4096: M = 2 10.9 (16.9), M = 8 23.7 (53.5).  With three bytes M = 8 took 35 and 21.4.  Bound by instruction issue (35 per
// warp for 32 outputs x 8 units, one column tile) and, on small weights, by the chain of line number, line, digits in front of the
// loop: those run on CUDA cores (lt_on_cuda_cores).
#include "common.cuh"

namespace sbvr {

constexpr int LT_WARPS = 8;
constexpr int LT_THREADS = LT_WARPS * 32;
constexpr int LT_ROWS = 8;                        // activation rows per launch: four tiles of eight columns
constexpr int LT_PT = 8;                          // k per thread while the digits are made
constexpr int LT_MAX_KC = LT_PT * LT_THREADS;
constexpr int LT_PRE = 4;                         // loads ahead

struct LtParams {
    const __half* x;          // [M, K]
    const uint32_t* bvr;      // [N/32, K, S]
    const void* idx;          // [N/G, K]
    const __half* coeff;      // [C, S]
    const __half* bias;       // [N] or NULL
    __half* y;                // [M, N]
    float* part;              // [KS, rows, outputs of the launch] partial sums (KS > 1)
    unsigned int* counters;   // [N/32/nw], zero between launches (KS > 1)
    int rows;                 // activation rows of this launch
    int N, K, g32, kchunk, KS, idx_bytes;
    int cta0, ctas;           // this launch's range of word-row blocks
    int nw;                   // word rows of a CTA (1, 2, 4, 8: all of one group); its other warps split the part of K
    int one;                  // the call has one activation row
};

// Contraction entries of one 16-byte unit: the planes of one k (S = 3: and a zero), or of two for S = 2
template <int S>
__device__ __forceinline__ uint4 lt_load(const uint32_t* row, int k, int k1) {
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (k >= k1) return v;
    const uint32_t* p = row + (size_t)k * S;
    if constexpr (S == 4) {
        v = __ldcs(reinterpret_cast<const uint4*>(p));
    } else if constexpr (S == 2) {
        const uint2 a = __ldcs(reinterpret_cast<const uint2*>(p));
        v.x = a.x, v.y = a.y;
        if (k + 1 < k1) {
            const uint2 b = __ldcs(reinterpret_cast<const uint2*>(p + 2));
            v.z = b.x, v.w = b.y;
        }
    } else {
        v.x = __ldcs(p), v.y = __ldcs(p + 1), v.z = __ldcs(p + 2);
    }
    return v;
}

__device__ __forceinline__ void lt_mma(int (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ float lt_max(float a, float b) { return (a > b || a != a) ? a : b; }      // a NaN wins

// The part's sum of output `bit` of word row `row` as the CUDA-core kernel forms it: one activation row, the products of the planes that
// are set; several, products with the element's value.
template <int S>
static __device__ __noinline__ float lt_multiply_out(const LtParams& p, int m, int row, int bit, int k0, int k1) {
    float acc = 0.0f;
    for (int k = k0; k < k1; ++k) {
        const size_t i = (size_t)(row / p.g32) * p.K + k;
        const uint32_t line = (p.idx_bytes == 1) ? (uint32_t)reinterpret_cast<const uint8_t*>(p.idx)[i]
                                                 : (uint32_t)reinterpret_cast<const uint16_t*>(p.idx)[i];
        const float x = __half2float(p.x[(size_t)m * p.K + k]);
        float w = 0.0f;
        for (int s = 0; s < S; ++s) {
            if (!((p.bvr[((size_t)row * p.K + k) * S + s] >> bit) & 1u)) continue;
            const float c = __half2float(p.coeff[(size_t)line * S + s]);
            if (p.one) acc += x * c;
            else w += c;
        }
        if (!p.one) acc = fmaf(x, w, acc);
    }
    return acc;
}

template <int S, int NT>
__global__ void __launch_bounds__(LT_THREADS, 2) linear_t_kernel(const __grid_constant__ LtParams p) {
    constexpr int KU = S == 2 ? 2 : 1;             // k per unit
    constexpr int NC = 8 * NT, MR = NC / 4;        // columns, activation rows: four columns per row
    extern __shared__ __align__(16) unsigned char lt_smem[];
    __shared__ __align__(16) uint4 stage[LT_WARPS][2][32];
    __shared__ float wmax[LT_WARPS][LT_ROWS];
    __shared__ float step_s[LT_ROWS];
    __shared__ unsigned int last_s;
    pdl_launch_dependents();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int K = p.K, N = p.N, rows = p.rows, nw = p.nw, cx = p.cta0 + (int)blockIdx.x;
    const int k0 = (int)blockIdx.y * p.kchunk, k1 = min(K, k0 + p.kchunk);
    const int nu = (k1 - k0 + KU - 1) / KU, blocks = (nu + 31) / 32;        // units, blocks of 32 units
    const int sl = warp / nw, nsl = LT_WARPS / nw;
    const int b0 = blocks * sl / nsl, b1 = blocks * (sl + 1) / nsl;         // this warp's blocks
    const uint32_t* wrow = p.bvr + (size_t)(cx * nw + warp % nw) * K * S;
    uint32_t* Bs = reinterpret_cast<uint32_t*>(lt_smem);                    // [step of 8 units][NT][32 lanes][2]

    uint4 pre[LT_PRE];                             // the weight does not depend on the previous kernel
#pragma unroll
    for (int i = 0; i < LT_PRE; ++i)
        pre[i] = (b0 + i < b1) ? lt_load<S>(wrow, k0 + ((b0 + i) * 32 + lane) * KU, k1) : make_uint4(0u, 0u, 0u, 0u);

    // ---- z of this CTA's part of K -> digits
    // Every load of a kind is issued before any is used: line numbers, lines, activations.
    const size_t irow = (size_t)(cx * nw / p.g32) * K;
    uint32_t ci[LT_PT];
#pragma unroll
    for (int i = 0; i < LT_PT; ++i) {
        const int k = k0 + i * LT_THREADS + (int)threadIdx.x;
        ci[i] = 0u;
        if (k < k1)
            ci[i] = (p.idx_bytes == 1) ? (uint32_t)__ldg(reinterpret_cast<const uint8_t*>(p.idx) + irow + k)
                                       : (uint32_t)__ldg(reinterpret_cast<const uint16_t*>(p.idx) + irow + k);
    }
    __half cf[LT_PT][S];
#pragma unroll
    for (int i = 0; i < LT_PT; ++i) {
        const __half* src = p.coeff + (size_t)ci[i] * S;
        if (k0 + i * LT_THREADS < k1) {
            if constexpr (S == 4) *reinterpret_cast<uint2*>(cf[i]) = __ldg(reinterpret_cast<const uint2*>(src));
            else if constexpr (S == 2) *reinterpret_cast<uint32_t*>(cf[i]) = __ldg(reinterpret_cast<const uint32_t*>(src));
            else {
#pragma unroll
                for (int s = 0; s < S; ++s) cf[i][s] = __ldg(src + s);
            }
        }
    }
    for (int i = threadIdx.x; i < blocks * 4 * NT * 64; i += LT_THREADS) Bs[i] = 0u;
    pdl_wait();                                    // the activations may come from the previous kernel on the stream
    __half xv[LT_PT][MR];
    float mx[MR];
#pragma unroll
    for (int m = 0; m < MR; ++m) mx[m] = 0.0f;
#pragma unroll
    for (int i = 0; i < LT_PT; ++i) {
        const int k = k0 + i * LT_THREADS + (int)threadIdx.x;
#pragma unroll
        for (int m = 0; m < MR; ++m) xv[i][m] = (k < k1 && m < rows) ? p.x[(size_t)m * K + k] : __half(0.0f);
    }
#pragma unroll
    for (int i = 0; i < LT_PT; ++i) {
        if (k0 + i * LT_THREADS >= k1) break;
        float cm = 0.0f;
#pragma unroll
        for (int s = 0; s < S; ++s) cm = lt_max(fabsf(__half2float(cf[i][s])), cm);
#pragma unroll
        for (int m = 0; m < MR; ++m) mx[m] = lt_max(fabsf(__half2float(xv[i][m])) * cm, mx[m]);
    }
#pragma unroll
    for (int m = 0; m < MR; ++m) {
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            mx[m] = lt_max(__shfl_xor_sync(0xffffffffu, mx[m], o), mx[m]);
        }
        if (lane == 0) wmax[warp][m] = mx[m];
    }
    __syncthreads();
    if (threadIdx.x < MR) {
        float v = wmax[0][threadIdx.x];
#pragma unroll
        for (int w = 1; w < LT_WARPS; ++w) v = lt_max(wmax[w][threadIdx.x], v);
        // step 2^(e - 29) for a largest value of 1.f * 2^e: |q| < 2^30
        float st = 0.0f;
        if (!(v < INFINITY)) st = __int_as_float(0x7fc00000);               // the row is multiplied out
        else if (v > 0.0f) st = ldexpf(1.0f, ilogbf(v) - 29);
        step_s[threadIdx.x] = st;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < LT_PT; ++i) {
        const int k = k0 + i * LT_THREADS + (int)threadIdx.x;
        if (k0 + i * LT_THREADS >= k1) break;
        if (k < k1) {
            const int u = (k - k0) / KU, half = (u >> 2) & 1, sh = (k - k0) % KU;
            uint32_t* dst = Bs + ((size_t)(u >> 3) * NT * 32 + (u & 3)) * 2 + half;
#pragma unroll
            for (int m = 0; m < MR; ++m) {
                if (m >= rows) break;
                const float st = step_s[m];
                // the step is a power of two of at least 2^-77; a step of zero or NaN makes zeros
                const float xi = (st > 0.0f) ? __half2float(xv[i][m]) * __uint_as_float(0x7F000000u - __float_as_uint(st)) : 0.0f;
                uint32_t d[4] = {0u, 0u, 0u, 0u};
#pragma unroll
                for (int s = 0; s < S; ++s) {
                    const uint32_t q = ((uint32_t)__float2int_rn(xi * __half2float(cf[i][s])) + 0x80808080u) ^ 0x80808080u;
#pragma unroll
                    for (int e = 0; e < 4; ++e) d[e] |= ((q >> (8 * e)) & 0xFFu) << (8 * s);
                }
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int col = m * 4 + e;
                    uint32_t* w = dst + ((col >> 3) * 32 + (col & 7) * 4) * 2;
                    if (KU == 1) *w = d[e];
                    else reinterpret_cast<uint16_t*>(w)[sh] = (uint16_t)d[e];
                }
            }
        }
    }
    __syncthreads();

    // ---- the product
    int d[2][NT][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) d[i][j][e] = 0;
    const uint32_t mask = 0x01010101u << g;
    auto block = [&](int b, uint4& v) {
        uint4* sb = stage[warp][b & 1];
        {                                          // 4 x 4 byte transpose, once per unit: byte b of the four words -> word b
            const uint32_t t0 = __byte_perm(v.x, v.y, 0x5140), t1 = __byte_perm(v.z, v.w, 0x5140);
            const uint32_t t2 = __byte_perm(v.x, v.y, 0x7362), t3 = __byte_perm(v.z, v.w, 0x7362);
            sb[lane] = make_uint4(__byte_perm(t0, t1, 0x5410), __byte_perm(t0, t1, 0x7632), __byte_perm(t2, t3, 0x5410),
                                  __byte_perm(t2, t3, 0x7632));
        }
        if (b + LT_PRE < b1) v = lt_load<S>(wrow, k0 + ((b + LT_PRE) * 32 + lane) * KU, k1);
        __syncwarp();
        const uint2* bb = reinterpret_cast<const uint2*>(Bs) + (size_t)b * 4 * NT * 32 + lane;
#pragma unroll
        for (int q = 0; q < 4; ++q) {              // eight units: t and t + 4 are this lane's
            uint32_t a[2][4];                      // [half][byte of the word row]
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint4 w = sb[q * 8 + h * 4 + t];
                a[h][0] = w.x & mask, a[h][1] = w.y & mask, a[h][2] = w.z & mask, a[h][3] = w.w & mask;
            }
#pragma unroll
            for (int j = 0; j < NT; ++j) {
                const uint2 z = bb[(q * NT + j) * 32];
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const uint32_t af[4] = {a[0][2 * i], a[0][2 * i + 1], a[1][2 * i], a[1][2 * i + 1]};
                    lt_mma(d[i][j], af, z.x, z.y);
                }
            }
        }
    };
#pragma unroll 1
    for (int b = b0; b < b1; b += LT_PRE) {
#pragma unroll
        for (int i = 0; i < LT_PRE; ++i)
            if (b + i < b1) block(b + i, pre[i]);
    }
    __syncthreads();                               // everyone is done with the digits: the sums take their place
    float* res = reinterpret_cast<float*>(lt_smem);                          // [LT_WARPS][32][NC]
    const float unit = (g < 7) ? __int_as_float((127 - g) << 23) : -1.0f / 128;
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e)
                res[(warp * 32 + i * 16 + (e >> 1) * 8 + g) * NC + j * 8 + 2 * t + (e & 1)] = (float)d[i][j][e] * unit;
    __syncthreads();
    const size_t pn = (size_t)p.ctas * nw * 32;    // outputs of this launch
    const int outs = nw * 32 * rows, n0 = cx * nw * 32;
    auto store = [&](int m, int n, float v) { p.y[(size_t)m * N + n] = __float2half_rn(v + (p.bias ? __half2float(p.bias[n]) : 0.0f)); };
    for (int e = threadIdx.x; e < outs; e += LT_THREADS) {
        const int nl = e % (nw * 32), m = e / (nw * 32);
        float v = 0.0f;
        for (int s = 0; s < nsl; ++s) {
            const float* r = res + ((size_t)(s * nw + nl / 32) * 32 + nl % 32) * NC + m * 4;
            v += fmaf(r[3], 16777216.0f, fmaf(r[2], 65536.0f, fmaf(r[1], 256.0f, r[0])));
        }
        const float st = step_s[m];
        v = (st == st) ? v * st : lt_multiply_out<S>(p, m, cx * nw + nl / 32, nl % 32, k0, k1);
        if (p.KS == 1) store(m, n0 + nl, v);
        else __stcg(p.part + ((size_t)blockIdx.y * rows + m) * pn + (int)blockIdx.x * nw * 32 + nl, v);
    }
    if (p.KS == 1) return;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last_s = (atomicAdd(p.counters + blockIdx.x, 1u) == (unsigned int)(p.KS - 1)) ? 1u : 0u;
    __syncthreads();
    if (!last_s) return;
    __threadfence();
    // Eight parts in flight per thread and, for three rows and more, of four results: one result at a time was a chain of
    // rows * KS / 8 round trips to L2 (8 rows of 1024 x 14336: 41.7 -> 28.3 us; one row is faster without).
    constexpr int U = NT == 1 ? 1 : 4;
    for (int e0 = threadIdx.x; e0 < outs; e0 += U * LT_THREADS) {
        const float* src[U];
        float v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int e = min(e0 + u * LT_THREADS, outs - 1);
            src[u] = p.part + (e / (nw * 32)) * pn + (int)blockIdx.x * nw * 32 + e % (nw * 32);
            v[u] = 0.0f;
        }
        for (int q = 0; q < p.KS; q += 8) {
            float tq[U][8];
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    tq[u][i] = (q + i < p.KS && e0 + u * LT_THREADS < outs) ? __ldcg(src[u] + (size_t)(q + i) * rows * pn) : 0.0f;
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int i = 0; i < 8; ++i) v[u] += tq[u][i];
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int e = e0 + u * LT_THREADS;
            if (e < outs) store(e / (nw * 32), n0 + e % (nw * 32), v[u]);
        }
    }
    if (threadIdx.x == 0) p.counters[blockIdx.x] = 0u;      // ready for the next launch
}

template <int S, int NT>
static int lt_launch_nt(const LtParams& p, cudaStream_t st) {
    constexpr int KU = S == 2 ? 2 : 1;
    const int blocks = ((p.kchunk + KU - 1) / KU + 31) / 32;
    int smem = blocks * 4 * NT * 256;
    const int res = LT_WARPS * 32 * 8 * NT * 4;
    if (smem < res) smem = res;
    static SmemOnce once;
    const int rc = set_max_smem_once(once, linear_t_kernel<S, NT>, 200 * 1024);
    if (rc) return rc;
    SBVR_CUDA_TRY(launch_pdl(linear_t_kernel<S, NT>, dim3(p.ctas, p.KS), dim3(LT_THREADS), (size_t)smem, st, p));
    return SBVR_OK;
}
template <int S>
static int lt_launch(const LtParams& p, cudaStream_t st) {
    switch ((p.rows + 1) / 2) {
        case 1: return lt_launch_nt<S, 1>(p, st);
        case 2: return lt_launch_nt<S, 2>(p, st);
        case 3: return lt_launch_nt<S, 3>(p, st);
        default: return lt_launch_nt<S, 4>(p, st);
    }
}

// ---------------------------------------------------------------------------------------------
// Small problems, on CUDA cores: fp32 products and sums.
//
// A THREAD owns one k at a time and all 32 outputs of the word: the lanes of a warp read 32 consecutive k of one word row (S * 128
// contiguous bytes, one 16-byte load per lane for S = 4), the line number of (group, k) and the activation, and add x * c_s to the
// accumulators whose bit is set: one predicated add per plane bit, no shifts (with several activation rows the element is formed
// once and costs one FMA per row).  32 fp32 accumulators per activation row live in registers; at the end a butterfly
// reduce-scatter over the lanes leaves the sum of output n = lane in each lane, the warps of the block are added in order through
// shared memory.  A block covers one word row and a part of K; partial sums go to the workspace and the block that arrives
// last at the word row's counter adds them in part order.
// ---------------------------------------------------------------------------------------------
constexpr int LC_THREADS = 256;
constexpr int LC_WARPS = LC_THREADS / 32;

struct LcParams {
    const __half* x;          // [M, K]
    const uint32_t* bvr;      // [N/32, K, S]
    const void* idx;          // [N/G, K]
    const __half* coeff;      // [C, S]
    const __half* bias;       // [N] or NULL
    __half* y;                // [M, N]
    float* part;              // [KS, MT, N] partial sums (KS > 1)
    unsigned int* counters;   // [N/32], zero between launches (KS > 1)
    int rows;                 // activation rows of this launch (<= MT)
    int N, K, g32, kchunk, KS;
};

template <int S>
__device__ __forceinline__ void lc_load_words(const uint32_t* p, uint32_t (&w)[S]) {
    if constexpr (S == 4) {
        const uint4 v = __ldg(reinterpret_cast<const uint4*>(p));
        w[0] = v.x, w[1] = v.y, w[2] = v.z, w[3] = v.w;
    } else if constexpr (S == 2) {
        const uint2 v = __ldg(reinterpret_cast<const uint2*>(p));
        w[0] = v.x, w[1] = v.y;
    } else {
#pragma unroll
        for (int s = 0; s < S; ++s) w[s] = __ldg(p + s);
    }
}

template <int S>
__device__ __forceinline__ void lc_load_coef(const __half* line, float (&c)[S]) {
    if constexpr (S == 4) {
        const uint2 v = __ldg(reinterpret_cast<const uint2*>(line));
        const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&v.x));
        const float2 b = __half22float2(*reinterpret_cast<const __half2*>(&v.y));
        c[0] = a.x, c[1] = a.y, c[2] = b.x, c[3] = b.y;
    } else if constexpr (S == 2) {
        const uint32_t v = __ldg(reinterpret_cast<const uint32_t*>(line));
        const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&v));
        c[0] = a.x, c[1] = a.y;
    } else {
#pragma unroll
        for (int s = 0; s < S; ++s) c[s] = __half2float(__ldg(line + s));
    }
}

template <int S, int MT, int IDXB>
__global__ void __launch_bounds__(LC_THREADS) linear_tc_kernel(const LcParams p) {
    __shared__ float red[LC_WARPS][MT][32];
    pdl_launch_dependents();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nw = blockIdx.x, ks = blockIdx.y;
    const int K = p.K;
    const int k0 = ks * p.kchunk, k1 = min(K, k0 + p.kchunk);
    const uint32_t* wrow = p.bvr + (size_t)nw * K * S;
    const size_t irow = (size_t)(nw / p.g32) * K;

    float acc[MT][32];
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int n = 0; n < 32; ++n) acc[m][n] = 0.0f;

    // what one k needs; the next k's loads are issued before the current one is used
    uint32_t w[S], wn[S];
    uint32_t ci = 0, cin = 0;
    auto load_idx = [&](int k) -> uint32_t {
        return (IDXB == 1) ? (uint32_t)__ldg(reinterpret_cast<const uint8_t*>(p.idx) + irow + k)
                           : (uint32_t)__ldg(reinterpret_cast<const uint16_t*>(p.idx) + irow + k);
    };
    int k = k0 + (int)threadIdx.x;
    if (k < k1) {                                  // weights and indices do not depend on the previous kernel
        lc_load_words<S>(wrow + (size_t)k * S, w);
        ci = load_idx(k);
    }
    pdl_wait();                                    // the activations may come from the previous kernel on the stream
    for (; k < k1; k += LC_THREADS) {
        const int kn = k + LC_THREADS;
        if (kn < k1) {
            lc_load_words<S>(wrow + (size_t)kn * S, wn);
            cin = load_idx(kn);
        }
        float c[S];
        lc_load_coef<S>(p.coeff + (size_t)ci * S, c);
        float xv[MT];
#pragma unroll
        for (int m = 0; m < MT; ++m) xv[m] = __half2float(p.x[(size_t)min(m, p.rows - 1) * K + k]);
        if constexpr (MT == 1) {                   // one row: add x * c_s where the bit is set, S predicated adds per output
#pragma unroll
            for (int s = 0; s < S; ++s) {
                const float xc = xv[0] * c[s];
#pragma unroll
                for (int n = 0; n < 32; ++n)
                    if (w[s] & (1u << n)) acc[0][n] += xc;
            }
        } else {                                   // several rows: dequantise the element once, one FMA per row
#pragma unroll
            for (int n = 0; n < 32; ++n) {
                float wv = 0.0f;
#pragma unroll
                for (int s = 0; s < S; ++s)
                    if (w[s] & (1u << n)) wv += c[s];
#pragma unroll
                for (int m = 0; m < MT; ++m) acc[m][n] = fmaf(xv[m], wv, acc[m][n]);
            }
        }
#pragma unroll
        for (int s = 0; s < S; ++s) w[s] = wn[s];
        ci = cin;
    }

    // lanes -> outputs: after the step with offset o a lane keeps the accumulators whose bit o of n equals its own
#pragma unroll
    for (int m = 0; m < MT; ++m) {
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1) {
            const bool up = (lane & o) != 0;
#pragma unroll
            for (int i = 0; i < o; ++i) {
                const float keep = up ? acc[m][i + o] : acc[m][i];
                const float send = up ? acc[m][i] : acc[m][i + o];
                acc[m][i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
            }
        }
        red[warp][m][lane] = acc[m][0];            // output n = nw * 32 + lane
    }
    __syncthreads();
    if (warp != 0) return;
    const int n = nw * 32 + lane;
    const float b = p.bias ? __half2float(p.bias[n]) : 0.0f;
    float v[MT];
#pragma unroll
    for (int m = 0; m < MT; ++m) {
        v[m] = 0.0f;
#pragma unroll
        for (int wi = 0; wi < LC_WARPS; ++wi) v[m] += red[wi][m][lane];
    }
    if (p.KS == 1) {
#pragma unroll
        for (int m = 0; m < MT; ++m)
            if (m < p.rows) p.y[(size_t)m * p.N + n] = __float2half_rn(v[m] + b);
        return;
    }
#pragma unroll
    for (int m = 0; m < MT; ++m) p.part[((size_t)ks * MT + m) * p.N + n] = v[m];
    __threadfence();
    __syncwarp();
    unsigned int last = 0;
    if (lane == 0) last = (atomicAdd(p.counters + nw, 1u) == (unsigned int)(p.KS - 1)) ? 1u : 0u;
    last = __shfl_sync(0xffffffffu, last, 0);
    if (!last) return;
    __threadfence();
#pragma unroll
    for (int m = 0; m < MT; ++m) {
        if (m >= p.rows) break;
        float t = 0.0f;
        for (int q = 0; q < p.KS; ++q) t += __ldcg(p.part + ((size_t)q * MT + m) * p.N + n);
        p.y[(size_t)m * p.N + n] = __float2half_rn(t + b);
    }
    if (lane == 0) p.counters[nw] = 0u;            // ready for the next launch
}

template <int S, int MT>
static int lc_launch_idx(const LcParams& p, int idxb, dim3 grid, cudaStream_t st) {
    if (idxb == 1)
        SBVR_CUDA_TRY(launch_pdl(linear_tc_kernel<S, MT, 1>, grid, dim3(LC_THREADS), 0, st, p));
    else
        SBVR_CUDA_TRY(launch_pdl(linear_tc_kernel<S, MT, 2>, grid, dim3(LC_THREADS), 0, st, p));
    return SBVR_OK;
}
template <int S>
static int lc_launch_m(const LcParams& p, int mt, int idxb, dim3 grid, cudaStream_t st) {
    switch (mt) {
        case 1: return lc_launch_idx<S, 1>(p, idxb, grid, st);
        case 2: return lc_launch_idx<S, 2>(p, idxb, grid, st);
        default: return lc_launch_idx<S, 4>(p, idxb, grid, st);
    }
}


static int launch_linear_tc(const LtParams& q, int M, int S, int sm_count, size_t dyn_bytes, cudaStream_t st) {
    const int nwords = q.N / 32, K = q.K;
    // K is split over blocks while at most four blocks per SM exist (one resident wave at 64 registers per thread); parts are
    // multiples of the block's 256 k
    const int mt_all = M >= 3 ? 4 : M;            // rows per launch as instantiated: 1, 2 or 4
    int KS = 4 * sm_count / nwords;                // rounded down: all blocks resident at once
    if (KS < 1) KS = 1;
    int kchunk = ((K + KS - 1) / KS + LC_THREADS - 1) / LC_THREADS * LC_THREADS;
    if (kchunk < 2 * LC_THREADS) kchunk = 2 * LC_THREADS;
    KS = (K + kchunk - 1) / kchunk;
    if (KS > 1 && (nwords > SBVR_WS_COUNTERS || (size_t)KS * mt_all * q.N * sizeof(float) > dyn_bytes)) KS = 1, kchunk = K;
    LcParams p;
    p.bvr = q.bvr, p.idx = q.idx, p.coeff = q.coeff, p.bias = q.bias, p.part = q.part, p.counters = q.counters;
    p.N = q.N, p.K = K, p.g32 = q.g32, p.kchunk = kchunk, p.KS = KS;
    const dim3 grid(nwords, KS);
    for (int m0 = 0; m0 < M; m0 += 4) {
        p.rows = (M - m0 < 4) ? M - m0 : 4;
        p.x = q.x + (size_t)m0 * K, p.y = q.y + (size_t)m0 * q.N;
        const int mt = p.rows >= 3 ? 4 : p.rows;
        int r;
        switch (S) {
            case 2: r = lc_launch_m<2>(p, mt, q.idx_bytes, grid, st); break;
            case 3: r = lc_launch_m<3>(p, mt, q.idx_bytes, grid, st); break;
            default: r = lc_launch_m<4>(p, mt, q.idx_bytes, grid, st); break;
        }
        if (r) return r;
    }
    return SBVR_OK;
}

// Where that is faster than the digits, whose preparation costs more than the sums there.  Both sides measured (S = 4, us, digits in
// brackets): 256 x 4096 M = 1 4.9 (6.6), M = 16 27.7 (36.2); 1024 x 4096 M = 1 6.4 (7.7), M = 2 7.1 (9.9), M = 4 11.9 (13.4), but M = 6
// 18.6 (17.2); 2048 x 4096 M = 1 6.6 (7.9), but M = 2 11.5 (10.7); 4096 x 4096 M = 1 9.15 (9.25); 1024 x 14336 M = 1 9.7 (10.0), but
// M = 2 17.7 (13.3).
static bool lt_on_cuda_cores(int M, int N, int K) {
    const long long elements = (long long)N * K;
    return elements * M <= (1LL << 24) && (M == 1 || elements <= (1LL << 22));
}

}  // namespace sbvr

using namespace sbvr;

extern "C" int sbvr_linear_t_f16(const void* x, const uint32_t* bvr_t, const void* coeff_idx, int idx_bytes,
                                  const void* coeff, int C, const void* bias, void* y, int M, int N, int K, int S, int G,
                                  sbvr_workspace_t* ws, sbvr_stream_t stream) {
    if (!x || !bvr_t || !coeff_idx || !coeff || !y || !ws) return SBVR_ERR_BAD_ARG;
    if (M < 1 || N < 1 || K < 1 || C < 1 || C > 65536) return SBVR_ERR_BAD_ARG;
    if ((idx_bytes != 1 && idx_bytes != 2) || (idx_bytes == 1 && C > 256)) return SBVR_ERR_BAD_ARG;
    if (S < 2 || S > 4) return SBVR_ERR_UNSUPPORTED;
    if (G < 32 || G % 32 || N % G) return SBVR_ERR_SHAPE;
    const uintptr_t walign = (S == 4) ? 15 : (S == 2) ? 7 : 3;
    const uintptr_t calign = (S == 4) ? 7 : (S == 2) ? 3 : 1;
    if ((reinterpret_cast<uintptr_t>(bvr_t) & walign) || (reinterpret_cast<uintptr_t>(coeff) & calign) ||
        (reinterpret_cast<uintptr_t>(x) & 1) || (reinterpret_cast<uintptr_t>(y) & 1) ||
        (idx_bytes == 2 && (reinterpret_cast<uintptr_t>(coeff_idx) & 1)))
        return SBVR_ERR_ALIGN;
    DeviceInfo di;
    const int rc = device_info(ws->device, &di);
    if (rc) return rc;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    WsLock lock(ws);
    LtParams p;
    p.bvr = bvr_t, p.idx = coeff_idx, p.coeff = reinterpret_cast<const __half*>(coeff), p.idx_bytes = idx_bytes;
    p.bias = reinterpret_cast<const __half*>(bias);
    p.counters = ws->counters;
    p.N = N, p.K = K, p.g32 = G / 32;
    p.one = M == 1;
    p.x = reinterpret_cast<const __half*>(x), p.y = reinterpret_cast<__half*>(y), p.part = reinterpret_cast<float*>(ws->dyn);
    if (lt_on_cuda_cores(M, N, K)) return launch_linear_tc(p, M, S, di.sm_count, ws->dyn_bytes, st);
    p.nw = p.g32 % 8 == 0 ? 8 : p.g32 % 4 == 0 ? 4 : p.g32 % 2 == 0 ? 2 : 1;
    const int gx = N / 32 / p.nw;
    for (int m0 = 0; m0 < M; m0 += LT_ROWS) {
        p.rows = (M - m0 < LT_ROWS) ? M - m0 : LT_ROWS;
        // Parts of K: as many as give every SM the two CTAs its registers hold, in steps of a block for every warp that shares a
        // word row; at most LT_MAX_KC long, and so short that the digits of two CTAs (1 KB per 32 units and tile) fit its shared memory.
        const int quantum = (S == 2 ? 64 : 32) * (LT_WARPS / p.nw);
        int KS = 2 * di.sm_count / gx;
        if (KS > 64) KS = 64;
        if (KS < 1) KS = 1;
        int kchunk = ((K + KS - 1) / KS + quantum - 1) / quantum * quantum;
        const int least = p.rows == 2 ? 256 : 128;      // two rows: fewer parts to add (10.2 -> 9.4 us at 1024 x 4096)
        if (kchunk < least) kchunk = (least + quantum - 1) / quantum * quantum;
        const int fit = 104 / ((p.rows + 1) / 2) * (S == 2 ? 64 : 32);
        const int cap = (fit < LT_MAX_KC ? fit : LT_MAX_KC) / quantum * quantum;
        if (kchunk > cap) kchunk = cap;
        KS = (K + kchunk - 1) / kchunk;
        p.kchunk = kchunk, p.KS = KS;
        p.x = reinterpret_cast<const __half*>(x) + (size_t)m0 * K;
        p.y = reinterpret_cast<__half*>(y) + (size_t)m0 * N;
        // as many word rows per launch as there is room for the parts and counters of (all of them but on enormous layers)
        int most = gx;
        if (KS > 1) {
            const size_t fit = ws->dyn_bytes / ((size_t)KS * p.rows * p.nw * 32 * sizeof(float));
            if (fit < 1) return SBVR_ERR_WORKSPACE;
            if ((size_t)most > fit) most = (int)fit;
            if (most > SBVR_WS_COUNTERS) most = SBVR_WS_COUNTERS;
        }
        for (p.cta0 = 0; p.cta0 < gx; p.cta0 += most) {
            p.ctas = gx - p.cta0 < most ? gx - p.cta0 : most;
            int r;
            switch (S) {
                case 2: r = lt_launch<2>(p, st); break;
                case 3: r = lt_launch<3>(p, st); break;
                default: r = lt_launch<4>(p, st); break;
            }
            if (r) return r;
        }
    }
    return SBVR_OK;
}
