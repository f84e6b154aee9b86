// SBVR linear for small activation batches (2 .. 16 rows): FP4 tensor-core dot products of plane bits with activation digits,
// like the decode GEMV, but with the digits' weights and the activations' block step carried by the MMA's own block scale
// factors, so that the tensor pipe sums over digits and nothing but one multiply-add per (row, plane, digit half, activation
// row, 256-k block) is left for the CUDA cores.
//
//   y[m, n] = sum_g sum_s c[g, n, s] * sum_{k in g} x[m, k] * bit_s[n, k]
//
// Operands of tcgen05.mma kind::mxf4.block_scale.scale_vec::2X (K = 64 per instruction, fp32 accumulation in tensor memory):
//
//  A (tensor memory)  128 lanes = TN output rows x their planes; a lane's 256 plane bits of a k block are expanded to 4-bit
//      E2M1 codes by six integer instructions per packed word (`(w << 1) & 0x2222.., w & 0x2222.., w & 0x4444..,
//      (w >> 1) & 0x4444..`): a set bit becomes 1, 1, 2, 2 for k % 4 = 0 .. 3.
//  B (shared memory)  x is quantised per (activation row, 256-k block) to block fixed point in two levels: q = round(x / step)
//      with the power of two step = 2^(e - 15) for a largest value of 1.f * 2^e, and what that rounding left over with step 2^-17.
//      q + 0x24924 is cut into six 3-bit fields t, digit = t - 4 in {-4 .. 3}, so that q = sum_d 8^d digit_d.  Every digit
//      is an exact E2M1 value (halved where the plane bit counts 2).  One MMA multiplies the plane bits by two digits of 16
//      activation rows (N = 2 x 16), with the scale factor 8^d * step of that digit and row as the B block scale (UE8M0, a power
//      of two): the two accumulator columns of an activation row (even and odd digits, added on the way out) then hold
//      sum_k bit * x^ directly, whatever the digit and its level.
//
// Precision.  |x - x^| <= 2^(e - 33): fp16 activations keep all of their bits down to 2^-22 of their block's largest, and what is
// lost below is far less than fp32's rounding of that largest value.  The first level alone, an error of 2^(e - 15), made zeros of
// everything below 2^-15 of the largest: with one activation of 2^13 in every block, outputs whose weight there is zero were off by
// 15 % (now 2.1e-4, the rounding of the result; 3.4e-4 for the fp16 GEMM, which sees the activations as they are and rounds weights).
//
// Structure.  K is cut into chunks of at most SB_CHUNK 256-k blocks, and a CTA works on one chunk: its digits (24 KB per block,
// written by the quantiser kernel) stay in shared memory and their scale factors in tensor memory for
// the whole launch, so the only things that move are packed words.  Four warpgroups take (row tile, k block) units in order,
// each on its own, with two A buffers and one D buffer: while the MMAs of unit i run, unit i + 1 is expanded into the other
// A buffer and unit i + 2 read from shared memory; as soon as they are done the sums are read and the MMAs of unit i + 1
// released, and the multiply-adds run beside those.  (Two groups per k block take two D buffers and leave room for one A.)  A
// warp holds all sums of a quarter of a tile's rows.  A tile that several warpgroups share is put together in shared memory at the
// end.  The chunks' sums meet in scratch when the CTAs of a group (the chunks of the same tiles) are through: each adds an equal
// share of them in chunk order (the same bits on every run), or leaves it to the last of them.  Added by whichever warp arrived last at a tile's counter, as
// before, the slow CTAs of a group got nearly all of that work on top: at 28672 x 8192 they ended 27 us behind the mean of 70.
// Every wait is bounded.
//
// What bounds it: the tensor pipe in the loop (a unit takes 485 cycles of its SM at 14336 x 4096, its 24 MMAs 391 of a pipe that
// does nothing else); around it, per launch, 4.7 us from the end of the kernel in front to the digits in shared memory (of it 1 to 1.7
// in the quantiser) and 2 to 3 us for the merge.  That the merge does not count on its CTAs running together costs 0.4 us where the sums
// are few (a fence and an atomic beside the sums), nothing elsewhere.  Per call with the quantiser, M = 16, S = 4, us (with sums added by
// the last warp to arrive; the fp16 GEMM): 1024 x 4096 9.8 (11.0; 10.4), 4096 x 4096 11.4 (12.7; 14.8), 14336 x 4096 22.3 (27.8; 32.1),
// 4096 x 14336 26.9 (39.7; 31.6), 28672 x 8192 60 (104; 112); groups of 128, 14336 x 4096: 24.6 (30.0; 31.9).
//
// Replaces the M > 1 use of `_sbvr_row_deq_mm_T` (reference sbvr/kernels/sbvr_kernel.cu:121-191) for 2 .. 16 rows.
#include <cuda.h>

#include "common.cuh"
#include "tc_stream.cuh"

namespace sbvr {

constexpr int SB_NWG = 4;
constexpr int SB_CW0 = 4;                       // warps 0 .. 3: issuers (warp 0 also sets up); compute warps behind
constexpr int SB_THREADS = (SB_CW0 + 4 * SB_NWG) * 32;
constexpr int SB_MP = 16;                       // activation rows the accumulators cover
constexpr int SB_ND = 12;                       // digits of an activation
constexpr int SB_NJ = SB_ND / 2;                // MMAs per 64 k: two digits each
constexpr int SB_BLOB = SB_NJ * 4096 + 512;     // digits of a k block, then 32 rows x 16 B of scale factors (and poison marks)
constexpr int SB_ASTAGE = TS_STAGE_WORDS + 512; // packed words of a unit + its coefficient data
constexpr int SB_MAX_STAGES = 4;
constexpr int SB_HDR = 1024;
constexpr int SB_CHUNK = 4;                     // k blocks of a CTA at most (shared memory)
constexpr int SB_SFCOLS = 12;
// Tensor memory: per warpgroup A (32 columns each) and D (32 per group of a block), then the B scale factors of every k block (12
// columns each, one 4-column block per two MMAs; an MMA's scale-factor address designates a block), then unit factors for A
constexpr int SB_WGCOLS = 96;                   // A x 2 and D, or A and D x 2
constexpr int SB_SFB_COL = SB_NWG * SB_WGCOLS, SB_SFA_COL = SB_SFB_COL + 64;
static_assert(SB_CHUNK * SB_SFCOLS <= 64 && SB_SFA_COL + 32 <= TS_TMEM_COLS, "tensor memory");

struct SbParams {
    const unsigned char* xb;      // [KB][SB_BLOB] written by sb_quant_kernel
    const __half* x;              // what was quantised, [M][K]; NULL: a row with a non-finite value becomes NaN
    const uint32_t* bvr;
    const void* idx;
    const __half* coeff;
    const __half* bias;
    __half* y;
    unsigned int* status;
    unsigned long long* arrive;   // a word per group of CTAs that work on the same tiles, zero between launches (see "the chunks of K meet")
    unsigned int patience;        // SM cycles a CTA waits for its siblings before it hands its share of the sums over
    float* part;                  // [KC][NT][SB_MP][TN] sums of the chunks (KC > 1)
    int M, N, K, KB, NT, C, KC, GN, cache_in_smem, stages, idx_bytes;
    int tagged;                   // `part` lies in the exchange region, all zero between launches, and a sum's arrival is its own mark
    int off_cache, off_ring, off_res;
};

struct SbQuant {
    const __half* x;
    unsigned char* xb;
    int M, K;
    int x_op;
    const __half* delta;
    const __half* norm_w;
    __half* h_out;
    float eps;
    __half* x_out;            // the row as it is quantised, or NULL
};

// ---------------------------------------------------------------------------------------------
// activations (with the op in front of the linear) -> digit blob, once per call
// ---------------------------------------------------------------------------------------------
// One block per 256-k block and (padded) activation row; its four warps take a level and three of its digits each, so that the chain
// from the arrival of the row to the last digit is a quarter as long (the product waits for it).  With at most 32 registers a thread
// the blocks fit beside a resident CTA of the product, and both wait for their predecessors there (with blocks that did not fit, a call
// took 6 us more: the quantiser started when the product had ended).  Lane (kw, j) owns the eight elements
// k = 32 kw + j + 4 e, which are one 32-bit word (nibble e) of every digit: the K order in which the weight expansion
// leaves the plane bits.  Blob of a k block: [MMA j (SB_NJ)][row group (4)][kw (8)][row (8)][16 B], then 32 rows x 16 B:
// words 0 .. 2 hold the scale bytes of MMA 2 i (bytes 0, 1) and 2 i + 1 (bytes 2, 3) for that B row, word 3 of row m whether
// activation row m of this block holds a non-finite value.
__global__ void __launch_bounds__(128, 16) sb_quant_kernel(const SbQuant p) {
    __shared__ __align__(16) __half row[4][256];
    __shared__ float ssum[4];
    pdl_launch_dependents();
    pdl_wait();                                    // the activations come from the previous kernel of the stream
    const int wl = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int kb = blockIdx.x, K = p.K, M = p.M, m = blockIdx.y;
    const int kw = lane >> 2, j = lane & 3;
    const int level = wl >> 1, d0 = (wl & 1) * 3;
    int ex = 15;
    bool poison = false;
    float inv = 0.0f;
    if (m < M) {
        // 256 activations: lane l of every warp brings elements 8 l .. 8 l + 7
        const size_t off = (size_t)m * K + (size_t)kb * 256 + lane * 8;
        uint4 o;
        __half2* oh = reinterpret_cast<__half2*>(&o);
        if (p.x_op == SBVR_XOP_SILU_MUL) {
            const __half* gp = p.x + (size_t)m * 2 * K + (size_t)kb * 256 + lane * 8;
            const uint4 g = __ldg(reinterpret_cast<const uint4*>(gp));
            const uint4 u = __ldg(reinterpret_cast<const uint4*>(gp + K));
            const __half2* gh = reinterpret_cast<const __half2*>(&g);
            const __half2* uh = reinterpret_cast<const __half2*>(&u);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float2 f = __half22float2(gh[e]);
                oh[e] = __hmul2(__floats2half2_rn(f.x / (1.0f + expf(-f.x)), f.y / (1.0f + expf(-f.y))), uh[e]);
            }
        } else if (p.x_op == SBVR_XOP_ADD_RMSNORM) {
            // mean of (h + delta)^2 over the whole row, the sum formed in fp16 like the separate kernel does
            float sq = 0.0f;
#pragma unroll 4
            for (int c = threadIdx.x; c < K / 8; c += 128) {
                uint4 a = __ldg(reinterpret_cast<const uint4*>(p.x + (size_t)m * K) + c);
                __half2* ah = reinterpret_cast<__half2*>(&a);
                if (p.delta) {
                    const uint4 b = __ldg(reinterpret_cast<const uint4*>(p.delta + (size_t)m * K) + c);
                    const __half2* bh = reinterpret_cast<const __half2*>(&b);
#pragma unroll
                    for (int e = 0; e < 4; ++e) ah[e] = __hadd2(ah[e], bh[e]);
                }
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float2 f = __half22float2(ah[e]);
                    sq += f.x * f.x + f.y * f.y;
                }
            }
#pragma unroll
            for (int s = 16; s; s >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, s);
            if (lane == 0) ssum[wl] = sq;
            __syncthreads();
            const float rs = rsqrtf((ssum[0] + ssum[1] + ssum[2] + ssum[3]) / (float)K + p.eps);
            uint4 a = __ldg(reinterpret_cast<const uint4*>(p.x + off));
            __half2* ah = reinterpret_cast<__half2*>(&a);
            if (p.delta) {
                const uint4 b = __ldg(reinterpret_cast<const uint4*>(p.delta + off));
                const __half2* bh = reinterpret_cast<const __half2*>(&b);
#pragma unroll
                for (int e = 0; e < 4; ++e) ah[e] = __hadd2(ah[e], bh[e]);
            }
            if (p.h_out && wl == 0) *reinterpret_cast<uint4*>(p.h_out + off) = a;
            const uint4 wv = __ldg(reinterpret_cast<const uint4*>(p.norm_w + (size_t)kb * 256 + lane * 8));
            const __half2* wh = reinterpret_cast<const __half2*>(&wv);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float2 f = __half22float2(ah[e]);
                oh[e] = __hmul2(wh[e], __floats2half2_rn(f.x * rs, f.y * rs));
            }
        } else if ((reinterpret_cast<uintptr_t>(p.x) & 15) == 0) {
            o = __ldg(reinterpret_cast<const uint4*>(p.x + off));
        } else {
            __half* e = reinterpret_cast<__half*>(&o);
#pragma unroll
            for (int i = 0; i < 8; ++i) e[i] = p.x[off + i];
        }
        if (p.x_out && wl == 0) *reinterpret_cast<uint4*>(p.x_out + off) = o;
        float a = 0.0f;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float2 f = __half22float2(oh[e]);
            float av = fmaxf(fabsf(f.x), fabsf(f.y));
            if (f.x != f.x || f.y != f.y) av = __int_as_float(0x7f800000);     // NaN counts as infinity
            a = fmaxf(a, av);
        }
        reinterpret_cast<uint4*>(row[wl])[lane] = o;
#pragma unroll
        for (int s = 16; s; s >>= 1) a = fmaxf(a, __shfl_xor_sync(0xffffffffu, a, s));
        if (a >= __int_as_float(0x7f800000)) {
            poison = true;
        } else if (a > 0.0f) {
            ex = (int)((__float_as_uint(a) >> 23) & 0xFF) - 127;              // a = 1.f * 2^ex, ex in [-24, 15]
            inv = __uint_as_float((uint32_t)(15 - ex + 127) << 23);
        }
        __syncwarp();
    }
    unsigned char* blob = p.xb + (size_t)kb * SB_BLOB;
    // E2M1 codes of digit t - 4 (t = 0 .. 7), one nibble each: the value itself for j = 0, 1, half of it for j = 2, 3
    const uint32_t lut = (j < 2) ? 0x5420ACDEu : 0x32109ABCu;
    uint32_t words[3] = {0u, 0u, 0u};
    if (m < M && !poison) {
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const float f = __half2float(row[wl][32 * kw + j + 4 * e]) * inv;                  // exact
            int q = __float2int_rn(f);                                                         // |q| <= 2^16
            if (level) q = __float2int_rn((f - (float)q) * 131072.0f);                         // the difference is exact; |q| <= 2^16
            const uint32_t u = (uint32_t)(q + 0x24924) >> (3 * d0);
#pragma unroll
            for (int d = 0; d < 3; ++d) words[d] |= ((lut >> (4u * ((u >> (3 * d)) & 7u))) & 0xFu) << (4 * e);
        }
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const int dd = level * 6 + d0 + d;
        const int r = (dd & 1) * 16 + m;
        *reinterpret_cast<uint32_t*>(blob + (dd >> 1) * 4096 + (r >> 3) * 1024 + kw * 128 + (r & 7) * 16 + j * 4) = words[d];
    }
    // scale bytes 127 + exponent, each twice (two 32-element blocks per MMA); rows beyond M: 2^0 on zero digits
    auto two = [&](int d) -> uint32_t { return (m < M ? (uint32_t)(127 + 3 * (d % 6) + ex - (d < 6 ? 15 : 32)) : 127u) * 0x0101u; };
    uint4* sf = reinterpret_cast<uint4*>(blob + SB_NJ * 4096);
    if (wl == 0 && lane < 2)                       // even digits in row m, odd ones in row 16 + m; MMA j has digits 2 j, 2 j + 1
        sf[lane * 16 + m] = make_uint4(two(lane) | (two(2 + lane) << 16), two(4 + lane) | (two(6 + lane) << 16),
                                       two(8 + lane) | (two(10 + lane) << 16), poison ? 1u : 0u);
}

// ---------------------------------------------------------------------------------------------
// the product
// ---------------------------------------------------------------------------------------------
// Two fp32 values in one 64-bit register: the packed add and multiply-add issue once for both.
struct SbPair {
    unsigned long long b;
    __device__ SbPair() {}
    __device__ SbPair(uint32_t lo, uint32_t hi) { asm("mov.b64 %0, {%1, %2};" : "=l"(b) : "r"(lo), "r"(hi)); }
    __device__ SbPair(float lo, float hi) { asm("mov.b64 %0, {%1, %2};" : "=l"(b) : "f"(lo), "f"(hi)); }
    __device__ void get(float& lo, float& hi) const { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(b)); }
    __device__ SbPair operator+(const SbPair& o) const {
        SbPair r;
        asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.b) : "l"(b), "l"(o.b));
        return r;
    }
    __device__ SbPair mul_add(const SbPair& f, const SbPair& o) const {      // this * f + o
        SbPair r;
        asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.b) : "l"(b), "l"(f.b), "l"(o.b));
        return r;
    }
};

// y[m, n] of an activation row that holds something non-finite, as products give it: the digits cannot say it and have left a NaN.
// Inlined where few values are live (76 to 79 registers with groups of 256, the limit of 88 with groups of 128): as a function that is
// called it took the kernel beyond 88, which leaves no room beside a CTA for the blocks of the next call (seven linears of a
// layer, 16 rows, with the GEMM among them: 154 against 146 us).
template <int S>
__device__ __forceinline__ void sb_multiply_out(const SbParams& p, int G, int m, int n) {
    float acc = 0.0f;
#pragma unroll 1
    for (int k = 0; k < p.K; ++k) {
        const __half* line = coeff_line(p.idx, p.idx_bytes, p.coeff, k / G, n, p.N, S);
        const uint32_t* words = p.bvr + ((size_t)(k >> 5) * p.N + n) * S;
        float w = 0.0f;
#pragma unroll 1
        for (int s = 0; s < S; ++s)
            if ((words[s] >> (k & 31)) & 1u) w += __half2float(line[s]);
        acc = fmaf(__half2float(__ldcg(p.x + (size_t)m * p.K + k)), w, acc);
    }
    p.y[(size_t)m * p.N + n] = __float2half_rn(acc + (p.bias ? __half2float(p.bias[n]) : 0.0f));
}

// A chunk's sum on its way to the CTA that adds it: never the bit pattern zero, which stands for "not there yet" (p.tagged).
__device__ __forceinline__ void sb_put(float* dst, float v) { __stcg(dst, v == 0.0f ? -0.0f : v); }

// Share `share` of the chunks' sums of the group's tiles [t0, t0 + ntc) -> y, in chunk order.  The KC shares are equal parts of the (tile,
// activation row, four output rows) list; four chunks' loads are in flight per thread.  Slots that mark themselves (p.tagged): a thread
// waits for the sums it needs, p.patience cycles at most, and clears their slots once it has all of them; what does not come is
// left as it is, and false returned.  `all_here`: every sum has been stored, so slots that are empty belong to what is done.
template <int S, int NSUB>
__device__ __forceinline__ bool sb_add_share(const SbParams& p, int t0, int ntc, int share, bool all_here) {
    constexpr int TN = ts_tn(S), Q = TN / 4;
    const int total = ntc * p.M * Q;               // (at most 65 536 x 16 x 8: sb_plan)
    const int e1 = (int)((long long)total * (share + 1) / p.KC);
    const size_t plane = (size_t)p.NT * (SB_MP * TN);
    const bool wide = (reinterpret_cast<uintptr_t>(p.y) & 7) == 0;
    bool done = true;
#pragma unroll 1
    for (int e = (int)((long long)total * share / p.KC) + (int)threadIdx.x; e < e1; e += SB_THREADS) {
        const int q = e % Q, m = e / Q % p.M, tile = t0 + e / (Q * p.M);
        float* src = p.part + ((size_t)tile * SB_MP + m) * TN + q * 4;
        float v[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        bool here = true;
#pragma unroll 1
        for (int c = 0; c < p.KC; c += 4) {
            float4 t[4];
            const long long c0 = clock64();
            for (;;) {
                here = true;
#pragma unroll
                for (int h = 0; h < 4; ++h) {
                    t[h] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    if (c + h < p.KC)
                        asm volatile("ld.relaxed.gpu.global.v4.f32 {%0, %1, %2, %3}, [%4];"
                                     : "=f"(t[h].x), "=f"(t[h].y), "=f"(t[h].z), "=f"(t[h].w)
                                     : "l"(src + (size_t)(c + h) * plane)
                                     : "memory");
                }
                if (!p.tagged) break;
#pragma unroll
                for (int h = 0; h < 4; ++h)
                    if (c + h < p.KC)
                        here = here && __float_as_uint(t[h].x) && __float_as_uint(t[h].y) && __float_as_uint(t[h].z) && __float_as_uint(t[h].w);
                if (here || all_here || !done || clock64() - c0 > (long long)p.patience) break;
            }
            if (!here) break;
#pragma unroll
            for (int h = 0; h < 4; ++h) v[0] += t[h].x, v[1] += t[h].y, v[2] += t[h].z, v[3] += t[h].w;
        }
        if (!here) {
            done = false;
            continue;
        }
        if (p.tagged) {
#pragma unroll 1
            for (int c = 0; c < p.KC; ++c) __stcg(reinterpret_cast<float4*>(src + (size_t)c * plane), make_float4(0.0f, 0.0f, 0.0f, 0.0f));
        }
        const int n = tile * TN + q * 4;
        __half* dst = p.y + (size_t)m * p.N + n;
        __align__(8) __half o[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) o[i] = __float2half_rn(v[i] + (p.bias ? __half2float(p.bias[n + i]) : 0.0f));
        if (wide) {                                // (N is a multiple of TN)
            *reinterpret_cast<uint2*>(dst) = *reinterpret_cast<const uint2*>(o);
        } else {
#pragma unroll
            for (int i = 0; i < 4; ++i) dst[i] = o[i];
        }
        if (p.x) {
#pragma unroll 1
            for (int i = 0; i < 4; ++i)
                if (v[i] != v[i]) sb_multiply_out<S>(p, 256 / NSUB, m, n + i);
        }
    }
    return done;
}

__device__ __forceinline__ unsigned long long sb_load_acquire(const unsigned long long* a) {
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(a) : "memory");
    return v;
}

// The upper half of a group's word counts arrivals in parts of 2^32: with the last of them it is zero again.
__device__ __forceinline__ unsigned int sb_part_of_group(int chunk, int KC) {
    const unsigned int q = 0xffffffffu / (unsigned int)KC;
    return chunk ? q : 0u - q * (unsigned int)(KC - 1);
}

// A CTA that has given up waiting: true if the others have all arrived in the meantime, else its share is the last one's.
__device__ __forceinline__ bool sb_hand_over(unsigned long long* word, int chunk) {
    unsigned long long v = sb_load_acquire(word);
    while (v >> 32) {
        const unsigned long long old = atomicCAS(word, v, v | (1ull << chunk));
        if (old == v) return false;
        v = old;
    }
    return true;
}

// (88 registers: beside a CTA there is room for two blocks of the next call's quantiser, which 16 rows of 4096 need to be resident at
// once; with 96, at 4096 x 4096 and groups of 128, a call took 16.5 us instead of 11.8.)
template <int S, int NSUB, int IDXB>
__global__ void __maxnreg__(88) linear_sb_kernel(const __grid_constant__ CUtensorMap tmap, const __grid_constant__ SbParams p) {
    pdl_launch_dependents();
    extern __shared__ __align__(1024) unsigned char smem[];
    constexpr int SP = ts_sp(S);
    constexpr int TN = ts_tn(S);
    constexpr int MP = SB_MP, NJ = SB_NJ;
    constexpr int NV = MP / SP;                    // ... and how many of them one thread finishes
    constexpr int ABUF = NSUB == 2 ? 1 : 2;        // A buffers
    constexpr int SFC = SB_SFCOLS, BLOB = SB_BLOB;
    constexpr int WROW = TN * S * 4;               // bytes of one 32-k row of a stage
    constexpr int CI_BYTES = (IDXB == 0) ? TN * S * 2 : TN * IDXB;
    constexpr uint32_t A_TX = 8 * WROW + NSUB * CI_BYTES;
    // instruction descriptor: A, B = E2M1, scales UE8M0, M = 128, N = 32, K-major both; the scale-factor byte pair is added per MMA
    constexpr uint32_t IDESC = (1u << 7) | (1u << 10) | ((uint32_t)(32 >> 3) << 17) | (1u << 23) | (8u << 24);

    uint64_t* a_full = reinterpret_cast<uint64_t*>(smem);                            // [SB_NWG][SB_MAX_STAGES] unit landed
    uint64_t* mma_bar = a_full + SB_NWG * SB_MAX_STAGES;                             // [SB_NWG] MMAs of a unit done
    uint64_t* b_full = mma_bar + SB_NWG;                                             // [8] digits of a k block landed
    uint64_t* sf_ready = b_full + 8;                                                 // [8] its scale factors in tensor memory
    uint64_t* cache_bar = sf_ready + 8;                                              // [1] codebook landed
    uint64_t* tmem_ready = cache_bar + 1;                                            // [1] tensor memory allocated
    constexpr int SF0 = SB_NWG * (SB_MAX_STAGES + 1) + 8, NBAR = SF0 + 8 + 2;
    volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + SB_HDR - 64);
    volatile unsigned int* poison_s = reinterpret_cast<volatile unsigned int*>(smem + SB_HDR - 48);      // activation rows with a non-finite value
    uint32_t* tmem_base_s = reinterpret_cast<uint32_t*>(smem + SB_HDR - 16);

    const int N = p.N, M = p.M, KC = p.KC;
    const int grp = (int)blockIdx.x / KC, chunk = (int)blockIdx.x - grp * KC;
    const int kb0 = chunk * p.KB / KC, nkb = (chunk + 1) * p.KB / KC - kb0;
    const int t0 = (int)((long long)grp * p.NT / p.GN), ntc = (int)((long long)(grp + 1) * p.NT / p.GN) - t0;
    const int units = ntc * nkb;
    unsigned char* Bs = smem + SB_HDR;                                               // [nkb][BLOB]
    __half* cache_s = reinterpret_cast<__half*>(smem + p.off_cache);
    unsigned char* ring = smem + p.off_ring;                                         // [SB_NWG][stages][SB_ASTAGE]
    float* res = reinterpret_cast<float*>(smem + p.off_res);                         // [SB_NWG][2][MP][TN]: first, last shared tile
    const int ST = p.stages;
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;

    if (threadIdx.x < NBAR) {
        mbar_init(&a_full[threadIdx.x], ((int)threadIdx.x >= SF0 && (int)threadIdx.x < SF0 + 8) ? 4u : 1u);      // (sf_ready: four warps)
        if (threadIdx.x == 0) *abort_flag = 0;
        fence_mbar_init();
    }
    __syncthreads();
    const bool bulk_cache = p.cache_in_smem && ((p.C * S * 2) % 16 == 0);

    if (warp < SB_NWG) {
        // ------------------------------ issuer warps, one per warpgroup ------------------------------
        const int w = warp;
        const int u0 = w * units / SB_NWG, n_w = (w + 1) * units / SB_NWG - u0;
        const uint32_t ring_ws = smem_u32(ring + (size_t)w * ST * SB_ASTAGE);
        const uint32_t full_ws = smem_u32(a_full + w * SB_MAX_STAGES);
        const unsigned char* cbytes_g = (IDXB == 0) ? reinterpret_cast<const unsigned char*>(p.coeff)
                                                    : reinterpret_cast<const unsigned char*>(p.idx);
        constexpr int CIROW_PER_N = (IDXB == 0) ? S * 2 : IDXB;
        int ltile = t0 + u0 / nkb, lkl = u0 % nkb, issued = 0, lslot = 0;
        auto load_unit = [&]() {
            const int kb = kb0 + lkl, tile = ltile;
            if (++lkl == nkb) lkl = 0, ++ltile;
            const uint32_t stg = ring_ws + (uint32_t)lslot * SB_ASTAGE;
            const uint32_t bar = full_ws + (uint32_t)lslot * 8u;
            const int c0 = tile * TN * S, c1 = kb * 8;
            const unsigned char* csrc = cbytes_g + ((size_t)(kb * NSUB) * N + (size_t)tile * TN) * CIROW_PER_N;
            if (elect_one()) {
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(A_TX) : "memory");
                asm volatile(
                    "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                    ::"r"(stg), "l"(reinterpret_cast<uint64_t>(&tmap)), "r"(c0), "r"(c1), "r"(bar)
                    : "memory");
#pragma unroll
                for (int sub = 0; sub < NSUB; ++sub)
                    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                                     stg + TS_STAGE_WORDS + sub * CI_BYTES),
                                 "l"(csrc + (size_t)sub * N * CIROW_PER_N), "r"((uint32_t)CI_BYTES), "r"(bar)
                                 : "memory");
            }
            __syncwarp();
            ++issued;
            lslot = (lslot + 1 == ST) ? 0 : lslot + 1;
        };
        {
            const int first = n_w < ST ? n_w : ST;                 // the weights do not depend on the kernel in front
#pragma unroll 1
            for (int i = 0; i < first; ++i) load_unit();
        }
        if (w == 0) {
            if (bulk_cache && lane == 0) {
                mbar_arrive_expect_tx(cache_bar, (uint32_t)(p.C * S * 2));
                bulk_g2s(cache_s, p.coeff, (uint32_t)(p.C * S * 2), cache_bar);
            }
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_base_s)),
                         "r"((uint32_t)TS_TMEM_COLS)
                         : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
            ts_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(tmem_ready);
            pdl_wait();                            // the blob is written by the kernel in front of this one
            if (lane == 0) {
#pragma unroll 1
                for (int b = 0; b < nkb; ++b) {
                    mbar_arrive_expect_tx(&b_full[b], (uint32_t)BLOB);
                    bulk_g2s(Bs + (size_t)b * BLOB, p.xb + (size_t)(kb0 + b) * BLOB, (uint32_t)BLOB, &b_full[b]);
                }
            }
            __syncwarp();
        }
        ts_wait(smem_u32(tmem_ready), 0u, abort_flag, p.status, 0x420u);
        ts_fence_after();
        const uint32_t tbase = __shfl_sync(0xffffffffu, *tmem_base_s, 0);
        const uint32_t ac0 = tbase + w * SB_WGCOLS, dc = ac0 + ABUF * 32, sfa = tbase + SB_SFA_COL;
        const uint32_t bs0 = smem_u32(Bs), mbar = smem_u32(&mma_bar[w]);
        int kl = u0 % nkb;
#pragma unroll 1
        for (int i = 0; i < n_w; ++i) {
            const uint64_t bd = ts_bdesc(bs0 + (uint32_t)kl * BLOB);
            const uint32_t sc = tbase + SB_SFB_COL + kl * SFC, ac = ac0 + (ABUF == 2 ? (i & 1) * 32 : 0);
            if (i < nkb) {                         // this block's digits and scale factors are in place (first time round)
                ts_wait(smem_u32(&b_full[kl]), 0u, abort_flag, p.status, 0x422u);
                ts_wait(smem_u32(&sf_ready[kl]), 0u, abort_flag, p.status, 0x421u);
            }
            if (++kl == nkb) kl = 0;
            named_bar_sync(1 + w, 160);            // A of unit i is in tensor memory, D has been read
            ts_fence_after();
            if (elect_one()) {
#pragma unroll
                for (int c = 0; c < 4; ++c)
#pragma unroll
                    for (int jm = 0; jm < NJ; ++jm) {
                        const int sub = (NSUB == 2) ? (c >> 1) : 0;
                        const bool first = (jm == 0) && ((NSUB == 2) ? ((c & 1) == 0) : (c == 0));
                        const uint32_t sfid = (uint32_t)((jm & 1) * 2);
                        ts_mma(dc + sub * 32, ac + c * 8, bd + (uint64_t)((jm * 4096 + c * 256) >> 4),
                               IDESC | (sfid << 4) | (sfid << 29), sfa, sc + 4 * (jm >> 1), (uint32_t)!first);
                    }
                asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar) : "memory");
            }
            __syncwarp();
            if (issued < n_w) {                    // every compute warp has read the stage of unit i: refill it
                fence_proxy_async();
                load_unit();
            }
        }
        if (lane == 0) {                           // no copy of this warp is in flight when the CTA leaves
            const int firstj = issued > ST ? issued - ST : 0;
#pragma unroll 1
            for (int jx = firstj; jx < issued; ++jx)
                ts_wait(full_ws + (uint32_t)(jx % ST) * 8u, (uint32_t)((jx / ST) & 1), abort_flag, p.status, 0x423u, false);
            if (w == 0 && bulk_cache) ts_wait(smem_u32(cache_bar), 0u, abort_flag, p.status, 0x411u, false);
            for (int b = 0; w == 0 && b < nkb; ++b) ts_wait(smem_u32(&b_full[b]), 0u, abort_flag, p.status, 0x412u, false);
        }
    } else {
        // ------------------------------ compute warpgroups ------------------------------
        const int w = (warp - SB_CW0) >> 2, wl = warp & 3;
        const int u0 = w * units / SB_NWG, n_w = (w + 1) * units / SB_NWG - u0;
        const int r = wl * 32 + lane;              // MMA row = tensor-memory lane
        const int nl = r / SP, s = r % SP;
        const bool live_row = (S != 3) || (s < S);
        const uint32_t lane_sel = (uint32_t)(wl * 32) << 16;
        const unsigned char* ring_w = ring + (size_t)w * ST * SB_ASTAGE;
        const uint32_t full_ws = smem_u32(a_full + w * SB_MAX_STAGES);
        const uint32_t mbar = smem_u32(&mma_bar[w]);

        if (p.cache_in_smem && !bulk_cache) {
            const int tid = threadIdx.x - SB_CW0 * 32;
            for (int i = tid; i < p.C * S; i += SB_NWG * 128) cache_s[i] = p.coeff[i];
            named_bar_sync(15, SB_NWG * 128);
        }
        ts_wait(smem_u32(tmem_ready), 0u, abort_flag, p.status, 0x430u);
        ts_fence_after();
        const uint32_t tbase = __shfl_sync(0xffffffffu, *tmem_base_s, 0);
        if (w == 0) {
            // scale factors, for the whole launch: every byte 2^0 for A; for B word i (MMAs 2 i, 2 i + 1) of a row in column 0 of
            // the block's i-th 4-column block, the same in all four lane quadrants
            uint32_t f[32];
#pragma unroll
            for (int i = 0; i < 32; ++i) f[i] = 0x7F7F7F7Fu;
            ts_st32(tbase + lane_sel + SB_SFA_COL, f);
            unsigned int pm = 0u;
#pragma unroll 1
            for (int b = 0; b < nkb; ++b) {
                ts_wait(smem_u32(&b_full[b]), 0u, abort_flag, p.status, 0x433u);
                const uint4 sf = reinterpret_cast<const uint4*>(Bs + (size_t)b * BLOB + NJ * 4096)[lane];
                const uint32_t at = tbase + lane_sel + SB_SFB_COL + b * SFC;
                ts_st8(at, sf.x, 0x7F7F7F7Fu, 0x7F7F7F7Fu, 0x7F7F7F7Fu, sf.y, 0x7F7F7F7Fu, 0x7F7F7F7Fu, 0x7F7F7F7Fu);
                ts_st8(at + 8, sf.z, 0x7F7F7F7Fu, 0x7F7F7F7Fu, 0x7F7F7F7Fu, 0x7F7F7F7Fu, 0x7F7F7F7Fu, 0x7F7F7F7Fu, 0x7F7F7F7Fu);
                pm |= __ballot_sync(0xffffffffu, lane < MP && sf.w != 0u);
                if (wl == 0 && b == nkb - 1) *poison_s = pm;
                ts_wait_st();
                ts_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&sf_ready[b]);
            }
        }
        if (bulk_cache) ts_wait(smem_u32(cache_bar), 0u, abort_flag, p.status, 0x431u);

        const uint32_t a_addr = tbase + w * SB_WGCOLS + lane_sel, d_addr = a_addr + ABUF * 32;
        SbPair acc[MP / 2];                        // sums of this lane's (row, plane), two activation rows each
#pragma unroll
        for (int m = 0; m < MP / 2; ++m) acc[m] = SbPair(0.0f, 0.0f);
        const int wpos = nl * S + s;
        int tile = t0 + u0 / nkb, have = 0;        // tile of the sums, units of it in them
        // Sums of one tile's units: planes added across their lanes, after which a lane has the activation rows
        // m = s NV .. s NV + NV - 1 of its output row.  A tile that is all this warpgroup's goes out at once, one that it
        // shares with a neighbour (its first or its last) to shared memory.
        auto deposit = [&](bool last) {
            float v[MP];
#pragma unroll
            for (int m = 0; m < MP / 2; ++m) acc[m].get(v[2 * m], v[2 * m + 1]), acc[m] = SbPair(0.0f, 0.0f);
#pragma unroll
            for (int o = SP / 2, n2 = MP / 2; o; o >>= 1, n2 >>= 1) {
                const bool up = (s & o) != 0;
#pragma unroll
                for (int i = 0; i < n2; ++i) {
                    const float keep = up ? v[i + n2] : v[i], send = up ? v[i] : v[i + n2];
                    v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
                }
            }
            if (have != nkb) {
                float* dst = res + (size_t)(w * 2 + (last ? 1 : 0)) * (MP * TN) + nl;
#pragma unroll
                for (int e = 0; e < NV; ++e) dst[(s * NV + e) * TN] = v[e];
            } else {
                const unsigned int pm = *poison_s;
#pragma unroll
                for (int e = 0; e < NV; ++e)
                    if ((pm >> (s * NV + e)) & 1u) v[e] = __int_as_float(0x7fc00000);
                if (KC > 1) {
                    float* dst = p.part + ((size_t)chunk * p.NT + tile) * (MP * TN) + nl;
#pragma unroll
                    for (int e = 0; e < NV; ++e)
                        if (s * NV + e < M) sb_put(dst + (s * NV + e) * TN, v[e]);
                } else {
                    const int n = tile * TN + nl;
                    const float bias = p.bias ? __half2float(p.bias[n]) : 0.0f;
#pragma unroll
                    for (int e = 0; e < NV; ++e)
                        if (s * NV + e < M) p.y[(size_t)(s * NV + e) * N + n] = __float2half_rn(v[e] + bias);
                    if (p.x && pm) {
#pragma unroll 1
                        for (int m = s * NV; m < s * NV + NV; ++m)
                            if ((pm >> m) & 1u) sb_multiply_out<S>(p, 256 / NSUB, m, n);
                    }
                }
            }
            have = 0;
            ++tile;
        };
        uint32_t wv[8];                            // packed words and coefficients of the unit to be expanded next
        float cf[NSUB], c1[NSUB], c0[NSUB];        // ... of the expanded one, and of the one whose sums are read
        int aslot = 0;
        uint32_t apar = 0u;
        auto fetch = [&]() {
            ts_wait(full_ws + (uint32_t)aslot * 8u, apar, abort_flag, p.status, 0x432u);
            const unsigned char* stg = ring_w + (size_t)aslot * SB_ASTAGE;
            const uint32_t* wsrc = reinterpret_cast<const uint32_t*>(stg) + wpos;
#pragma unroll
            for (int kw = 0; kw < 8; ++kw) wv[kw] = live_row ? wsrc[kw * (WROW / 4)] : 0u;
#pragma unroll
            for (int sub = 0; sub < NSUB; ++sub) {
                const unsigned char* cs = stg + TS_STAGE_WORDS + sub * CI_BYTES;
                float c = 0.0f;
                if constexpr (IDXB == 0) {
                    if (live_row) c = __half2float(reinterpret_cast<const __half*>(cs)[nl * S + s]);
                } else {
                    const uint32_t ci = (IDXB == 1) ? (uint32_t)cs[nl] : (uint32_t)reinterpret_cast<const unsigned short*>(cs)[nl];
                    if (live_row) c = __half2float((p.cache_in_smem ? cache_s : p.coeff)[(size_t)ci * S + s]);
                }
                cf[sub] = c;
            }
            if (++aslot == ST) {
                aslot = 0;
                apar ^= 1u;
            }
        };
        // packed words of this thread's row -> 32 words of 4-bit elements {0, 1 | 1 | 2 | 2}
        auto expand = [&](int buf) {
#pragma unroll
            for (int h = 0; h < 4; ++h) {
                const uint32_t w0 = wv[2 * h], w1 = wv[2 * h + 1];
                ts_st8(a_addr + buf * 32 + h * 8, (w0 << 1) & 0x22222222u, w0 & 0x22222222u, w0 & 0x44444444u, (w0 >> 1) & 0x44444444u,
                       (w1 << 1) & 0x22222222u, w1 & 0x22222222u, w1 & 0x44444444u, (w1 >> 1) & 0x44444444u);
            }
        };
        if (n_w > 0) {
            fetch();
            expand(0);
#pragma unroll
            for (int sub = 0; sub < NSUB; ++sub) c1[sub] = cf[sub];
            if (n_w > 1) fetch();
            ts_wait_st();
            ts_fence_before();
            ts_bar_arrive(1 + w, 160);             // releases the MMAs of unit 0
        }
        int kl = u0 % nkb;                         // k block of unit i
#pragma unroll 1
        for (int i = 0; i < n_w; ++i) {
            const bool more = i + 1 < n_w;
            auto next = [&]() {                    // unit i + 1 into A, unit i + 2 out of shared memory
                if (more) {
                    expand(ABUF == 2 ? (i + 1) & 1 : 0);
#pragma unroll
                    for (int sub = 0; sub < NSUB; ++sub) c1[sub] = cf[sub];
                    if (i + 2 < n_w) fetch();
                }
            };
#pragma unroll
            for (int sub = 0; sub < NSUB; ++sub) c0[sub] = c1[sub];
            if (ABUF == 2) next();
            ts_wait(mbar, (uint32_t)(i & 1), abort_flag, p.status, 0x434u);
            ts_fence_after();
            // the sums of one group: even and odd digits of every activation row
            SbPair v[MP / 2];
            auto read = [&](int sub) {
                uint32_t d[4][8];
                ts_ld16_issue(d_addr + sub * 32, d[0], d[1]);
                ts_ld16_issue(d_addr + sub * 32 + 16, d[2], d[3]);
                if (ABUF == 1 && sub == 0) next();
#pragma unroll
                for (int g4 = 0; g4 < 4; ++g4) ts_wait_ld(d[g4]);
#pragma unroll
                for (int m = 0; m < MP; m += 2)
                    v[m / 2] = SbPair(d[m >> 3][m & 7], d[m >> 3][(m & 7) + 1]) + SbPair(d[2 + (m >> 3)][m & 7], d[2 + (m >> 3)][(m & 7) + 1]);
            };
            auto fold = [&](int sub) {
#pragma unroll
                for (int m = 0; m < MP / 2; ++m) acc[m] = v[m].mul_add(SbPair(c0[sub], c0[sub]), acc[m]);
            };
#pragma unroll
            for (int sub = 0; sub < NSUB; ++sub) { // (one after the other: both groups' sums at once need 96 registers)
                read(sub);
                if (sub + 1 < NSUB) fold(sub);
            }
            if (more) {
                ts_wait_st();
                ts_fence_before();
                ts_bar_arrive(1 + w, 160);         // releases the MMAs of unit i + 1; also: its stage has been read
            }
            fold(NSUB - 1);
            ++have;
            if (++kl == nkb || !more) {
                kl = 0;
                // (a shared tile's sums: the last tile of the warpgroup's range unless the range lies inside one tile)
                deposit(!more && tile > t0 + u0 / nkb);
            }
        }
    }
    ts_fence_before();
    __syncthreads();
    ts_fence_after();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(*tmem_base_s), "r"((uint32_t)TS_TMEM_COLS)
                     : "memory");

    // ------------------------------ tiles shared by warpgroups ------------------------------
    // Tile `tl` of the range has units [tl nkb, (tl + 1) nkb), warpgroup w the units [w U / 4, (w + 1) U / 4); where a boundary
    // lies inside a tile its warpgroups' sums are added here, in warpgroup order, by a warp per quarter of the tile.
    if (warp < 4 * (SB_NWG - 1)) {
        constexpr int QR = TN / 4;                 // rows of a quarter
        const int wb = (warp >> 2) + 1, qt = warp & 3;
        const int bd = wb * units / SB_NWG, tl = bd / nkb;
        // (a tile with several boundaries belongs to the first of them)
        if (bd != tl * nkb && (wb == 1 || (wb - 1) * units / SB_NWG <= tl * nkb)) {
            const unsigned int pm = *poison_s;
            for (int q = lane; q < MP * QR; q += 32) {
                const int m = q / QR, nl = qt * QR + q % QR, n = (t0 + tl) * TN + nl;
                if (m >= M) break;
                float v = 0.0f;
#pragma unroll
                for (int w = 0; w < SB_NWG; ++w) {
                    const int a = w * units / SB_NWG, b = (w + 1) * units / SB_NWG;
                    if (a < (tl + 1) * nkb && b > tl * nkb && a < b) v += res[(size_t)(w * 2 + (tl > a / nkb ? 1 : 0)) * (MP * TN) + m * TN + nl];
                }
                if ((pm >> m) & 1u) v = __int_as_float(0x7fc00000);
                if (KC > 1) sb_put(p.part + ((size_t)chunk * p.NT + t0 + tl) * (MP * TN) + m * TN + nl, v);
                else p.y[(size_t)m * N + n] = __float2half_rn(v + (p.bias ? __half2float(p.bias[n]) : 0.0f));
                if (KC == 1 && p.x && ((pm >> m) & 1u)) sb_multiply_out<S>(p, 256 / NSUB, m, n);
            }
        }
    }
    // ------------------------------ the chunks of K meet ------------------------------
    // The CTAs of a group add equal shares of its sums, but nothing depends on their running at the same time: other streams' kernels may
    // hold the SMs that some of them need.  A CTA that is through counts itself in the upper half of the group's word, which is zero
    // again when all have: every sum is there then.  One that has stopped waiting for that leaves its bit in the lower half, unless the upper
    // half is zero by now, and ends; the last one finds the bits in the value that its count met, and takes those shares over.  Few
    // sums: their slots are zero before the launch, whoever needs one takes it as soon as it is not, and clears it; the word then
    // only says who is last (waiting for it before the sums are read takes 1.5 us longer).
    if (KC > 1) {
        volatile unsigned int* share_s = reinterpret_cast<volatile unsigned int*>(smem + SB_HDR - 32);
        unsigned long long* word = p.arrive + grp;
        const bool speaker = threadIdx.x == SB_THREADS - 32;          // (of a warp that has few sums to add or none)
        const unsigned int part = sb_part_of_group(chunk, KC);
        unsigned long long before = 0ull;
        __syncwarp();
        if (warp == SB_THREADS / 32 - 1) named_bar_sync(14, SB_THREADS);        // every warp's sums are stored
        else ts_bar_arrive(14, SB_THREADS);
        if (speaker) {
            __threadfence();
            before = atomicAdd(word, (unsigned long long)part << 32);
        }
        bool done = false;
        if (p.tagged) done = __syncthreads_and(sb_add_share<S, NSUB>(p, t0, ntc, chunk, false));
        if (speaker) {
            const unsigned int mine = done ? 0u : 1u << chunk;
            unsigned int shares = 0u;
            if ((unsigned int)(before >> 32) + part == 0u) {          // the last one; nobody sets a bit from here on
                shares = (unsigned int)before | mine;
                if ((unsigned int)before) atomicExch(word, 0ull);
            } else if (!done) {
                const long long c0 = clock64();
                bool all = false;
                while (!p.tagged && !(all = (sb_load_acquire(word) >> 32) == 0ull) && clock64() - c0 <= (long long)p.patience) {
                }
                if (!all) __threadfence();         // (slots cleared here come before the bit that leaves the rest to another)
                if (all || sb_hand_over(word, chunk)) shares = mine;
            }
            if (shares) __threadfence();
            *share_s = shares;
        }
        __syncthreads();
#pragma unroll 1
        for (unsigned int shares = *share_s; shares; shares &= shares - 1)
            sb_add_share<S, NSUB>(p, t0, ntc, __ffs((int)shares) - 1, true);
    }
    if (threadIdx.x == 0 && *abort_flag) {         // which problem gave up: N, and K / 256 | M | CTA (for the host's message)
        atomicExch(p.status + 2, (unsigned int)p.N);
        atomicExch(p.status + 3, ((unsigned int)p.KB << 16) | ((unsigned int)M << 8) | (blockIdx.x & 0xFFu));
    }
}

// ---------------------------------------------------------------------------------------------
// host
// ---------------------------------------------------------------------------------------------
struct SbPlan {
    int KB, NT, KC, GN, cache_in_smem, stages, smem;
    int off_cache, off_ring, off_res;
    size_t blob_bytes, part_bytes;
};

static int sb_plan(const PackedW& w, const DeviceInfo& di, SbPlan* pl) {
    const int TN = ts_tn(w.S), MP = SB_MP;
    pl->KB = w.K / 256;
    pl->NT = w.N / TN;
    if (pl->KB < 1 || pl->NT < 1) return SBVR_ERR_UNSUPPORTED;
    // Chunks as large as shared memory holds; smaller ones while less than two thirds of the SMs would have work and a
    // warpgroup more than one unit.
    pl->KC = (pl->KB + SB_CHUNK - 1) / SB_CHUNK;
    auto groups = [&](int kc) { const int g = di.sm_count / kc; return g < 1 ? 1 : (g < pl->NT ? g : pl->NT); };
    while (groups(pl->KC) * pl->KC * 3 <= di.sm_count * 2 && pl->KC * 2 <= pl->KB && pl->KC * 2 <= 16 &&
           (pl->NT + groups(pl->KC) - 1) / groups(pl->KC) * (pl->KB / pl->KC) > SB_NWG)
        pl->KC *= 2;
    pl->GN = groups(pl->KC);
    const int nkb = (pl->KB + pl->KC - 1) / pl->KC;
    if (pl->KC > 1 && pl->NT > 65536) return SBVR_ERR_UNSUPPORTED;       // (what has been covered: two million rows)
    if (pl->KC > 32) return SBVR_ERR_UNSUPPORTED;                        // bits of a group's word
    pl->blob_bytes = ((size_t)pl->KB * SB_BLOB + 255) / 256 * 256;
    pl->part_bytes = pl->KC > 1 ? (size_t)pl->KC * pl->NT * MP * TN * 4 : 0;
    const int cache_bytes = w.idx_bytes ? ts_round_up(w.C * w.S * 2, 16) : 0;
    auto layout = [&](int cb, int stages) {
        pl->off_cache = SB_HDR + nkb * SB_BLOB;
        pl->off_ring = ts_round_up(pl->off_cache + cb, 128);
        pl->off_res = pl->off_ring + SB_NWG * stages * SB_ASTAGE;
        return pl->off_res + SB_NWG * 2 * MP * TN * 4;
    };
    pl->cache_in_smem = (w.idx_bytes && cache_bytes <= 65536 && layout(cache_bytes, 2) <= di.smem_optin) ? 1 : 0;
    const int cb = pl->cache_in_smem ? cache_bytes : 0;
    int st = SB_MAX_STAGES;
    while (st > 2 && layout(cb, st) > di.smem_optin) --st;
    pl->stages = st;
    pl->smem = layout(cb, st);
    if (pl->smem > di.smem_optin) return SBVR_ERR_UNSUPPORTED;
    return SBVR_OK;
}

bool linear_sb_supported(const PackedW& w, int M) {
    if (w.S < 2 || w.S > 4) return false;
    if (w.G != 256 && w.G != 128) return false;
    if (M < 2 || M > SB_MP) return false;
    if (w.N % ts_tn(w.S) || w.K % 256 || w.K > 32768) return false;
    if (w.idx_bytes < 0 || w.idx_bytes > 2) return false;
    if (reinterpret_cast<uintptr_t>(w.coeff) & 15) return false;                 // bulk copies
    if (reinterpret_cast<uintptr_t>(w.bvr) & 15) return false;                   // tensor map base
    if (w.idx_bytes && (reinterpret_cast<uintptr_t>(w.idx) & 15)) return false;
    if ((size_t)(w.N / ts_tn(w.S)) * (size_t)(w.K / 256) >= ((size_t)1 << 24)) return false;   // 32-bit unit arithmetic
    if ((size_t)w.N * w.S >= ((size_t)1 << 31)) return false;                    // 32-bit tensor coordinates
    DeviceInfo di;
    int dev = 0;
    SbPlan pl;
    if (cudaGetDevice(&dev) != cudaSuccess || device_info(dev, &di) != SBVR_OK) return false;
    return sb_plan(w, di, &pl) == SBVR_OK;
}

// Where the automatic choice takes it.  Up to four chunks of K, and few rows of a long K, it is the faster one: M = 16, S = 4, us, here and the GEMM:
// 1024 x 4096 11.2, 11.1; 4096 x 4096 12.5, 13.8; 14336 x 4096 23.8, 27.9; 32768 x 1024 15.4, 20.9; 128 x 14336 12.8, 20.2.  Up to 2048 rows the
// chunks' merge costs what the product gains: 1024 x 14336 17.5, 15.0; 512 x 28672 19.7, 22.0.
// More chunks and more rows: the line lies where it was drawn against an earlier GEMM, which split K evenly (linear_gemm_split still says how), by
// estimates of both kernels' times.  It stays there for the sake of the results: this kernel's are off by 2.1e-4 (2-norm;
// the rounding to fp16), the GEMM's by 3.1e-4 to 3.6e-4 with its weights formed in fp16, and a call that had the former keeps it.  What that costs
// now, over 140 calls drawn from 2048 .. 14336 rows, K 4352 .. 28672, 5 .. 16 rows of x: 10 % on average, nothing at half of them, at most 73 % (2176 x
// 26368, S = 3, groups of 128, M = 16: 41.9 us, 24.3).
bool linear_sb_preferred(const PackedW& w, int M, const DeviceInfo& di) {
    if (w.K <= 4096 || w.N <= 256) return true;
    if (w.N < 2048) return false;
    SbPlan pl;
    if (sb_plan(w, di, &pl) != SBVR_OK) return false;
    const int tiles = (pl.NT + pl.GN - 1) / pl.GN, blocks = (pl.KB + pl.KC - 1) / pl.KC;
    const float units = (float)((tiles * blocks + SB_NWG - 1) / SB_NWG);
    const float here = 10.0f + (w.G == 128 ? 1.6f : 1.15f) * units + 0.15f * (float)pl.KC + 4.2e-6f * (float)pl.KC * (float)w.N * (float)M;
    int parts, stages;
    linear_gemm_split(w, M, di.sm_count, &parts, &stages);
    return here < 4.5f + (0.1f + 0.12f * (float)w.S) * (w.idx_bytes ? 1.0f : 0.87f) * (float)stages + 1.8e-4f * (float)parts * (float)w.N;
}

size_t linear_sb_workspace_bytes(const PackedW& w, const DeviceInfo& di) {
    SbPlan pl;
    if (sb_plan(w, di, &pl) != SBVR_OK) return 0;
    return pl.blob_bytes + pl.part_bytes + (size_t)SB_MP * w.K * 2;
}

// The kernel asks for all of the SM's shared memory, once per device: a CTA whose size just filled a smaller carve-out (196 KB
// with three planes and 4 096 lines) left no room for the next call's quantiser beside it, and a call took 8 us more.
template <typename Kernel>
static int sb_setup(SmemOnce& once, Kernel kernel, int bytes) {
    int dev = 0;
    SBVR_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return SBVR_ERR_BAD_ARG;
    std::lock_guard<std::mutex> lock(once.mu);
    if (!once.done[dev]) {
        SBVR_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
        SBVR_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
        once.done[dev] = true;
    }
    return SBVR_OK;
}

template <int S, int NSUB, int IDXB>
static int sb_launch_inst(const CUtensorMap& tm, const SbParams& p, int grid, int smem, cudaStream_t st) {
    static SmemOnce once;
    const int rc = sb_setup(once, linear_sb_kernel<S, NSUB, IDXB>, 227 * 1024);
    if (rc) return rc;
    SBVR_CUDA_TRY(launch_pdl(linear_sb_kernel<S, NSUB, IDXB>, dim3(grid), dim3(SB_THREADS), (size_t)smem, st, tm, p));
    return SBVR_OK;
}
template <int S, int NSUB>
static int sb_launch_idx(const CUtensorMap& tm, const SbParams& p, int idxb, int grid, int smem, cudaStream_t st) {
    switch (idxb) {
        case 0: return sb_launch_inst<S, NSUB, 0>(tm, p, grid, smem, st);
        case 1: return sb_launch_inst<S, NSUB, 1>(tm, p, grid, smem, st);
        default: return sb_launch_inst<S, NSUB, 2>(tm, p, grid, smem, st);
    }
}
template <int S>
static int sb_launch_g(const CUtensorMap& tm, const SbParams& p, int G, int idxb, int grid, int smem, cudaStream_t st) {
    return G == 128 ? sb_launch_idx<S, 2>(tm, p, idxb, grid, smem, st) : sb_launch_idx<S, 1>(tm, p, idxb, grid, smem, st);
}

// `xchg` (SBVR_WS_XCHG_BYTES), `arrive` (8 bytes per SM) -- both zero between calls: the kernel leaves them zero -- and `scratch`
// (256-byte aligned, linear_sb_workspace_bytes long: digit blob, the chunks' sums, rows an op has made) are the caller's.
int launch_linear_sb(const __half* x, const PackedW& w, const __half* bias, __half* y, int M, int device, unsigned int* status,
                     float* xchg, unsigned long long* arrive, unsigned int patience, char* scratch, size_t scratch_bytes,
                     bool multiply_out, cudaStream_t st, const XOp* xop) {
    if (!linear_sb_supported(w, M)) return SBVR_ERR_UNSUPPORTED;
    if (!status || !xchg || !arrive || !scratch) return SBVR_ERR_WORKSPACE;
    if (reinterpret_cast<uintptr_t>(x) & 1) return SBVR_ERR_ALIGN;
    if (reinterpret_cast<uintptr_t>(scratch) & 255) return SBVR_ERR_ALIGN;
    DeviceInfo di;
    int rc = device_info(device, &di);
    if (rc) return rc;
    if (di.cc_major != 10) return SBVR_ERR_UNSUPPORTED;
    SbPlan pl;
    rc = sb_plan(w, di, &pl);
    if (rc) return rc;
    if (linear_sb_workspace_bytes(w, di) > scratch_bytes) return SBVR_ERR_WORKSPACE;
    CUtensorMap tm;
    rc = ts_tensor_map(w, 1, &tm);
    if (rc) return rc;
    SbQuant q;
    q.x = x, q.xb = reinterpret_cast<unsigned char*>(scratch), q.M = M, q.K = w.K;
    rc = xop_check(xop, x, M, w.K, &q.x_op, &q.delta, &q.norm_w, &q.h_out, &q.eps);
    if (rc) return rc;
    // (an op in front: its result is kept for rows that have to be multiplied out)
    q.x_out = q.x_op != SBVR_XOP_NONE && multiply_out ? reinterpret_cast<__half*>(scratch + pl.blob_bytes + pl.part_bytes) : nullptr;
    SBVR_CUDA_TRY(launch_pdl(sb_quant_kernel, dim3(pl.KB, SB_MP), dim3(128), 0, st, q));
    SbParams p;
    p.xb = q.xb;
    p.idx = w.idx, p.coeff = w.coeff, p.bias = bias, p.y = y, p.status = status, p.arrive = arrive, p.patience = patience;
    p.tagged = pl.KC > 1 && pl.part_bytes <= SBVR_WS_XCHG_BYTES;
    p.part = p.tagged ? xchg : reinterpret_cast<float*>(scratch + pl.blob_bytes);
    p.x = !multiply_out ? nullptr : q.x_out ? q.x_out : x, p.bvr = w.bvr, p.idx_bytes = w.idx_bytes;
    p.M = M, p.N = w.N, p.K = w.K, p.KB = pl.KB, p.NT = pl.NT, p.C = w.C, p.KC = pl.KC, p.GN = pl.GN;
    p.cache_in_smem = pl.cache_in_smem, p.stages = pl.stages;
    p.off_cache = pl.off_cache, p.off_ring = pl.off_ring, p.off_res = pl.off_res;
    const int grid = pl.GN * pl.KC;
    switch (w.S) {
        case 2: return sb_launch_g<2>(tm, p, w.G, w.idx_bytes, grid, pl.smem, st);
        case 3: return sb_launch_g<3>(tm, p, w.G, w.idx_bytes, grid, pl.smem, st);
        default: return sb_launch_g<4>(tm, p, w.G, w.idx_bytes, grid, pl.smem, st);
    }
}

}  // namespace sbvr
