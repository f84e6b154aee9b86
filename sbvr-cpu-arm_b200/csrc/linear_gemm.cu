// SBVR linear for more than four activation rows (small batches and prefill): a tcgen05 fp16 GEMM whose
// weight operand is dequantised inside the kernel and never exists in memory.
//
//   y[m, n] = sum_k x[m, k] * W[n, k] (+ bias[n]),   W[n, k] = sum_s c[k/G, n, s] * bit_s[n, k]
//
// Operands of tcgen05.mma kind::f16 (fp32 accumulation in tensor memory), D[128 weight rows, NX activation rows]:
//
//  A (weights, from tensor memory)  Decoder thread r of a warpgroup owns weight row r of the tile.  Per 64 k it
//      loads its 2 x S packed words, turns them into 64 fp16 values and stores them to its tensor-memory lane
//      (tcgen05.st): decoded weights never touch shared or global memory.  The value of an element is the sum of
//      the c_s whose plane bit is set, formed two elements at a time in half2: a lone bit at position 10 .. 14 of a
//      half is a power of two, so `word & (0x04000400 << i)` is (2^e * bit_j, 2^e * bit_{j+16}) and one HFMA2 with
//      c_s / 2^e adds c_s where the bits are set: a mask and an HFMA2 per plane per pair of elements, plus three
//      shifted copies per word (rows with |c_s| >= 3.9 use sign flips around sum_s c_s / 2 instead: shift, LOP3,
//      HADD2).  Elements j and j + 16 of a word share a 32-bit column, so the K order inside each 32-k word is
//      permuted (position p <-> k = p/2 + 16 (p & 1)).
//  B (activations, from shared memory)  x is first re-tiled by a small kernel into the blocked layout the MMA
//      reads (8-row x 16-byte core matrices, K-major, no swizzle) with the same K permutation, one contiguous
//      block per (NX rows, 64 k); the GEMM fetches a block with a single bulk asynchronous copy.
//
// Replaces `x @ decode().T` of the reference's Llama flow for prefill (reference sbvr_utils/utils_llama.py:147,
// sbvr/core.py:926-949) and the M > 1 use of `_sbvr_row_deq_mm_T` (sbvr/kernels/sbvr_kernel.cu:121-191).
// Accuracy: weights are formed in fp16 with one rounding per plane (not the single rounding of decode()), which
// perturbs a weight by at most a few fp16 ulps of its partial sums; products accumulate in fp32.
//
// Structure: persistent CTAs of 18 warps.  Warps 0-15 are four decoder warpgroups that take the 64-k stages
// round-robin and, once the MMAs of a work item have finished, read D from tensor memory, add the bias and
// write fp16 (or fp32 partial sums when K is split over several CTAs: small activation batches on wide GPUs;
// the last CTA to arrive adds the parts in a fixed order, so results do not depend on timing).  Warp 16 issues
// the MMAs from one elected lane; warp 17 streams the activation blocks.
//
// What bounds it (2048 x 14336 x 4096, S = 4, 256-row tiles, about 850 cycles per 64-k stage): the decoders, about 540 instructions
// per scheduler and stage with half of the integer pipe busy; without their arithmetic a stage takes 640, with 512 of tensor time.
// The issuing lane was as long before (a probe of two barriers for the next stages, elections and descriptor arithmetic on the path
// between two stages: 740 cycles with everything in place); now one barrier stands for both operands, the next stage's is read
// ahead, descriptors move by constants and the tensor-memory addresses are immediates.  Every wait is bounded; on a time-out
// the kernel records it in the status word, skips the remaining work without skipping a barrier, frees its
// tensor memory and returns.
#include "common.cuh"

namespace sbvr {

constexpr int GM_DWGS = 4;
constexpr int GM_DTHREADS = GM_DWGS * 128;
constexpr int GM_IWARP = GM_DWGS * 4;
constexpr int GM_PWARP = GM_IWARP + 1;
constexpr int GM_THREADS = (GM_PWARP + 1) * 32;
constexpr int GM_TMEM_COLS = 512;
// NX activation rows per tile.  NX = GM_WIDE stands for any multiple of 32 in (256, 384] (GmParams::nx): every stage is then two
// MMAs per 16 k, 256 columns and the rest, and a decoded weight tile serves up to 1.5 times as many activations.
constexpr int GM_WIDE = 384;
// Ring of 64-k stages: a decoded 128 x 64 weight tile in tensor memory and the activation block in shared memory.
__host__ __device__ constexpr int gm_slots(int NX, bool EXACT) { return (NX == GM_WIDE || EXACT) ? 4 : 6; }
__host__ __device__ constexpr int gm_a_col(int NX) { return NX == GM_WIDE ? 384 : 256; }   // D occupies columns [0, NX), the A ring is behind
constexpr int GM_HDR = 1024;

struct GmParams {
    const __half* xt;            // re-tiled activations [MT][K/64][NX*64]
    const uint32_t* bvr;
    const void* idx;
    const __half* coeff;
    const __half* bias;
    __half* y;
    float* part;                 // [KS][MT*NX][N] fp32 partial sums (KS > 1)
    unsigned int* counters;      // one per output tile, zero between launches
    unsigned int* status;
    int M, N, K, C, G, idx_bytes;
    int nx;                      // activation rows of a tile
    int NT, MT, KS, SPP, items;  // weight-row tiles, activation-row tiles, k parts, 64-k stages per part
};

__device__ __forceinline__ void gm_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void gm_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// B descriptor: K-major, no swizzle, 128 B between core matrices along K, 1024 B between 8-row groups; version 1.  Its upper word is
// a constant; the lower one moves by (bytes >> 4).
__device__ __forceinline__ uint32_t gm_bdesc_lo(uint32_t saddr) { return (saddr >> 4) | ((128u >> 4) << 16); }
__device__ __forceinline__ void gm_mma(uint32_t d_t, uint32_t a_t, uint32_t bdesc_lo, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 d;\n\tsetp.ne.b32 p, %4, 0;\n\tmov.b64 d, {%2, %5};\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], d, %3, p;\n\t}" ::"r"(d_t),
        "r"(a_t), "r"(bdesc_lo), "r"(idesc), "r"(accumulate), "r"((1024u >> 4) | (1u << 14))
        : "memory");
}
__device__ __forceinline__ void gm_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ void gm_st32(uint32_t taddr, const uint32_t (&a)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
        "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};" ::"r"(taddr),
        "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]), "r"(a[7]), "r"(a[8]), "r"(a[9]),
        "r"(a[10]), "r"(a[11]), "r"(a[12]), "r"(a[13]), "r"(a[14]), "r"(a[15]), "r"(a[16]), "r"(a[17]), "r"(a[18]),
        "r"(a[19]), "r"(a[20]), "r"(a[21]), "r"(a[22]), "r"(a[23]), "r"(a[24]), "r"(a[25]), "r"(a[26]), "r"(a[27]),
        "r"(a[28]), "r"(a[29]), "r"(a[30]), "r"(a[31])
        : "memory");
}
__device__ __forceinline__ void gm_st16(uint32_t taddr, const uint32_t (&a)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr),
        "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]), "r"(a[7]), "r"(a[8]), "r"(a[9]),
        "r"(a[10]), "r"(a[11]), "r"(a[12]), "r"(a[13]), "r"(a[14]), "r"(a[15])
        : "memory");
}
// A pair of weights as two fp16 parts each, of the same sign and never zero unless the weight is at most 2^-24: part one is cut
// towards zero a little below the weight, part two is the rest (weights are multiples of 2^-24, so below 2^-3 it is exact; above,
// the two parts hold 21 bits).  Same signs and no zeros, so that an infinite activation gives what one product would.
__device__ __forceinline__ void gm_two_parts(float v0, float v1, bool odd, uint32_t& hi, uint32_t& lo) {
    constexpr float BELOW = 1.0f - 1.0f / 4096;
    asm("cvt.rz.f16x2.f32 %0, %1, %2;" : "=r"(hi) : "f"(v1 * BELOW), "f"(v0 * BELOW));
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&hi));
    float r0 = v0 - f.x, r1 = v1 - f.y;
    if (odd) {                                     // a coefficient that is not finite: part one says it all
        if (!(fabsf(v0) < INFINITY)) r0 = 0.0f;
        if (!(fabsf(v1) < INFINITY)) r1 = 0.0f;
    }
    const __half2 r = __floats2half2_rn(r0, r1);
    lo = *reinterpret_cast<const uint32_t*>(&r);
}
__device__ __forceinline__ void gm_ld32(uint32_t taddr, float (&d)[32]) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
        "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; ++i) d[i] = __uint_as_float(r[i]);
}

// ---------------------------------------------------------------------------------------------
// activations -> blocked, K-permuted layout
// ---------------------------------------------------------------------------------------------
// Position p of a 64-k stage is k = 64 kst + 32 (p / 32) + (p % 32) / 2 + 16 (p & 1): eight elements and the eight sixteen
// further on interleave into two 16-byte chunks.  One thread makes such a pair from two 16-byte loads; the 32 lanes of a
// warp are 8 rows x the 4 pairs of a stage, so that a warp reads whole 128-byte row segments and writes one whole 1 KB
// core-matrix block [kc (8)][row (8)][16 B].  (One chunk per thread, gathered with eight 2-byte loads, took 32 us at
// 2048 x 4096.)  Rows of Kin <= K elements are padded with zeros; rows that cannot be read in 16-byte pieces element by element.
__global__ void __launch_bounds__(256) gemm_retile_x_kernel(const __half* __restrict__ x, __half* __restrict__ xt, int M, int Kin,
                                                            int K, int NX, int MT) {
    pdl_launch_dependents();
    pdl_wait();
    const int KST = K / 64, RG = NX / 8;
    const int lane = threadIdx.x & 31, rr = lane & 7, pr = lane >> 3;     // row of the group; pair: k offset 32 (pr / 2) + 8 (pr % 2)
    const size_t blocks = (size_t)MT * KST * RG;                          // 1 KB blocks, in the order they lie in xt
    const bool vec = (Kin % 8 == 0) && ((reinterpret_cast<uintptr_t>(x) & 15) == 0);
    const int koff = 32 * (pr >> 1) + 8 * (pr & 1);
    for (size_t b = (size_t)blockIdx.x * 8 + (threadIdx.x >> 5); b < blocks; b += (size_t)gridDim.x * 8) {
        const int rg = (int)(b % RG);
        const size_t rest = b / RG;
        const int kst = (int)(rest % KST), mt = (int)(rest / KST);
        const int m = mt * NX + rg * 8 + rr;
        const int k = kst * 64 + koff;
        uint4 lo = make_uint4(0u, 0u, 0u, 0u), hi = lo;
        if (m < M) {
            const __half* row = x + (size_t)m * Kin;
            if (vec) {
                if (k < Kin) lo = __ldg(reinterpret_cast<const uint4*>(row + k));
                if (k + 16 < Kin) hi = __ldg(reinterpret_cast<const uint4*>(row + k + 16));
            } else {
                __align__(16) __half a[8], c[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    a[e] = (k + e < Kin) ? row[k + e] : __float2half(0.0f);
                    c[e] = (k + 16 + e < Kin) ? row[k + 16 + e] : __float2half(0.0f);
                }
                lo = *reinterpret_cast<const uint4*>(a), hi = *reinterpret_cast<const uint4*>(c);
            }
        }
        uint4* dst = reinterpret_cast<uint4*>(xt) + b * 64 + (size_t)(2 * pr) * 8 + rr;
        dst[0] = make_uint4(__byte_perm(lo.x, hi.x, 0x5410), __byte_perm(lo.x, hi.x, 0x7632), __byte_perm(lo.y, hi.y, 0x5410),
                            __byte_perm(lo.y, hi.y, 0x7632));
        dst[8] = make_uint4(__byte_perm(lo.z, hi.z, 0x5410), __byte_perm(lo.z, hi.z, 0x7632), __byte_perm(lo.w, hi.w, 0x5410),
                            __byte_perm(lo.w, hi.w, 0x7632));
    }
}

// ---------------------------------------------------------------------------------------------
// the GEMM
// ---------------------------------------------------------------------------------------------
// Split K: the sum of the KS parts of one output tile (rows activation rows x cols weight rows, row pitch N), in part order.
// A thread takes four neighbouring weight rows of U activation rows and loads Q parts of them together: one element and one part at a
// time was a chain of 64 x KS L2 round trips (71 -> 38 us at 512 x 4096 x 4096), one part at a time of few rows one of KS.
template <int U, int Q>
static __device__ __forceinline__ void gm_add_rows(const float* part, size_t plane, int KS, int rows, int cols, int N,
                                                   const __half* bias, __half* y, int tid) {
    constexpr int W = GM_DTHREADS / 32;
    const int c = (tid & 31) * 4;
    if (c >= cols) return;
    const bool quad = (N % 4 == 0) && c + 4 <= cols;
    float b[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) b[j] = (bias && c + j < cols) ? __half2float(bias[c + j]) : 0.0f;
    for (int m = tid >> 5; m < rows; m += U * W) {
        float v[U][4];
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int j = 0; j < 4; ++j) v[u][j] = 0.0f;
        for (int q0 = 0; q0 < KS; q0 += Q) {
            float t[Q][U][4];
#pragma unroll
            for (int q = 0; q < Q; ++q)
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    const int mu = m + u * W;
                    const bool on = mu < rows && q0 + q < KS;
                    const float* s = part + (size_t)(q0 + q) * plane + c + (size_t)mu * N;
                    if (on && quad) {
                        const float4 f = __ldcg(reinterpret_cast<const float4*>(s));
                        t[q][u][0] = f.x, t[q][u][1] = f.y, t[q][u][2] = f.z, t[q][u][3] = f.w;
                    } else {
#pragma unroll
                        for (int j = 0; j < 4; ++j) t[q][u][j] = (on && c + j < cols) ? __ldcg(s + j) : 0.0f;
                    }
                }
#pragma unroll
            for (int q = 0; q < Q; ++q)
#pragma unroll
                for (int u = 0; u < U; ++u)
#pragma unroll
                    for (int j = 0; j < 4; ++j) v[u][j] += t[q][u][j];
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int mu = m + u * W;
            if (mu >= rows) break;
            __half* dst = y + (size_t)mu * N + c;
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (c + j < cols) dst[j] = __float2half_rn(v[u][j] + b[j]);
        }
    }
}
static __device__ __forceinline__ void gm_add_parts(const float* part, size_t plane, int KS, int rows, int cols, int N,
                                                 const __half* bias, __half* y, int tid) {
    constexpr int W = GM_DTHREADS / 32;
    if (rows <= W) gm_add_rows<1, 4>(part, plane, KS, rows, cols, N, bias, y, tid);
    else if (rows <= 2 * W) gm_add_rows<2, 2>(part, plane, KS, rows, cols, N, bias, y, tid);
    else gm_add_rows<4, 1>(part, plane, KS, rows, cols, N, bias, y, tid);
}

// SPLIT: K is split over several CTAs (p.KS > 1).  A kernel of its own: its CTAs have one work item each (gm_plan), so that the
// epilogue, which needs the registers of the decoding loop, comes behind that loop and not inside it.
// EXACT: weights are formed in fp32 and multiplied in two fp16 parts (gm_two_parts), two MMAs per 16 k on the same activations, for
// the row counts that are no multiple of 128, which the CUDA-core kernel with its fp32 weights served before.  Formed in fp16 with
// one rounding per plane the weights gave errors of 3.1e-4 of the result (2-norm) where that kernel has 2.1e-4, the rounding of
// the result; so have two parts.  37 x 3000 x 3000, S = 3: 17 us (14 with fp16 weights, 70 on CUDA cores); 1000 x 3000 x 4096,
// S = 4: 62 us (37, 2 190).
template <int S, int NX, bool SPLIT, bool EXACT>
__global__ void __launch_bounds__(GM_THREADS, 1) linear_gemm_kernel(const GmParams p) {
    extern __shared__ __align__(1024) unsigned char smem[];
    constexpr int NX1 = NX == GM_WIDE ? 256 : NX;  // columns of the first MMA
    constexpr uint32_t IDESC = (1u << 4) | ((uint32_t)(NX1 >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
    constexpr int GM_SLOTS = gm_slots(NX, EXACT), GM_A_COL = gm_a_col(NX);
    constexpr int ACOLS = EXACT ? 64 : 32;         // tensor-memory columns of a decoded tile
    static_assert(GM_A_COL + GM_SLOTS * ACOLS <= GM_TMEM_COLS && NX <= GM_A_COL, "tensor memory");
    const int nx = NX == GM_WIDE ? p.nx : NX;
    const uint32_t STAGE_BYTES = (uint32_t)nx * 128u;
    const uint32_t idesc2 = (1u << 4) | ((uint32_t)((nx - NX1) >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);

    uint64_t* full = reinterpret_cast<uint64_t*>(smem);          // [GM_SLOTS] activation block landed and weight tile stored
    uint64_t* empty = full + GM_SLOTS;                           // [GM_SLOTS] both read by the stage's MMAs
    uint64_t* d_full = empty + GM_SLOTS;                         // [1] all MMAs of a work item done
    uint64_t* d_empty = d_full + 1;                              // [1] D read out
    volatile int* flags = reinterpret_cast<volatile int*>(d_empty + 1);     // [0] abort, [1] "last part" flag
    uint32_t* tmem_base_s = reinterpret_cast<uint32_t*>(smem + GM_HDR - 16);
    unsigned char* xs = smem + GM_HDR;                           // [GM_SLOTS][STAGE_BYTES]

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    pdl_launch_dependents();
    pdl_wait();                                    // the re-tiled activations come from the previous kernel
    if (threadIdx.x == 0) {
        for (int i = 0; i < GM_SLOTS; ++i) {
            mbar_init(&full[i], 5);                // the activation producer and four decoder warps
            mbar_init(&empty[i], 1);
        }
        mbar_init(d_full, 1);
        mbar_init(d_empty, GM_DWGS * 4);
        flags[0] = 0;
        flags[1] = 0;
        fence_mbar_init();
    }
    if (warp == GM_PWARP) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_base_s)),
                     "r"((uint32_t)GM_TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        gm_fence_before();
    }
    __syncthreads();
    gm_fence_after();
    const uint32_t tbase = *tmem_base_s;
    const int grid = (int)gridDim.x;
    const int SPP = p.SPP;

    if (warp == GM_PWARP) {
        // ------------------------------ activation producer ------------------------------
        if (lane == 0) {
            int it = 0;
            bool ok = true;
            for (int item = blockIdx.x; item < p.items && ok; item += grid) {
                const int kp = item % p.KS, mt = (item / p.KS) % p.MT;
                const unsigned char* src = reinterpret_cast<const unsigned char*>(p.xt) +
                                           ((size_t)mt * (p.K / 64) + (size_t)kp * SPP) * STAGE_BYTES;
                for (int ks = 0; ks < SPP; ++ks, ++it) {
                    const int st = it % GM_SLOTS;
                    const uint32_t ph = (uint32_t)(it / GM_SLOTS) & 1u;
                    if (flags[0] || !mbar_wait_async(&empty[st], ph ^ 1u)) {
                        ok = false;
                        break;
                    }
                    mbar_arrive_expect_tx(&full[st], STAGE_BYTES);
                    bulk_g2s(xs + (size_t)st * STAGE_BYTES, src + (size_t)ks * STAGE_BYTES, STAGE_BYTES, &full[st]);
                }
            }
            if (!ok) {
                flags[0] = 1;
                atomicExch(p.status, 1u);
                atomicExch(p.status + 1, 0x500u + blockIdx.x);
            }
        }
    } else if (warp == GM_IWARP) {
        // ------------------------------ MMA issuer ------------------------------
        // One barrier per stage says that both operands are in place, and the barrier of the next stage is read before
        // the MMAs of this one are issued, so that its latency runs beside them.
        const int total = (int)blockIdx.x < p.items ? ((p.items - 1 - (int)blockIdx.x) / grid + 1) * SPP : 0;
        bool ok = tbase == 0;                      // (an allocation of all columns can only start at column 0)
        if (elect_one()) {
            const uint32_t d0 = gm_bdesc_lo(smem_u32(xs)), dstep = STAGE_BYTES >> 4;
            int ks = 0;
            uint32_t ph = 0, dph = 1;              // dph: parity of the read-out of the item before
            bool rdy = mbar_test(&full[0], 0u);
            for (int it = 0; it < total && ok; it += GM_SLOTS, ph ^= 1u) {
#pragma unroll
                for (int slot = 0; slot < GM_SLOTS; ++slot) {
                    if (it + slot >= total) break;
                    if (ks == 0) {
                        if (it + slot > 0 && !mbar_wait_timed(d_empty, dph)) ok = false;       // D of the previous item must have been read out
                        dph ^= 1u;
                    }
                    if (!rdy) {                    // (spins: a warp parked by try_wait comes back later than the phase)
                        const long long t0 = clock64();
                        while (!mbar_test(&full[slot], ph))
                            if (clock64() - t0 > 2000000000LL) {
                                ok = false;
                                break;
                            }
                    }
                    if (!ok) break;
                    gm_fence_after();
                    rdy = mbar_test(&full[(slot + 1) % GM_SLOTS], slot + 1 == GM_SLOTS ? ph ^ 1u : ph);
                    const uint32_t d = d0 + (uint32_t)slot * dstep;
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const uint32_t acc = q ? 1u : (uint32_t)(ks != 0);
                        gm_mma(0, GM_A_COL + slot * ACOLS + q * 8, d + q * 16, IDESC, acc);
                        if (EXACT) gm_mma(0, GM_A_COL + slot * ACOLS + 32 + q * 8, d + q * 16, IDESC, 1u);
                        if (NX == GM_WIDE) gm_mma(NX1, GM_A_COL + slot * ACOLS + q * 8, d + NX1 * 8 + q * 16, idesc2, acc);
                    }
                    gm_commit(&empty[slot]);
                    if (++ks == SPP) {
                        gm_commit(d_full);
                        ks = 0;
                    }
                }
            }
        }
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) {
            flags[0] = 1;
            if (lane == 0) {
                atomicExch(p.status, 1u);
                atomicExch(p.status + 1, 0x600u + blockIdx.x);
            }
        }
    } else {
        // ------------------------------ decoder warpgroups ------------------------------
        const int wg = warp >> 2, wl = warp & 3;
        const int r = wl * 32 + lane;
        const int dtid = threadIdx.x;              // 0 .. 511
        const uint32_t lane_sel = (uint32_t)(wl * 32) << 16;
        const int N = p.N;
        bool dead = false;

        // The stages of all work items of this CTA form one sequence; this warpgroup takes every fourth one.
        struct Pos {
            int item, ks, it;
            int kst0, n;                           // first 64-k stage of the item's k part; this thread's weight row
        };
        auto set_item = [&](Pos& q) {              // the divisions happen once per work item, not per stage
            q.kst0 = (q.item % p.KS) * SPP;
            q.n = min((q.item / (p.KS * p.MT)) * 128 + r, p.N - 1);      // rows past the last one repeat it and are dropped
        };
        auto advance = [&](Pos& q, int by) {
            q.ks += by;
            q.it += by;
            if (q.ks >= SPP) {
                do {
                    q.ks -= SPP;
                    q.item += grid;
                } while (q.ks >= SPP);
                set_item(q);
            }
        };
        const int group_shift = (p.G == 256) ? 2 : 1;      // 64-k stages per coefficient group, as a shift
        auto load_words = [&](const Pos& q, uint32_t (&w)[2][S]) {
            if (q.item >= p.items) return;
            const uint32_t* src = p.bvr + ((size_t)(2 * (q.kst0 + q.ks)) * N + q.n) * S;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint32_t* g = src + (size_t)h * N * S;
                if constexpr (S == 4) {
                    const uint4 v = __ldg(reinterpret_cast<const uint4*>(g));
                    w[h][0] = v.x, w[h][1] = v.y, w[h][2] = v.z, w[h][3] = v.w;
                } else if constexpr (S == 2) {
                    const uint2 v = __ldg(reinterpret_cast<const uint2*>(g));
                    w[h][0] = v.x, w[h][1] = v.y;
                } else {
#pragma unroll
                    for (int s = 0; s < S; ++s) w[h][s] = __ldg(g + s);
                }
            }
        };
        // D of one finished work item -> y (or fp32 parts); every decoder warp takes part, also when dead.
        int ep_item = blockIdx.x, ep_seq = 0;
        auto epilogue = [&]() {
            const int item = ep_item;
            const int kp = item % p.KS, mt = (item / p.KS) % p.MT, nt = item / (p.KS * p.MT);
            const int n = nt * 128 + r;
            if (!dead && !mbar_wait_async(d_full, (uint32_t)ep_seq & 1u)) {
                dead = true;
                flags[0] = 1;
            }
            dead = __any_sync(0xffffffffu, dead);
            const int m0 = mt * nx;
            if (!dead) {
                gm_fence_after();
                const bool on = n < N;
                const float bias = (p.bias && !SPLIT && on) ? __half2float(p.bias[n]) : 0.0f;
                for (int c = wg; c < nx / 32; c += GM_DWGS) {
                    float d[32];
                    gm_ld32(tbase + lane_sel + c * 32, d);
                    if constexpr (!SPLIT) {
#pragma unroll
                        for (int i = 0; i < 32; ++i) {
                            const int m = m0 + c * 32 + i;
                            if (on && m < p.M) p.y[(size_t)m * N + n] = __float2half_rn(d[i] + bias);
                        }
                    } else {
                        float* dst = p.part + ((size_t)kp * p.MT * NX + m0 + c * 32) * N + n;
#pragma unroll
                        for (int i = 0; i < 32; ++i)
                            if (on) dst[(size_t)i * N] = d[i];
                    }
                }
                gm_fence_before();
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(d_empty);
            if constexpr (SPLIT) {
                // split K: the CTA that delivers the last part adds all parts in part order
                __threadfence();
                named_bar_sync(1, GM_DTHREADS);
                if (dtid == 0) {
                    const unsigned int tile = (unsigned int)(mt * p.NT + nt);
                    const unsigned int old = dead ? 0u : atomicAdd(p.counters + tile, 1u);
                    const int last = (!dead && old == (unsigned int)(p.KS - 1)) ? 1 : 0;
                    if (last) p.counters[tile] = 0u;           // ready for the next launch
                    flags[1] = last;
                }
                named_bar_sync(1, GM_DTHREADS);
                const bool last = flags[1] != 0;
                named_bar_sync(1, GM_DTHREADS);                // everyone has read the flag before it is rewritten
                if (last) {
                    __threadfence();
                    gm_add_parts(p.part + (size_t)m0 * N + nt * 128, (size_t)p.MT * NX * N, p.KS, min(NX, p.M - m0), min(128, N - nt * 128),
                                 N, p.bias ? p.bias + nt * 128 : nullptr, p.y + (size_t)m0 * N + nt * 128, dtid);
                }
            }
            ep_item += grid;
            ++ep_seq;
        };

        // Coefficients are fetched ahead as well: the line index of a stage two steps before its use, the
        // coefficient line itself one step before (it needs the index), so neither latency is exposed.
        auto line_of = [&](const Pos& q) -> uint32_t {
            if (q.item >= p.items) return 0u;
            const int g = (q.kst0 + q.ks) >> group_shift;
            const size_t e = (size_t)g * N + q.n;
            if (p.idx_bytes == 1) return __ldg(reinterpret_cast<const uint8_t*>(p.idx) + e);
            if (p.idx_bytes == 2) return __ldg(reinterpret_cast<const uint16_t*>(p.idx) + e);
            return (uint32_t)e;
        };
        auto load_coef = [&](const Pos& q, uint32_t line, unsigned short (&c)[S]) {
            if (q.item >= p.items) return;
            const unsigned short* src = reinterpret_cast<const unsigned short*>(p.coeff) + (size_t)line * S;
#pragma unroll
            for (int s = 0; s < S; ++s) c[s] = __ldg(src + s);
        };

        Pos cur{(int)blockIdx.x, 0, 0, 0, 0};
        set_item(cur);
        advance(cur, wg);
        Pos nxt = cur;
        advance(nxt, GM_DWGS);
        Pos nn = nxt;
        advance(nn, GM_DWGS);
        uint32_t w0[2][S], w1[2][S];               // packed words of `cur` and `nxt`: loads run one stage ahead
        unsigned short c0[S], c1[S];               // their coefficient lines (fp16 bits)
        load_words(cur, w0);
        load_words(nxt, w1);
        {
            const uint32_t lc = line_of(cur), ln = line_of(nxt);
            load_coef(cur, lc, c0);
            load_coef(nxt, ln, c1);
        }
        uint32_t l_nn = line_of(nn);

        auto decode_stage = [&](const Pos& q, const uint32_t (&w)[2][S], const unsigned short (&c)[S]) {
            if constexpr (!SPLIT)                  // (a CTA of a split problem has one item)
                while (ep_item < q.item) epilogue();   // items whose stages have all been handed to the issuer
            const int slot = q.it % GM_SLOTS;
            // false: a wait ran out here or elsewhere
            auto slot_free = [&]() -> bool {
                if (!dead && !mbar_wait_async(&empty[slot], ((uint32_t)(q.it / GM_SLOTS) & 1u) ^ 1u)) {
                    dead = true;
                    flags[0] = 1;
                }
                dead = __any_sync(0xffffffffu, dead);
                if (!dead) gm_fence_after();
                return !dead;
            };
            auto hand_over = [&]() {
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                gm_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&full[slot]);
            };
            if constexpr (EXACT) {
                float cf[S];
                bool odd = false;
#pragma unroll
                for (int s = 0; s < S; ++s) {
                    cf[s] = __half2float(__ushort_as_half(c[s]));
                    odd |= !(fabsf(cf[s]) < INFINITY);
                }
                odd = __any_sync(0xffffffffu, odd);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    uint32_t hi[16], lo[16];
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        float v0 = 0.0f, v1 = 0.0f;
#pragma unroll
                        for (int s = 0; s < S; ++s) {
                            if (w[h][s] & (1u << j)) v0 += cf[s];
                            if (w[h][s] & (0x10000u << j)) v1 += cf[s];
                        }
                        gm_two_parts(v0, v1, odd, hi[j], lo[j]);
                    }
                    if (h == 0 && !slot_free()) return;
                    gm_st16(tbase + lane_sel + GM_A_COL + slot * ACOLS + h * 16, hi);
                    gm_st16(tbase + lane_sel + GM_A_COL + slot * ACOLS + 32 + h * 16, lo);
                }
                hand_over();
                return;
            }
            // A lone bit at position 10 .. 14 of a half is the number 2^-14, 2^-13, 2^-11, 2^-7, 2^1: masking a packed
            // word with 0x04000400 << i leaves (bit, bit + 16) as such a half2, and one HFMA2 with c_s divided by that
            // number adds c_s where the bit is set.  Three shifted copies of the word bring all 16 bit pairs into the
            // window, so an element pair costs one mask and one HFMA2 per plane (the integer pipe, half as wide as the
            // fp16 pipe, was this kernel's limit with a shift and a mask-xor per pair).  |c_s| >= 4 would overflow the
            // largest multiplier: such a row takes the sign-flip form below instead.
            bool big = false;
            __half2 mul[S][5];
#pragma unroll
            for (int s = 0; s < S; ++s) {
                const __half ch = __ushort_as_half(c[s]);
                big |= !(__habs(ch) < __float2half_rn(3.9f));
                const __half2 c2 = __half2half2(ch);
                mul[s][0] = __hmul2(c2, __float2half2_rn(16384.0f));
                mul[s][1] = __hmul2(c2, __float2half2_rn(8192.0f));
                mul[s][2] = __hmul2(c2, __float2half2_rn(2048.0f));
                mul[s][3] = __hmul2(c2, __float2half2_rn(128.0f));
                mul[s][4] = __hmul2(c2, __float2half2_rn(0.5f));
            }
            uint32_t a[32];
            if (!__any_sync(0xffffffffu, big)) {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    __half2 acc[16];
#pragma unroll
                    for (int j = 0; j < 16; ++j) acc[j] = __float2half2_rn(0.0f);
#pragma unroll
                    for (int s = 0; s < S; ++s) {
                        // window copies: bits 0..4 / 5..9 / 10..14 / 15 of each half at positions 10..14 / 10..14 / 10..14 / 14
                        const uint32_t v0 = w[h][s] << 10, v1 = w[h][s] << 5, v2 = w[h][s], v3 = w[h][s] >> 1;
#pragma unroll
                        for (int j = 0; j < 16; ++j) {
                            const uint32_t v = (j < 5) ? v0 : (j < 10) ? v1 : (j < 15) ? v2 : v3;
                            const int pos = (j < 15) ? j % 5 : 4;
                            const uint32_t t = v & (0x04000400u << pos);
                            acc[j] = __hfma2(*reinterpret_cast<const __half2*>(&t), mul[s][pos], acc[j]);
                        }
                    }
#pragma unroll
                    for (int j = 0; j < 16; ++j) a[16 * h + j] = *reinterpret_cast<const uint32_t*>(&acc[j]);
                }
            } else {
                uint32_t hc[S];                    // (c_s / 2, c_s / 2)
                float sum = 0.0f;
#pragma unroll
                for (int s = 0; s < S; ++s) {
                    const float chf = __half2float(__ushort_as_half(c[s])) * 0.5f;
                    sum += chf;
                    const uint32_t hb = (uint32_t)__half_as_ushort(__float2half_rn(chf));
                    hc[s] = hb | (hb << 16);
                }
                const uint32_t bb = (uint32_t)__half_as_ushort(__float2half_rn(sum));
                const uint32_t base2 = bb | (bb << 16);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        __half2 acc = *reinterpret_cast<const __half2*>(&base2);
#pragma unroll
                        for (int s = 0; s < S; ++s) {
                            const uint32_t v = w[h][s] << (15 - j);
                            const uint32_t t = (~v & 0x80008000u) ^ hc[s];
                            acc = __hadd2(acc, *reinterpret_cast<const __half2*>(&t));
                        }
                        a[16 * h + j] = *reinterpret_cast<const uint32_t*>(&acc);
                    }
                }
            }
            // the slot is waited for with the values in registers: the decode runs beside the MMAs that still read the slot
            if (!slot_free()) return;
            gm_st32(tbase + lane_sel + GM_A_COL + slot * ACOLS, a);
            hand_over();
        };

        while (cur.item < p.items) {
            decode_stage(cur, w0, c0);
            cur = nxt, nxt = nn;
            advance(nn, GM_DWGS);
            {
                const uint32_t ln = l_nn;          // index of the new look-ahead stage, loaded a step ago
                l_nn = line_of(nn);
                load_words(nxt, w0);               // the set just used is free: it becomes the look-ahead set
                load_coef(nxt, ln, c0);
            }
            if (cur.item >= p.items) break;
            decode_stage(cur, w1, c1);
            cur = nxt, nxt = nn;
            advance(nn, GM_DWGS);
            {
                const uint32_t ln = l_nn;
                l_nn = line_of(nn);
                load_words(nxt, w1);
                load_coef(nxt, ln, c1);
            }
        }
        while (ep_item < p.items) epilogue();

        if (dead) {
            flags[0] = 1;
            if (lane == 0) {
                atomicExch(p.status, 1u);
                atomicExch(p.status + 1, 0x400u + blockIdx.x);
            }
        }
    }
    // ------------------------------ teardown ------------------------------
    gm_fence_before();
    __syncthreads();
    gm_fence_after();
    if (warp == GM_PWARP)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tbase), "r"((uint32_t)GM_TMEM_COLS)
                     : "memory");
}

// ---------------------------------------------------------------------------------------------
// host
// ---------------------------------------------------------------------------------------------
struct GmPlan {
    int NX, MT, NT, KS, SPP, items, grid, smem;
    bool exact;
    size_t xt_bytes, part_bytes;
};

// Activation rows of a tile.  More than 256 rows: the width with the least work on the busiest SM, whole rounds of tiles times the
// time of a 64-k stage.  A stage of a 256-row tile waits for the decoders (the more planes the longer), one of a wider tile for
// its MMAs; measured per stage at 2048 x 14336 x 4096, in cycles: 850 (S = 4), about 730 (S = 2) at 256 rows, 3 per row for wider
// tiles (a second, small MMA costs more than its share of the columns).  Wide tiles win where they save rounds: 232 -> 210 us at
// 2048 x 14336 x 4096 (7 rounds -> 5 of 352 rows), 350 -> 302 us at 3000 x 4096 x 14336 (3 -> 2), 78 -> 59 us at 1500 x 4096 x
// 4096 (2 -> 1 of 384 rows); 2048 x 4096 stays at 256 rows (2 rounds either way).  Problems that do not fill the GPU at 256 rows
// split K instead.
// Two-part weights fill the tensor memory of wide tiles: 256 rows at most, 64 at least (one instantiation less).
static int gm_nx(int M, int NT, int S, int sm_count, bool exact) {
    if (M <= 256 || exact) return (M <= 32 && !exact) ? 32 : M <= 64 ? 64 : M <= 128 ? 128 : 256;
    int best = 256;
    long long cost = 0;
    for (int nx = 256; nx <= GM_WIDE; nx += 32) {
        const long long items = (long long)NT * ((M + nx - 1) / nx);
        if (nx == 256 && items < sm_count) break;
        const long long c = (items + sm_count - 1) / sm_count * (nx == 256 ? 610 + 60 * S : 3 * nx);
        if (nx == 256 || c < cost) best = nx, cost = c;
    }
    return best;
}

bool linear_gemm_supported(const PackedW& w, int M) {
    if (w.S < 2 || w.S > 4) return false;
    if (w.G != 256 && w.G != 128) return false;
    if (M < 1) return false;
    if (w.K % 64) return false;
    if (w.idx_bytes < 0 || w.idx_bytes > 2) return false;
    if (w.S != 3 && (reinterpret_cast<uintptr_t>(w.bvr) & (w.S * 4 - 1))) return false;   // vector loads of a row's planes
    return true;
}

static void gm_plan(const PackedW& w, int M, int sm_count, GmPlan* pl) {
    pl->NT = (w.N + 127) / 128;
    pl->exact = w.N % 128 != 0;
    pl->NX = gm_nx(M, pl->NT, w.S, sm_count, pl->exact);
    pl->MT = (M + pl->NX - 1) / pl->NX;
    const int KST = w.K / 64;
    int ks = 1;
    const int tiles = pl->NT * pl->MT;
    if (pl->NX <= 256 && tiles < sm_count && tiles <= SBVR_WS_COUNTERS) {
        // split K so that more SMs work, keeping at least 4 stages per part
        for (int cand = 2; cand <= KST / 4; ++cand) {
            if (KST % cand) continue;
            if (tiles * cand > sm_count) break;
            ks = cand;
        }
    }
    pl->KS = ks;
    pl->SPP = KST / ks;
    pl->items = tiles * ks;
    pl->grid = pl->items < sm_count ? pl->items : sm_count;
    pl->smem = GM_HDR + gm_slots(pl->NX > 256 ? GM_WIDE : pl->NX, pl->exact) * pl->NX * 128;
    pl->xt_bytes = ((size_t)pl->MT * pl->NX * w.K * 2 + 255) / 256 * 256;
    pl->part_bytes = ks > 1 ? (size_t)ks * pl->MT * pl->NX * w.N * 4 : 0;
}

// Estimate of a call's time in ns for more than 256 rows, to choose between this kernel and the one over CTA pairs: rounds of tiles at
// the stage times of gm_nx and 9 000 cycles for a tile's end, at 1.9 GHz; re-tiling; the parts of a split K (16.8 MB of them took
// about 10 us).  Measured and estimated, us: 2048 x 14336 x 4096 209, 209; 512 x 8192 x 8192 67, 67; 1024 x 4096 x 4096 38, 38; 300 x
// 14336 x 4096 41.5, 41; 3000 x 4096 x 14336 303, 307; 2048 x 1024 x 4096 37, 36.
static long long gm_ns(const PackedW& w, const GmPlan& pl, int sm_count) {
    const long long rounds = (pl.items + sm_count - 1) / sm_count;
    const long long cycles = rounds * ((long long)pl.SPP * (pl.NX == 256 ? 610 + 60 * w.S : 3 * pl.NX) + 9000) +
                             (long long)(pl.xt_bytes / 2000) + (long long)(pl.part_bytes / 900) + 6000;
    return cycles * 10 / 19;
}

size_t linear_gemm_workspace_bytes(const PackedW& w, int M, int sm_count) {
    GmPlan pl;
    gm_plan(w, M, sm_count, &pl);
    return pl.xt_bytes + pl.part_bytes;
}

void linear_gemm_split(const PackedW& w, int M, int sm_count, int* parts, int* stages) {
    GmPlan pl;
    gm_plan(w, M, sm_count, &pl);
    *parts = pl.KS, *stages = pl.SPP * ((pl.items + sm_count - 1) / sm_count);
}

template <int S, int NX, bool SPLIT, bool EXACT>
static int gm_launch_split(const GmParams& p, int grid, int smem, cudaStream_t st) {
    static SmemOnce once;
    const int rc = set_max_smem_once(once, linear_gemm_kernel<S, NX, SPLIT, EXACT>, 227 * 1024);
    if (rc) return rc;
    SBVR_CUDA_TRY(launch_pdl(linear_gemm_kernel<S, NX, SPLIT, EXACT>, dim3(grid), dim3(GM_THREADS), (size_t)smem, st, p));
    return SBVR_OK;
}
template <int S, int NX, bool EXACT = false>
static int gm_launch_inst(const GmParams& p, int grid, int smem, cudaStream_t st) {
    return p.KS > 1 ? gm_launch_split<S, NX, true, EXACT>(p, grid, smem, st) : gm_launch_split<S, NX, false, EXACT>(p, grid, smem, st);
}
template <int S>
static int gm_launch_nx(const GmParams& p, const GmPlan& pl, cudaStream_t st) {
    if (pl.exact) switch (pl.NX) {
        case 64: return gm_launch_inst<S, 64, true>(p, pl.grid, pl.smem, st);
        case 128: return gm_launch_inst<S, 128, true>(p, pl.grid, pl.smem, st);
        default: return gm_launch_inst<S, 256, true>(p, pl.grid, pl.smem, st);
    }
    switch (pl.NX) {
        case 32: return gm_launch_inst<S, 32>(p, pl.grid, pl.smem, st);
        case 64: return gm_launch_inst<S, 64>(p, pl.grid, pl.smem, st);
        case 128: return gm_launch_inst<S, 128>(p, pl.grid, pl.smem, st);
        case 256: return gm_launch_inst<S, 256>(p, pl.grid, pl.smem, st);
        default: return gm_launch_split<S, GM_WIDE, false, false>(p, pl.grid, pl.smem, st);
    }
}

int launch_linear_gemm(const __half* x, int Kin, const PackedW& w, const __half* bias, __half* y, int M, const sbvr_workspace* ws,
                       cudaStream_t st) {
    if (!linear_gemm_supported(w, M)) return SBVR_ERR_UNSUPPORTED;
    if (!ws) return SBVR_ERR_WORKSPACE;
    DeviceInfo di;
    int rc = device_info(ws->device, &di);
    if (rc) return rc;
    if (di.cc_major != 10) return SBVR_ERR_UNSUPPORTED;
    GmPlan pl;
    gm_plan(w, M, di.sm_count, &pl);
    if (pl.xt_bytes + pl.part_bytes > ws->dyn_bytes) return SBVR_ERR_WORKSPACE;
    if (linear_pair_supported(x, Kin, w, y, M) &&
        linear_pair_ns(w, M, di.sm_count, ws->device, ws->dyn_bytes) < gm_ns(w, pl, di.sm_count))
        return launch_linear_pair(x, Kin, w, bias, y, M, ws->status, ws->dyn, ws->dyn_bytes, di.sm_count, ws->device, st);
    __half* xt = reinterpret_cast<__half*>(ws->dyn);
    {
        const size_t nblk = ((size_t)pl.MT * pl.NX / 8 * (w.K / 64) + 7) / 8;
        const int blocks = (int)(nblk < (size_t)di.sm_count * 16 ? nblk : (size_t)di.sm_count * 16);
        SBVR_CUDA_TRY(launch_pdl(gemm_retile_x_kernel, dim3(blocks), dim3(256), 0, st, x, xt, M, Kin, w.K, pl.NX, pl.MT));
    }
    GmParams p;
    p.xt = xt, p.bvr = w.bvr, p.idx = w.idx, p.coeff = w.coeff, p.bias = bias, p.y = y;
    p.part = reinterpret_cast<float*>(ws->dyn + pl.xt_bytes);
    p.counters = ws->counters, p.status = ws->status;
    p.M = M, p.N = w.N, p.K = w.K, p.C = w.C, p.G = w.G, p.idx_bytes = w.idx_bytes, p.nx = pl.NX;
    p.NT = pl.NT, p.MT = pl.MT, p.KS = pl.KS, p.SPP = pl.SPP, p.items = pl.items;
    switch (w.S) {
        case 2: return gm_launch_nx<2>(p, pl, st);
        case 3: return gm_launch_nx<3>(p, pl, st);
        default: return gm_launch_nx<4>(p, pl, st);
    }
}

}  // namespace sbvr
