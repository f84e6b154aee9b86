// SBVR linear for more than a few activation rows (batches and prefill): a tcgen05 fp16 GEMM whose
// weight operand is dequantised inside the kernel and never exists in memory.
//
//   y[m, n] = sum_k x[m, k] * W[n, k] (+ bias[n]),   W[n, k] = sum_s c[k/G, n, s] * bit_s[n, k]
//
// Operands of tcgen05.mma kind::f16 (fp32 accumulation in tensor memory), D[128 weight rows, 32 .. 384 activation rows]:
//
//  A (weights, from tensor memory)  Decoder thread r of a warpgroup owns weight row r of the tile.  Per 64 k it
//      turns its 2 x S packed words into 64 fp16 values and stores them to its tensor-memory lane
//      (tcgen05.st): decoded weights never touch shared or global memory.  The value of an element is the sum of
//      the c_s whose plane bit is set, formed two elements at a time in half2: a lone bit at position 10 .. 14 of a
//      half is a power of two, so `word & (0x04000400 << i)` is (2^e * bit_j, 2^e * bit_{j+16}) and one HFMA2 with
//      c_s / 2^e adds c_s where the bits are set: a mask and an HFMA2 per plane per pair of elements, plus three
//      shifted copies per word (rows with |c_s| >= 3.9 use sign flips around sum_s c_s / 2 instead: shift, LOP3,
//      HADD2).  One byte permute per pair brings the elements into their natural order.
//  B (activations, from shared memory)  TMA boxes of those rows x 64 k straight from x (128-byte swizzle); rows and columns past the end
//      are filled with zeros by the copy.  Rows that do not start on 16 bytes are copied into such first.
//
// Replaces `x @ decode().T` of the reference's Llama flow for prefill (reference sbvr_utils/utils_llama.py:147,
// sbvr/core.py:926-949) and the M > 1 use of `_sbvr_row_deq_mm_T` (sbvr/kernels/sbvr_kernel.cu:121-191).
// Accuracy: weights are formed in fp16 with one rounding per plane (not the single rounding of decode()), which
// perturbs a weight by at most a few fp16 ulps of its partial sums; products accumulate in fp32.
//
// Structure: persistent CTAs of 20 warps.  Warps 0-15 are four decoder warpgroups, one for each 64-k stage of a window of 256 k; when
// the MMAs of a tile (or of a CTA's part of one) have finished they read D from tensor memory, add the bias and write fp16, or fp32 sums
// where several CTAs share the tile (a second, small kernel adds them in the order of K).  Warp 16 issues the MMAs from one elected lane,
// warp 17 fetches activations, warps 18 and 19 packed words and coefficient lines, a window each in turn.  The work is split by windows
// (TsSegs): whole tiles, and the tiles that are left over cut into equal runs of windows.  Every wait is bounded; on a time-out the kernel
// records it in the status word, skips the remaining work without skipping a barrier, frees its tensor memory and returns.
//
// What bounds it: up to 128 rows the decoders' integer pipe, about 200 half-rate instructions per thread and stage, 480 cycles with four
// warps per scheduler (850 when they loaded words and lines themselves, a stage ahead); with more rows the MMAs, 520 for 256.  Around that,
// per call, 1.5 us until a CTA has set itself up, 2 until its first words and coefficients are there, 2 for the last tile; and 3 to 5
// where sums of parts of K are added by the second launch.  S = 4, us (and when activations were re-tiled by a kernel in front, K was split
// evenly and the last CTA added the parts): 64 x 14336 x 4096 27.0 (34.3), 64 x 4096 x 14336 28.6 (36.1), 64 x 4096 x 4096 16.7 (17.8),
// 64 x 1024 x 4096 11.7 (17.8), 256 x 14336 x 4096 31.7 (40.3), 256 x 4096 x 4096 24.1 (32.3), 256 x 1024 x 4096 17.2 (48.5), 300 x 4096 x
// 14336 40.3 (68.2), 1024 x 4096 x 4096 32.4 (37.9); two parts: 37 x 3000 x 3000, S = 3, 14.3 (17.7), 200 x 3001 x 4096 27.7 (44.7).
#include <algorithm>

#include "tc_stream.cuh"

namespace sbvr {

constexpr int GM_DWGS = 4;
constexpr int GM_IWARP = GM_DWGS * 4;              // MMA issuer
constexpr int GM_XWARP = GM_IWARP + 1;             // fetches activations
constexpr int GM_PWARP = GM_XWARP + 1;             // first of two that fetch packed words and coefficient lines
constexpr int GM_THREADS = (GM_PWARP + 2) * 32;
constexpr int GM_TMEM_COLS = 512;
// Ring of 64-k stages: a decoded 128 x 64 weight tile in tensor memory and the activations in shared memory; ring of windows: packed words
// of 128 rows x 256 k, and the coefficients (four halves) of a row for one or two groups.
constexpr int GM_WIDE = 384;                       // variant for tiles of 288 .. 384 activation rows (GmParams::nx, multiples of 32)
__host__ __device__ constexpr int gm_slots(int NX, bool EXACT) { return EXACT || NX == GM_WIDE ? 4 : NX == 256 ? 5 : 6; }
__host__ __device__ constexpr int gm_windows(int NX, bool EXACT) { return NX >= 256 && !EXACT ? 2 : 4; }
__host__ __device__ constexpr int gm_word_bytes(int S) { return 8 * 128 * S * 4; }
__host__ __device__ constexpr int gm_coef_bytes(int G) { return 256 / G * 128 * 8; }
__host__ __device__ constexpr int gm_a_col(int NX) { return NX == GM_WIDE ? 384 : 256; }       // D occupies columns [0, nx), the A ring is behind
constexpr int GM_HDR = 1024, GM_SMEM_MAX = 227 * 1024;
__host__ __device__ constexpr int gm_smem_with(int NX, int nx, bool EXACT, int S, int G, int coefs) {
    return GM_HDR + gm_slots(NX, EXACT) * nx * 128 + gm_windows(NX, EXACT) * gm_word_bytes(S) + coefs * gm_coef_bytes(G);
}
// Windows whose coefficients have a place: all of the ring, or where those do not fit (384 rows, four planes, groups of 128: 2 KB over) one,
// filled when the decoders have taken the window before (384 x 28672 x 8192: 166 us in tiles that leave room for two, 151 so).
__host__ __device__ constexpr int gm_coef_windows(int NX, int nx, bool EXACT, int S, int G) {
    return NX == GM_WIDE && gm_smem_with(NX, nx, EXACT, S, G, gm_windows(NX, EXACT)) > GM_SMEM_MAX ? 1 : gm_windows(NX, EXACT);
}
__host__ __device__ constexpr int gm_smem(int NX, int nx, bool EXACT, int S, int G) {
    return gm_smem_with(NX, nx, EXACT, S, G, gm_coef_windows(NX, nx, EXACT, S, G));
}
static_assert(gm_smem(256, 256, false, 4, 128) <= GM_SMEM_MAX && gm_smem(256, 256, true, 4, 128) <= GM_SMEM_MAX &&
              gm_smem(GM_WIDE, 384, false, 4, 256) <= GM_SMEM_MAX && gm_smem(GM_WIDE, 384, false, 4, 128) <= GM_SMEM_MAX, "shared memory");

struct GmParams {
    const uint32_t* bvr;
    const void* idx;
    const __half* coeff;
    const __half* bias;
    __half* y;
    float* part;                 // [CTA + left-over tile][nx][128] fp32 sums of tiles that several CTAs share
    unsigned int* status;
    int M, N, K, G, idx_bytes;
    int vec;                     // lines of S = 4 (2) can be read as 8 (4) bytes
    int nx;                      // activation rows of a tile
    int MT, tiles, KBS;          // activation-row tiles, tiles, windows of a tile
    int whole;                   // tiles are not split
};

__device__ __forceinline__ void gm_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void gm_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// B descriptor: K-major, 128-byte swizzle, 1024 B between 8-row groups; version 1.  Its upper word is a constant; the lower one moves by
// (bytes >> 4).
__device__ __forceinline__ uint32_t gm_bdesc_lo(uint32_t saddr) { return (saddr >> 4) | (1u << 16); }
__device__ __forceinline__ void gm_mma(uint32_t d_t, uint32_t a_t, uint32_t bdesc_lo, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 d;\n\tsetp.ne.b32 p, %4, 0;\n\tmov.b64 d, {%2, %5};\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], d, %3, p;\n\t}" ::"r"(d_t),
        "r"(a_t), "r"(bdesc_lo), "r"(idesc), "r"(accumulate), "r"((1024u >> 4) | (1u << 14) | (2u << 29))
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
// the GEMM
// ---------------------------------------------------------------------------------------------
// A CTA's work: its runs of windows of the left-over tiles first, then its own tiles.
struct GmSegs {
    TsSegs sg;
    int KBS, cta;
    bool whole;
    __device__ __forceinline__ GmSegs(const GmParams& p) : KBS(p.KBS), cta((int)blockIdx.x), whole(p.whole != 0) {
        sg.init(p.tiles, whole ? 1 : KBS, gridDim.x, blockIdx.x);
    }
    __device__ __forceinline__ int k0(int q) const { return whole ? 0 : sg.k0(q); }
    __device__ __forceinline__ int k1(int q) const { return whole ? KBS : sg.k1(q); }
};

// EXACT: weights are formed in fp32 and multiplied in two fp16 parts (gm_two_parts), two MMAs per 16 k on the same activations, for
// the row counts that are no multiple of 128, which the CUDA-core kernel with its fp32 weights served before.  Formed in fp16 with
// one rounding per plane the weights gave errors of 3.1e-4 of the result (2-norm) where that kernel has 2.1e-4, the rounding of
// the result; so have two parts.
template <int S, int NX, bool EXACT>
__global__ void __launch_bounds__(GM_THREADS, 1) linear_gemm_kernel(const __grid_constant__ CUtensorMap xmap, const GmParams p) {
    extern __shared__ __align__(1024) unsigned char smem[];
    constexpr int BOXES = NX == GM_WIDE ? 2 : 1;   // an MMA has at most 256 columns, a box 256 rows
    const int nx = NX == GM_WIDE ? p.nx : NX, box = nx / BOXES;
    const uint32_t idesc = (1u << 4) | ((uint32_t)(box >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
    constexpr int SLOTS = gm_slots(NX, EXACT), WINDOWS = gm_windows(NX, EXACT);
    constexpr int ACOLS = EXACT ? 64 : 32;         // tensor-memory columns of a decoded tile
    constexpr int A_COL = gm_a_col(NX);
    constexpr uint32_t word_bytes = gm_word_bytes(S);
    const uint32_t stage_bytes = (uint32_t)nx * 128, coef_bytes = gm_coef_bytes(p.G);
    const bool one_coef = NX == GM_WIDE && gm_coef_windows(NX, nx, EXACT, S, p.G) == 1;
    static_assert(A_COL + SLOTS * ACOLS <= GM_TMEM_COLS && NX <= A_COL, "tensor memory");

    uint64_t* full = reinterpret_cast<uint64_t*>(smem);          // [SLOTS] activations landed and weight tile stored
    uint64_t* empty = full + SLOTS;                              // [SLOTS] both read by the stage's MMAs
    uint64_t* d_full = empty + SLOTS;                            // [1] all MMAs of a segment done
    uint64_t* d_empty = d_full + 1;                              // [1] D read out
    uint64_t* p_full = d_empty + 1;                              // [WINDOWS] packed words and coefficients landed
    uint64_t* p_empty = p_full + WINDOWS;                        // [WINDOWS] read by the decoders
    volatile int* flags = reinterpret_cast<volatile int*>(p_empty + WINDOWS);      // [0] abort
    uint32_t* tmem_base_s = reinterpret_cast<uint32_t*>(smem + GM_HDR - 16);
    unsigned char* xs = smem + GM_HDR;                           // [SLOTS][stage_bytes]
    unsigned char* ps = xs + SLOTS * stage_bytes;                // [WINDOWS][word_bytes]
    unsigned char* cs = ps + WINDOWS * word_bytes;               // [WINDOWS, or one][coef_bytes]

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    pdl_launch_dependents();
    const GmSegs segs(p);
    const TsSegs& sg = segs.sg;
    const int KBS = p.KBS, N = p.N;
    const int tail = (p.K & 255) ? 2 : 4;          // stages of a tile's last window
    auto stages_of = [&](int kb) { return kb == KBS - 1 ? tail : 4; };
    auto seg_stages = [&](int q) { return (segs.k1(q) - segs.k0(q)) * 4 - (segs.k1(q) == KBS ? 4 - tail : 0); };

    // What the two fetching warps work with; they ask for their first window before anything else.
    const int sets = p.G == 128 ? 2 : 1, groups = p.K / p.G;
    struct Pos {
        int q, kb, k1, n;                          // segment, window, end of its windows, this lane's first row
    };
    auto set_seg = [&](Pos& a) {
        if (a.q >= sg.nseg) return;
        a.kb = segs.k0(a.q), a.k1 = segs.k1(a.q), a.n = sg.tile(a.q) / p.MT * 128 + lane;
    };
    auto next = [&](Pos& a) {
        if (a.q < sg.nseg && ++a.kb >= a.k1) {
            ++a.q;
            set_seg(a);
        }
    };
    auto row = [&](const Pos& a, int i) { return min(a.n + 32 * i, N - 1); };                  // rows past the last one repeat it and are dropped
    auto lines_of = [&](const Pos& a, uint32_t (&l)[2][4]) {
        if (a.q >= sg.nseg) return;
#pragma unroll
        for (int t = 0; t < 2; ++t) {
            if (t >= sets) break;
            const size_t g = (size_t)min(a.kb * sets + t, groups - 1) * N;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const size_t e = g + row(a, i);
                if (p.idx_bytes == 1) l[t][i] = __ldg(reinterpret_cast<const uint8_t*>(p.idx) + e);
                else if (p.idx_bytes == 2) l[t][i] = __ldg(reinterpret_cast<const uint16_t*>(p.idx) + e);
                else l[t][i] = (uint32_t)e;
            }
        }
    };
    auto load_coef = [&](const Pos& a, const uint32_t (&l)[2][4], uint2 (&c)[2][4]) {
#pragma unroll
        for (int t = 0; t < 2; ++t)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                c[t][i] = make_uint2(0u, 0u);
                if (t >= sets || a.q >= sg.nseg) continue;
                const unsigned short* src = reinterpret_cast<const unsigned short*>(p.coeff) + (size_t)l[t][i] * S;
                if (S == 4 && p.vec) c[t][i] = __ldg(reinterpret_cast<const uint2*>(src));
                else if (S == 2 && p.vec) c[t][i].x = __ldg(reinterpret_cast<const uint32_t*>(src));
                else {
                    c[t][i].x = __ldg(src) | ((uint32_t)__ldg(src + 1) << 16);
                    if (S > 2) c[t][i].y = __ldg(src + 2);
                    if (S > 3) c[t][i].y |= (uint32_t)__ldg(src + 3) << 16;
                }
            }
    };
    auto copy_words = [&](const Pos& a, int slot) {
        const uint32_t dst = smem_u32(ps) + slot * word_bytes + (uint32_t)(lane * S * 4);
        const int runs = 2 * stages_of(a.kb);
        const uint32_t* src[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) src[i] = p.bvr + ((size_t)a.kb * 8 * N + row(a, i)) * S;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            if (k >= runs) break;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint32_t d = dst + (uint32_t)((k * 128 + 32 * i) * S * 4);
                if constexpr (S == 4) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src[i]) : "memory");
                else if constexpr (S == 2) asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src[i]) : "memory");
                else
#pragma unroll
                    for (int s = 0; s < S; ++s) asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d + 4 * s), "l"(src[i] + s) : "memory");
                src[i] += (size_t)N * S;
            }
        }
    };
    Pos win{0, 0, 0, 0};                           // the window at hand: its coefficients in coef, the line numbers of the one after in lines
    uint2 coef[2][4];
    uint32_t lines[2][4] = {};
    bool first_words = true;
    if (warp >= GM_PWARP) {
        set_seg(win);
        if (warp != GM_PWARP) next(win);
        lines_of(win, lines);
        if (win.q < sg.nseg) copy_words(win, warp - GM_PWARP);
        load_coef(win, lines, coef);               // (the line numbers have come meanwhile)
        Pos ahead = win;
        next(ahead), next(ahead);
        lines_of(ahead, lines);
    }
    if (threadIdx.x == 0) {
        for (int i = 0; i < SLOTS; ++i) {
            mbar_init(&full[i], 5);                // the activation producer and four decoder warps
            mbar_init(&empty[i], 1);
        }
        mbar_init(d_full, 1);
        mbar_init(d_empty, GM_DWGS * 4);
        for (int i = 0; i < WINDOWS; ++i) {
            mbar_init(&p_full[i], 33);             // every lane's copies, and its coefficients
            mbar_init(&p_empty[i], GM_DWGS * 4);
        }
        flags[0] = 0;
        fence_mbar_init();
    }
    if (warp == GM_XWARP) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_base_s)),
                     "r"((uint32_t)GM_TMEM_COLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        gm_fence_before();
    }
    __syncthreads();
    gm_fence_after();
    const uint32_t tbase = *tmem_base_s;

    if (warp == GM_XWARP) {
        // ------------------------------ activation producer ------------------------------
        if (lane == 0) {
            pdl_wait();                            // x comes from the previous kernel
            int slot = 0;
            uint32_t ph = 1;
            bool ok = true;
            for (int q = 0; q < sg.nseg && ok; ++q) {
                const int m = sg.tile(q) % p.MT * nx, s0 = segs.k0(q) * 4, s1 = s0 + seg_stages(q);
                for (int s = s0; s < s1; ++s) {
                    if (flags[0] || !mbar_wait_async(&empty[slot], ph)) {
                        ok = false;
                        break;
                    }
                    mbar_arrive_expect_tx(&full[slot], stage_bytes);
#pragma unroll
                    for (int b = 0; b < BOXES; ++b) ts_tma_2d(xs + (size_t)slot * stage_bytes + b * box * 128, &xmap, s * 64, m + b * box, &full[slot]);
                    if (++slot == SLOTS) slot = 0, ph ^= 1u;
                }
            }
            if (!ok) {
                flags[0] = 1;
                atomicExch(p.status, 1u);
                atomicExch(p.status + 1, 0x500u + blockIdx.x);
                const long long t0 = clock64();    // (the copies that were issued land before the CTA leaves)
                while (clock64() - t0 < (1LL << 22)) {}
            }
        }
    } else if (warp == GM_IWARP) {
        // ------------------------------ MMA issuer ------------------------------
        // One barrier per stage says that both operands are in place, and the barrier of the next stage is read before
        // the MMAs of this one are issued, so that its latency runs beside them.
        int total = 0;
        for (int q = 0; q < sg.nseg; ++q) total += seg_stages(q);
        bool ok = tbase == 0;                      // (an allocation of all columns can only start at column 0)
        if (elect_one()) {
            const uint32_t d0 = gm_bdesc_lo(smem_u32(xs));
            int q = 0, left = 0;
            uint32_t first = 0, ph = 0, dph = 1;   // dph: parity of the read-out of the segment before
            bool rdy = mbar_test(&full[0], 0u);
            for (int it = 0; it < total && ok; it += SLOTS, ph ^= 1u) {
#pragma unroll
                for (int slot = 0; slot < SLOTS; ++slot) {
                    if (it + slot >= total) break;
                    if (left == 0) {
                        left = seg_stages(q++);
                        first = 1;
                        if (!mbar_wait_timed(d_empty, dph)) ok = false;        // D of the previous segment must have been read out
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
                    rdy = mbar_test(&full[(slot + 1) % SLOTS], slot + 1 == SLOTS ? ph ^ 1u : ph);
                    const uint32_t d = d0 + (uint32_t)slot * (stage_bytes >> 4);
#pragma unroll
                    for (int b = 0; b < BOXES; ++b)
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            gm_mma(b * box, A_COL + slot * ACOLS + k * 8, d + b * box * 8 + k * 2, idesc, k ? 1u : first ^ 1u);
                            if (EXACT) gm_mma(b * box, A_COL + slot * ACOLS + 32 + k * 8, d + b * box * 8 + k * 2, idesc, 1u);
                        }
                    gm_commit(&empty[slot]);
                    first = 0;
                    if (--left == 0) gm_commit(d_full);
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
    } else if (warp >= GM_PWARP) {
        // ------------------------------ packed words and coefficients ------------------------------
        // Every second window.  A lane copies the words of four rows, asynchronously, and gathers their coefficient lines: line numbers
        // two of its windows ahead, lines one ahead.  (By the decoders, a stage ahead, the loads were what they waited for most.)
        int slot = warp - GM_PWARP;
        uint32_t ph = 1;
        bool ok = true;
        while (win.q < sg.nseg) {
            if (!first_words) {                    // (of its first window before the barriers were set up)
                if (flags[0] || !mbar_wait_timed(&p_empty[slot], ph)) ok = false;
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                copy_words(win, slot);
            }
            first_words = false;
            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(&p_full[slot])) : "memory");
            Pos ahead = win;
            next(ahead), next(ahead);
            uint2 c1[2][4];
            load_coef(ahead, lines, c1);           // (its line numbers came with the window before)
            if (one_coef) {                        // (the window before is in the other of two slots; the parity of its phase, which its warp has met)
                static_assert(NX != GM_WIDE || WINDOWS == 2, "a window before in the other slot");
                const int mine = warp - GM_PWARP;
                if (flags[0] || !mbar_wait_timed(&p_empty[slot ^ 1], ph ^ (uint32_t)mine)) ok = false;
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
            }
            const uint32_t dst = smem_u32(cs) + (one_coef ? 0 : slot * coef_bytes);
#pragma unroll
            for (int t = 0; t < 2; ++t) {
                if (t >= sets) break;
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    asm volatile("st.shared.v2.b32 [%0], {%1,%2};" ::"r"(dst + t * 1024 + (lane + 32 * i) * 8), "r"(coef[t][i].x), "r"(coef[t][i].y) : "memory");
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&p_full[slot]);
            win = ahead;
            next(ahead), next(ahead);
            lines_of(ahead, lines);
#pragma unroll
            for (int t = 0; t < 2; ++t)
#pragma unroll
                for (int i = 0; i < 4; ++i) coef[t][i] = c1[t][i];
            slot += 2;
            if (slot >= WINDOWS) slot -= WINDOWS, ph ^= 1u;
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        if (!ok) {
            flags[0] = 1;
            if (lane == 0) {
                atomicExch(p.status, 1u);
                atomicExch(p.status + 1, 0xE00u + blockIdx.x);
            }
        }
    } else {
        // ------------------------------ decoder warpgroups ------------------------------
        const int wg = warp >> 2, wl = warp & 3;
        const int r = wl * 32 + lane;
        const uint32_t lane_sel = (uint32_t)(wl * 32) << 16;
        bool dead = false;

        // D of one finished segment -> y (or fp32 sums); every decoder warp takes part, also when dead.
        auto epilogue = [&](int q, uint32_t seq) {
            const int tile = sg.tile(q), mt = tile % p.MT, nt = tile / p.MT, n = nt * 128 + r;
            if (!dead && !mbar_wait_async(d_full, seq & 1u)) {
                dead = true;
                flags[0] = 1;
            }
            dead = __any_sync(0xffffffffu, dead);
            const int m0 = mt * nx;
            const bool shared = sg.shared(q);
            const int rt = shared ? sg.rt_first + q : 0;
            if (!dead) {
                gm_fence_after();
                const bool on = n < N;
                const float bias = (p.bias && !shared && on) ? __half2float(p.bias[n]) : 0.0f;
                for (int c = wg; c < nx / 32; c += GM_DWGS) {
                    float d[32];
                    gm_ld32(tbase + lane_sel + c * 32, d);
                    if (!shared) {
#pragma unroll
                        for (int i = 0; i < 32; ++i) {
                            const int m = m0 + c * 32 + i;
                            if (on && m < p.M) p.y[(size_t)m * N + n] = __float2half_rn(d[i] + bias);
                        }
                    } else {
                        float* dst = p.part + ((size_t)(segs.cta + rt) * nx + c * 32) * 128 + r;
#pragma unroll
                        for (int i = 0; i < 32; ++i)
                            if (m0 + c * 32 + i < p.M) __stcg(dst + i * 128, d[i]);
                    }
                }
                gm_fence_before();
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(d_empty);
        };

        // The slot of stage `it` may be stored to; false: a wait ran out here or elsewhere.  A parity tells a phase only from the next, so
        // it must be certain that the slot's stage before last, it - 2 SLOTS, has been read.  At its stage before, it - 4, this warpgroup
        // waited for it - 4 - SLOTS, and MMAs run in order: four slots are enough.  (After a window of two stages, which two warpgroups sit
        // out, all of them wait for the end of the tile.)
        static_assert(SLOTS >= GM_DWGS, "phases of the ring");
        auto slot_free = [&](int it) -> bool {
            if (!dead && !mbar_wait_async(&empty[it % SLOTS], ((uint32_t)(it / SLOTS) & 1u) ^ 1u)) {
                dead = true;
                flags[0] = 1;
            }
            dead = __any_sync(0xffffffffu, dead);
            if (!dead) gm_fence_after();
            return !dead;
        };
        auto decode_stage = [&](int it, const uint32_t (&w)[2][S], const unsigned short (&c)[4]) {
            const int slot = it % SLOTS;
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
                            if (w[h][s] & (1u << (2 * j))) v0 += cf[s];
                            if (w[h][s] & (2u << (2 * j))) v1 += cf[s];
                        }
                        gm_two_parts(v0, v1, odd, hi[j], lo[j]);
                    }
                    if (h == 0 && !slot_free(it)) return;
                    gm_st16(tbase + lane_sel + A_COL + slot * ACOLS + h * 16, hi);
                    gm_st16(tbase + lane_sel + A_COL + slot * ACOLS + 32 + h * 16, lo);
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
            auto natural = [&](int h, const __half2 (&acc)[16]) {              // pairs (j, j + 16) -> pairs (2 j, 2 j + 1)
                const uint32_t* f = reinterpret_cast<const uint32_t*>(acc);
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    a[16 * h + j] = __byte_perm(f[2 * j], f[2 * j + 1], 0x5410);
                    a[16 * h + 8 + j] = __byte_perm(f[2 * j], f[2 * j + 1], 0x7632);
                }
            };
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
                    natural(h, acc);
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
                    __half2 acc[16];
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        acc[j] = *reinterpret_cast<const __half2*>(&base2);
#pragma unroll
                        for (int s = 0; s < S; ++s) {
                            const uint32_t v = w[h][s] << (15 - j);
                            const uint32_t t = (~v & 0x80008000u) ^ hc[s];
                            acc[j] = __hadd2(acc[j], *reinterpret_cast<const __half2*>(&t));
                        }
                    }
                    natural(h, acc);
                }
            }
            // the slot is waited for with the values in registers: the decode runs beside the MMAs that still read the slot
            if (!slot_free(it)) return;
            gm_st32(tbase + lane_sel + A_COL + slot * ACOLS, a);
            hand_over();
        };

        int it0 = 0, wi = 0;                       // stages and windows before the current window
        bool waited = false;
        for (int q = 0; q < sg.nseg; ++q) {
            const int k1 = segs.k1(q);
            for (int kb = segs.k0(q); kb < k1; ++kb, ++wi) {
                const int nst = stages_of(kb), slot = wi % WINDOWS;
                const unsigned char *src = ps + slot * word_bytes, *csrc = cs + (one_coef ? 0 : slot * coef_bytes);
                if (!dead && !mbar_wait_timed(&p_full[slot], (uint32_t)(wi / WINDOWS) & 1u)) {
                    dead = true;
                    flags[0] = 1;
                }
                dead = __any_sync(0xffffffffu, dead);
                uint32_t w[2][S];
                unsigned short c[4];
                if (wg < nst) {
                    const uint2 cc = *reinterpret_cast<const uint2*>(csrc + (p.G == 128 ? (wg >> 1) * 1024 : 0) + r * 8);
                    c[0] = (unsigned short)cc.x, c[1] = (unsigned short)(cc.x >> 16), c[2] = (unsigned short)cc.y, c[3] = (unsigned short)(cc.y >> 16);
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const uint32_t* g = reinterpret_cast<const uint32_t*>(src) + ((2 * wg + h) * 128 + r) * S;
                        if constexpr (S == 4) {
                            const uint4 v = *reinterpret_cast<const uint4*>(g);
                            w[h][0] = v.x, w[h][1] = v.y, w[h][2] = v.z, w[h][3] = v.w;
                        } else if constexpr (S == 2) {
                            const uint2 v = *reinterpret_cast<const uint2*>(g);
                            w[h][0] = v.x, w[h][1] = v.y;
                        } else {
#pragma unroll
                            for (int s = 0; s < S; ++s) w[h][s] = g[s];
                        }
                    }
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&p_empty[slot]);
                if (wg < nst && !dead) decode_stage(it0 + wg, w, c);
                it0 += nst;
            }
            if (!waited) {
                pdl_wait();                        // y and the parts may still be in use by the previous kernels
                waited = true;
            }
            epilogue(q, (uint32_t)q);
        }
        if (dead) {
            flags[0] = 1;
            if (lane == 0) {
                atomicExch(p.status, 1u);
                atomicExch(p.status + 1, 0x800u + blockIdx.x);
            }
        }
    }
    // ------------------------------ teardown ------------------------------
    gm_fence_before();
    __syncthreads();
    gm_fence_after();
    if (warp == GM_XWARP)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tbase), "r"((uint32_t)GM_TMEM_COLS)
                     : "memory");
}

// The sums of the shared tiles, added in the order of K: a thread four weight rows of an activation row.  A launch of its own, over the
// whole GPU: the last CTA to arrive at a tile had up to eighteen sums of 128 KB to add (256 x 1024 x 4096: 39 us, now 15).  Blocks of 128
// threads with 32 registers fit beside a CTA of the product.  Where little is to be added one per SM does it, and is there when the
// product ends, so that the next call's product may start (37 x 3000 x 3000: 16.1 -> 14.3 us); else a warp has one row, in as many
// blocks as that takes (128 x 14336 x 4096: 33 us, 47 by a block per SM).
constexpr int GM_ADD_WARPS = 4;
__global__ void __launch_bounds__(GM_ADD_WARPS * 32, 16) gm_add_kernel(const float* __restrict__ part, const __half* __restrict__ bias,
                                                                                  __half* __restrict__ y, int M, int N, int MT, int nx, int tiles, int KBS,
                                                                                  int ctas) {
    pdl_launch_dependents();
    TsSegs sg;
    sg.init(tiles, KBS, (unsigned int)ctas, 0u);
    const int rows = min(nx, M), left = tiles - sg.rem_tile0, c = (threadIdx.x & 31) * 4;      // (rows past the last of a last tile are skipped)
    const bool wide = N % 4 == 0 && !(reinterpret_cast<uintptr_t>(y) & 7);
    const long long jobs = (long long)left * rows;
    pdl_wait();
    int rt0 = -1, c0 = 0, parts = 0, m0 = 0, n = 0;
    for (long long job = (long long)blockIdx.x * GM_ADD_WARPS + (threadIdx.x >> 5); job < jobs; job += (long long)gridDim.x * GM_ADD_WARPS) {
        const int rt = (int)(job / rows), i = (int)(job - (long long)rt * rows);
        if (rt != rt0) {
            rt0 = rt;
            c0 = sg.cta_of((unsigned int)(rt * sg.KBS)), parts = sg.cta_of((unsigned int)(rt * sg.KBS + sg.KBS - 1)) - c0 + 1;
            const int tile = sg.rem_tile0 + rt;
            m0 = tile % MT * nx, n = tile / MT * 128 + c;
        }
        if (parts == 1 || m0 + i >= M || n >= N) continue;     // (one CTA has done the tile alone)
        const float* src = part + ((size_t)(c0 + rt) * nx + i) * 128 + c;
        float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        for (int q = 0; q < parts; q += 3) {
            float4 t[3];
#pragma unroll
            for (int h = 0; h < 3; ++h) {
                t[h] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                if (q + h < parts) t[h] = __ldcg(reinterpret_cast<const float4*>(src));
                src += (size_t)nx * 128;
            }
#pragma unroll
            for (int h = 0; h < 3; ++h) v.x += t[h].x, v.y += t[h].y, v.z += t[h].z, v.w += t[h].w;
        }
        const float o[4] = {v.x, v.y, v.z, v.w};
        __half* dst = y + (size_t)(m0 + i) * N + n;
        __align__(8) __half h[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) h[k] = __float2half_rn(o[k] + (bias && n + k < N ? __half2float(bias[n + k]) : 0.0f));
        if (wide) {
            *reinterpret_cast<uint2*>(dst) = *reinterpret_cast<const uint2*>(h);
        } else {
#pragma unroll
            for (int k = 0; k < 4; ++k)
                if (n + k < N) dst[k] = h[k];
        }
    }
}

// ---------------------------------------------------------------------------------------------
// host
// ---------------------------------------------------------------------------------------------
// The scratch that a call is accepted by, and the shares of K that the choice between this kernel and the small-batch kernel counts
// with: both as they were when activations were re-tiled into blocks of NX rows (up to 384 where that saved rounds of tiles) and K
// was split evenly, so that workspaces, the fixed array of the no-allocation entry and the precision of few rows stay what they were.
struct GmScratch {
    int KS, SPP, items;
    size_t bytes;
};
static int gm_scratch_rows(int M, int NT, int S, int sm_count, bool exact) {
    if (M <= 256 || exact) return (M <= 32 && !exact) ? 32 : M <= 64 ? 64 : M <= 128 ? 128 : 256;
    int best = 256;
    long long cost = 0;
    for (int nx = 256; nx <= 384; nx += 32) {
        const long long items = (long long)NT * ((M + nx - 1) / nx);
        if (nx == 256 && items < sm_count) break;
        const long long c = (items + sm_count - 1) / sm_count * (nx == 256 ? 610 + 60 * S : 3 * nx);
        if (nx == 256 || c < cost) best = nx, cost = c;
    }
    return best;
}
static GmScratch gm_scratch(const PackedW& w, int M, int sm_count) {
    const int NT = (w.N + 127) / 128, NX = gm_scratch_rows(M, NT, w.S, sm_count, w.N % 128 != 0), MT = (M + NX - 1) / NX, KST = w.K / 64;
    const int tiles = NT * MT;
    GmScratch s;
    s.KS = 1;
    if (NX <= 256 && tiles < sm_count && tiles <= SBVR_WS_COUNTERS)
        for (int cand = 2; cand <= KST / 4 && tiles * cand <= sm_count; ++cand)
            if (KST % cand == 0) s.KS = cand;
    s.SPP = KST / s.KS, s.items = tiles * s.KS;
    s.bytes = ((size_t)MT * NX * w.K * 2 + 255) / 256 * 256 + (s.KS > 1 ? (size_t)s.KS * MT * NX * w.N * 4 : 0);
    return s;
}
size_t linear_gemm_workspace_bytes(const PackedW& w, int M, int sm_count) { return gm_scratch(w, M, sm_count).bytes; }
void linear_gemm_split(const PackedW& w, int M, int sm_count, int* parts, int* stages) {
    const GmScratch s = gm_scratch(w, M, sm_count);
    *parts = s.KS, *stages = s.SPP * ((s.items + sm_count - 1) / sm_count);
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

struct GmPlan {
    int nx, MT, tiles, KBS, grid;
    bool exact, whole;
    size_t part_bytes;
    long long ns;
};

// Activation rows of a tile, and whether the tiles that are left over after whole rounds are cut: the least time in ns by these figures.
// Up to 256 rows, and in two parts (17 .. 256 rows, 1024 .. 28672 x 2048 .. 14336, S = 2 .. 4): a 64-k stage takes its decoding, 150 + 50 S (in two
// parts 200 + 120 S), or 1.05 a row + 40 S (2.1 a row + 120); a call 3 000 + 8 a row, another round's ends 1 500; cutting adds a launch, 5 000,
// and 0.36 per KB of sums out and back.  Measured whole and cut, us, S = 4: 64 x 14336 x 4096 (112 tiles) 27.6, 30.8; 64 x 4096 x 14336 76.7, 29.1; 64 x
// 4096 x 4096 23.6, 16.9; 64 x 28672 x 8192 95, 80.
// More rows: see gm_many_ns.  270 x 28672 x 8192 in two tiles and in one 212, 119; 384 x 14336 x 4096 62, 40; 384 x 4096 x 4096 28, 36.
//
// gm_many_ns and the figures of gp_plan (linear_pair.cu), which decide between the kernels, were fitted to both kernels' times, this one's in tiles
// of 256 .. 384 rows, at 278 sizes (257 .. 4096 rows, 1024 .. 28672 x 256 .. 14336, S = 2 .. 4, both group lengths) in loops of 25 to 60 ms: long runs meet
// the power limit, as in a model's prefill, and this kernel, which decodes a weight twice as often, more than the other (1024 x 4096 x 14336 101 us, the
// other 100, in bursts; 124, 111 in loops).  A choice by them costs 0.8 % on average against the fastest of the six, 0.9 % at 220 other sizes, 22 % at most.
// (By figures that took 1 500 for the ends of every round it was 3.6 and 7 % in bursts, 51 % at most: a tile's results take 4 to 8 us out of D,
// in which this kernel's MMAs rest.)
static long long gm_many_ns(int S, int nx, long long rounds, long long last, long long stages, int sm_count) {
    const long long t = stages * (115 * nx / 100 + 29 * S), run = t + t * 26 / 100 * std::min(std::max(t - 40000, 0LL), 110000LL) / 110000;
    return 4100 + run + (rounds - 1) * (4000 + 10 * nx) + 33 * nx / 2 * last / sm_count;
}
static GmPlan gm_plan_nx(const PackedW& w, int M, int nx, int sm_count, size_t scratch) {
    GmPlan pl;
    pl.exact = w.N % 128 != 0;
    pl.nx = nx;
    pl.MT = (M + nx - 1) / nx;
    pl.tiles = (w.N + 127) / 128 * pl.MT;
    pl.KBS = (w.K + 255) / 256;
    const bool many = M > 256 && !pl.exact;
    const long long call = 3000 + 8 * std::min(nx, 256), rounds = (pl.tiles + sm_count - 1) / sm_count;
    const int row = rounds <= 2 ? 105 : 120;
    const long long stage = pl.exact ? std::max(200 + 120 * w.S, 21 * nx / 10 + 120) : std::max(150 + 50 * w.S, row * nx / 100 + 40 * w.S);
    pl.whole = true, pl.part_bytes = 0;
    pl.grid = std::min(pl.tiles, sm_count);
    pl.ns = many ? gm_many_ns(w.S, nx, rounds, pl.tiles - (rounds - 1) * sm_count, rounds * (w.K / 64), sm_count)
                 : call + rounds * (w.K / 64 * stage + 1500) - 1500;
    const long long windows = (long long)pl.tiles * pl.KBS, ctas = std::min<long long>(windows, sm_count), left = pl.tiles % ctas;
    if (left && left * pl.KBS >= ctas && left * pl.KBS * ctas < (1LL << 32)) {             // (every CTA has a window of them at least)
        const size_t bytes = (size_t)(ctas + left) * nx * 512;
        const long long run = (windows + ctas - 1) / ctas * 4;
        const long long ns = many ? gm_many_ns(w.S, nx, rounds, 0, run, sm_count) - 600 + (long long)(bytes * 13 / 25000)
                                  : call + 5000 + run * stage + (rounds - 1) * 1500 + (long long)(bytes * 9 / 25000);
        if (ns < pl.ns && bytes <= scratch) pl.whole = false, pl.part_bytes = bytes, pl.grid = (int)ctas, pl.ns = ns;
    }
    return pl;
}
static GmPlan gm_plan(const PackedW& w, int M, int sm_count, size_t scratch) {
    const bool exact = w.N % 128 != 0;
    GmPlan best = gm_plan_nx(w, M, (M <= 32 && !exact) ? 32 : M <= 64 ? 64 : M <= 128 ? 128 : 256, sm_count, scratch);
    if (M <= 256 || exact) return best;
    for (int nx = 288; nx <= GM_WIDE; nx += 32) {
        const GmPlan pl = gm_plan_nx(w, M, nx, sm_count, scratch);
        if (pl.ns < best.ns) best = pl;
    }
    return best;
}

template <int S, int NX, bool EXACT = false>
static int gm_launch(const CUtensorMap& xmap, const GmParams& p, int grid, cudaStream_t st) {
    static SmemOnce once;
    const int rc = set_max_smem_once(once, linear_gemm_kernel<S, NX, EXACT>, GM_SMEM_MAX);
    if (rc) return rc;
    SBVR_CUDA_TRY(launch_pdl(linear_gemm_kernel<S, NX, EXACT>, dim3(grid), dim3(GM_THREADS), (size_t)gm_smem(NX, p.nx, EXACT, S, p.G), st, xmap, p));
    return SBVR_OK;
}
template <int S>
static int gm_launch_nx(const CUtensorMap& xmap, const GmParams& p, const GmPlan& pl, cudaStream_t st) {
    if (pl.exact) switch (pl.nx) {
        case 64: return gm_launch<S, 64, true>(xmap, p, pl.grid, st);
        case 128: return gm_launch<S, 128, true>(xmap, p, pl.grid, st);
        default: return gm_launch<S, 256, true>(xmap, p, pl.grid, st);
    }
    switch (pl.nx) {
        case 32: return gm_launch<S, 32>(xmap, p, pl.grid, st);
        case 64: return gm_launch<S, 64>(xmap, p, pl.grid, st);
        case 128: return gm_launch<S, 128>(xmap, p, pl.grid, st);
        case 256: return gm_launch<S, 256>(xmap, p, pl.grid, st);
        default: return gm_launch<S, GM_WIDE>(xmap, p, pl.grid, st);
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
    if (linear_gemm_workspace_bytes(w, M, di.sm_count) > ws->dyn_bytes) return SBVR_ERR_WORKSPACE;
    // What a plan may count on beside the padded rows: what sbvr_workspace_bytes promises, whatever the workspace has grown to for other calls.
    size_t promised = 0;
    if (sbvr_workspace_bytes(ws->device, M, w.N, w.K, &promised) != SBVR_OK) promised = SBVR_WS_FIXED_BYTES;
    const size_t rows = ((size_t)M * w.K * 2 + 255) / 256 * 256, scratch = std::min(ws->dyn_bytes, promised - SBVR_WS_FIXED_BYTES);
    const GmPlan pl = gm_plan(w, M, di.sm_count, scratch > rows ? scratch - rows : 0);
    if (linear_pair_supported(x, Kin, w, y, M) && linear_pair_ns(w, M, di.sm_count, ws->device, ws->dyn_bytes) < pl.ns)
        return launch_linear_pair(x, Kin, w, bias, y, M, ws->status, ws->dyn, ws->dyn_bytes, di.sm_count, ws->device, st);
    if (Kin % 8 || (reinterpret_cast<uintptr_t>(x) & 15)) {        // rows that TMA cannot read
        __half* xp = reinterpret_cast<__half*>(ws->dyn);
        rc = launch_pad_rows(x, xp, M, Kin, w.K, st);
        if (rc) return rc;
        x = xp, Kin = w.K;
    }
    CUtensorMap xmap;
    rc = ts_map_2d(&xmap, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, CU_TENSOR_MAP_SWIZZLE_128B, x, (size_t)M, (size_t)Kin, (size_t)Kin * 2,
                   pl.nx > 256 ? pl.nx / 2 : pl.nx, 64);
    if (rc) return rc;
    GmParams p;
    p.bvr = w.bvr, p.idx = w.idx, p.coeff = w.coeff, p.bias = bias, p.y = y;
    p.part = reinterpret_cast<float*>(ws->dyn + rows);
    p.status = ws->status;
    p.M = M, p.N = w.N, p.K = w.K, p.G = w.G, p.idx_bytes = w.idx_bytes;
    p.vec = !(reinterpret_cast<uintptr_t>(w.coeff) & (2 * w.S - 1));
    p.nx = pl.nx, p.MT = pl.MT, p.tiles = pl.tiles, p.KBS = pl.KBS, p.whole = pl.whole;
    switch (w.S) {
        case 2: rc = gm_launch_nx<2>(xmap, p, pl, st); break;
        case 3: rc = gm_launch_nx<3>(xmap, p, pl, st); break;
        default: rc = gm_launch_nx<4>(xmap, p, pl, st);
    }
    if (rc || pl.whole) return rc;
    const long long left = pl.tiles % pl.grid, jobs = left * std::min(pl.nx, M);
    if (jobs) {
        const bool few = jobs <= 2LL * GM_ADD_WARPS * di.sm_count && pl.grid <= 8 * left;
        SBVR_CUDA_TRY(launch_pdl(gm_add_kernel, dim3(few ? (unsigned)di.sm_count : (unsigned)((jobs + GM_ADD_WARPS - 1) / GM_ADD_WARPS)),
                                 dim3(GM_ADD_WARPS * 32), 0, st, p.part, bias, y, M, w.N, pl.MT, pl.nx, pl.tiles, pl.KBS, pl.grid));
    }
    return SBVR_OK;
}

}  // namespace sbvr
