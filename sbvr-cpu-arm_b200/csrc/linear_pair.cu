// SBVR linear for many activation rows (prefill): a tcgen05 fp16 GEMM over CTA pairs whose weight operand is dequantised inside
// the kernel, once per 512 activation rows.
//
//   y[m, n] = sum_k x[m, k] * W[n, k] (+ bias[n]),   W[n, k] = sum_s c[k/G, n, s] * bit_s[n, k]
//
// What bounds the one-CTA kernel (linear_gemm.cu) there is the decoding: 730 to 870 cycles per 64 k of 128 weight rows, which then serve
// 256 to 384 activation rows (512 to 768 cycles of tensor time).  Here two SMs share one MMA (`cta_group::2`): each decodes HALF of the
// tile's weight rows into its own shared memory, where the MMAs of both read them, and a decoded row serves 2 x 256 activation rows, so
// that a stage is up to 1024 cycles of tensor time for the same decoding.  What bounds this kernel is the power limit (the clock falls to
// 1.35 .. 1.5 GHz with the tensor pipe 85 % busy).  S = 4, us in bursts of eight calls one after the other on one GPU, with the one-CTA kernel's time
// (its best tile) and that of a dense fp16 product of the same shape by cuBLAS: 2048 x 14336 x 4096 195 (207, 185), 2048 x 4096 x 14336 187 (204, 161),
// 2048 x 4096 x 4096 55 (69, 64), 3000 x 28672 x 4096 579 (632, 505), 512 x 28672 x 8192 181 (258, 234), 512 x 28672 x 4096 92 (130, 114); about
// equal 3000 x 4096 x 4096 83 (82, 95) and 1100 x 14336 x 4096 116 (119), slower 300 x 4096 x 14336 57 (41).
//
// Operands of tcgen05.mma kind::f16, D[256 activation rows, n weight rows] (128 rows of D in each SM's tensor memory), n <= 256:
//  A (activations, shared memory)  TMA boxes of 128 rows x 64 k straight from x (128-byte swizzle): no re-tiled copy of x exists.
//      Rows and columns past the end are filled with zeros by the copy.
//  B (weights, shared memory)  Decoder thread r of a warpgroup owns weight row r of its SM's n / 2; the values are formed two at a
//      time in half2 exactly as in linear_gemm.cu (same roundings), brought into their natural order with one byte permute per pair,
//      and stored as 16-byte chunks of the MMA's core matrices (chunk-major: a warp's stores cover all banks).
//
// A work item is 512 activation rows (two blocks of 256 with a D of 256 columns each) x n weight rows x all of K.  Whole rounds of items
// are done pair by pair; items left over may be cut into ranges of K (TsSegs), whose fp32 sums a second, small kernel adds in the order
// of K.
//
// Roles per CTA (23 warps): 0-15 four decoder warpgroups (64-k stages round-robin), 16-19 read D out and store y (rows through shared
// memory, 64 bytes at a time), 20 issues the MMAs (first CTA of the pair only, one lane), 21 fetches activations, 22 fetches packed words
// and gathers coefficient lines.  Barriers that the issuer waits on live in the first CTA; decoders and read-out warps of the second
// arrive there remotely, its TMA copies count there.  Commits go to both CTAs.  Every wait is bounded; a time-out is recorded in the
// status words, ends the roles one after the other, and the pair meets before it frees its tensor memory.
#include <algorithm>

#include "tc_stream.cuh"

namespace sbvr {

constexpr int GP_DWGS = 4;                         // decoder warpgroups
constexpr int GP_EWARP = GP_DWGS * 4;              // first of four read-out warps
constexpr int GP_IWARP = GP_EWARP + 4;             // MMA issuer
constexpr int GP_XWARP = GP_IWARP + 1;             // fetches activations
constexpr int GP_PWARP = GP_XWARP + 1;             // fetches packed words and coefficient lines
constexpr int GP_THREADS = (GP_PWARP + 1) * 32;
constexpr int GP_WSLOTS = 4;                       // decoded 128 x 64 weight tiles
constexpr int GP_ASLOTS = 3;                       // activations of a stage: a box of 128 x 64 per block
// Packed words and coefficients of a group of 128 weight rows: 8 x S words (G = 128: 4 x S) and four halves per row.  With G = 128 a
// decoder warpgroup uses every second group: an even number of slots, so that it meets every phase of those that it waits on (the parity of a
// phase tells it only from the next).
constexpr int GP_PSLOTS = 4;                       // at most
__host__ __device__ constexpr int gp_pslots(int spg) { return spg == 4 ? 3 : 4; }
__host__ __device__ constexpr uint32_t gp_coef_at(int spg) { return 128 * 2 * spg * 16; }
__host__ __device__ constexpr uint32_t gp_pbytes(int spg) { return gp_coef_at(spg) + 128 * 8; }
constexpr uint32_t GP_SLOT = 128 * 64 * 2;         // bytes of a decoded tile, of an activation box
constexpr int GP_OUT_PITCH = 80;                   // bytes between staged rows of 32 results: 16-byte accesses without bank conflicts
constexpr int GP_HDR = 1024;
constexpr int GP_SMEM = GP_HDR + (GP_WSLOTS + 2 * GP_ASLOTS) * (int)GP_SLOT + gp_pslots(4) * (int)gp_pbytes(4) + 4 * 32 * GP_OUT_PITCH;
static_assert(GP_SMEM <= 227 * 1024 && gp_pslots(2) * gp_pbytes(2) <= gp_pslots(4) * gp_pbytes(4), "shared memory");
constexpr int GP_TURN = 12;                        // stages after which both rings are at their start again, that of the activations in its first phase
static_assert(GP_TURN % GP_WSLOTS == 0 && GP_TURN % (2 * GP_ASLOTS) == 0, "the issuer's unrolled stages");

struct GpParams {
    const uint32_t* bvr;
    const void* idx;
    const __half* coeff;
    const __half* bias;
    __half* y;
    unsigned int* status;
    int M, N, idx_bytes;
    int vec;                     // lines of S = 4 (2) can be read as 8 (4) bytes
    int n;                       // weight rows of an item (multiple of 16)
    int MT, MB;                  // activation tiles of 512 rows, blocks of 256 rows
    int MF, full;                // activation tiles that are dealt out together, and their items: see gp_m
    int NG, spg;                 // coefficient groups along K, 64-k stages of each
    int items, steps;            // work items; steps of an item in the split over the pairs: NG, or 1 where items stay whole
    float* part;                 // sums of items that several pairs work on: [pair + left-over item][512 x n], see gp_part
};

// ---------------------------------------------------------------------------------------------
// PTX wrappers
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t gp_mapa(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ uint32_t gp_cta_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void gp_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Arrive on a barrier of either CTA of the pair (a shared::cluster address).  What it announces was made visible to the tensor cores by
// the proxy fence (or tcgen05 fence) in front of it; with release semantics at cluster scope on top every arrival took about a
// thousand cycles (189 -> 183 us at 512 x 28672 x 8192 without).
__device__ __forceinline__ void gp_arrive(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ bool gp_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
// false: about a second of SM clock has passed, or another role of this CTA has given up
__device__ __noinline__ bool gp_wait_slow(uint32_t bar, uint32_t parity, volatile int* dead) {
    const long long t0 = clock64();
    for (;;) {
        if (gp_try(bar, parity)) return true;
        if (*dead || clock64() - t0 > 2000000000LL) return false;
    }
}
__device__ __forceinline__ bool gp_wait(uint32_t bar, uint32_t parity, volatile int* dead) {
    return gp_try(bar, parity) || gp_wait_slow(bar, parity, dead);
}
// the commit of this thread's MMAs arrives at the barrier of this offset in both CTAs
__device__ __forceinline__ void gp_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
                 "h"((unsigned short)3)
                 : "memory");
}
// A: 128-byte swizzle, K-major, 1024 B between groups of 8 rows.  B: no swizzle, K-major, 2048 B between 16-byte chunks along K, 128 B
// between groups of 8 rows.  Both descriptors version 1; their upper words are constants.
constexpr uint32_t GP_ADESC_HI = (1024u >> 4) | (1u << 14) | (2u << 29);
constexpr uint32_t GP_BDESC_HI = (128u >> 4) | (1u << 14);
__device__ __forceinline__ void gp_mma(uint32_t d, uint32_t adesc_lo, uint32_t bdesc_lo, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 a, b;\n\tsetp.ne.b32 p, %4, 0;\n\tmov.b64 a, {%1, %5};\n\tmov.b64 b, {%2, %6};\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], a, b, %3, p;\n\t}" ::"r"(d),
        "r"(adesc_lo), "r"(bdesc_lo), "r"(idesc), "r"(accumulate), "r"(GP_ADESC_HI), "r"(GP_BDESC_HI)
        : "memory");
}
// one box of x into this CTA's shared memory; the bytes count at a barrier of the pair's first CTA
__device__ __forceinline__ void gp_tma(uint32_t dst, const CUtensorMap* tmap, int k, int m, uint32_t bar0) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
        "l"(reinterpret_cast<uint64_t>(tmap)), "r"(k), "r"(m), "r"(bar0)
        : "memory");
}
__device__ __forceinline__ void gp_ld32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
        "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]),
                   "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15]), "+r"(r[16]), "+r"(r[17]),
                   "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23]), "+r"(r[24]), "+r"(r[25]), "+r"(r[26]),
                   "+r"(r[27]), "+r"(r[28])
                 :
                 : "memory");
    asm volatile("" : "+r"(r[29]), "+r"(r[30]), "+r"(r[31])::"memory");
}

// A pair's work: the left-over items (TsSegs) first, cut into ranges of groups, then its own.
struct GpSegs {
    TsSegs sg;
    int NG, pair;
    __device__ __forceinline__ GpSegs(const GpParams& p, int pair_, int pairs) : NG(p.NG), pair(pair_) {
        sg.init(p.items, p.steps, (unsigned int)pairs, (unsigned int)pair_);
    }
    __device__ __forceinline__ int count() const { return sg.nseg; }
    __device__ __forceinline__ int item(int q) const { return sg.tile(q); }
    __device__ __forceinline__ int g0(int q) const { return sg.KBS == 1 ? 0 : sg.k0(q); }
    __device__ __forceinline__ int g1(int q) const { return sg.KBS == 1 ? NG : sg.k1(q); }
    // number of the part that the pair's sums of segment q are (a left-over item that it does not do alone), or -1
    __device__ __forceinline__ int part(int q) const { return sg.shared(q) ? pair + sg.rt_first + q : -1; }
};
// Activation tile and first weight row of an item.  Where the last activation tile has one block, its items, which are half as long, come
// after all others: next to the others of the same weight rows they fell to the same
// pairs every time (1100 x 14336 x 4096, where this kernel did it: 134 us, so 115).
__device__ __forceinline__ int gp_m(const GpParams& p, int item) { return item < p.full ? item % p.MF : p.MF; }
__device__ __forceinline__ int gp_n0(const GpParams& p, int item) { return (item < p.full ? item / p.MF : item - p.full) * p.n; }
// A part holds the sums of 32 activation rows x 32 weight rows one after the other, each as eight runs of one float4 per activation
// row: float4 i of row r is columns 4 i .. 4 i + 3.  `unit`: (block, CTA of the pair, warp), `chunk`: columns 32 chunk ..
__device__ __forceinline__ float4* gp_part(float* part, int n, int number, int unit, int chunk) {
    const int chunks = (n + 31) / 32;
    return reinterpret_cast<float4*>(part) + ((size_t)((number * 16 + unit) * chunks + chunk)) * 256;
}
// 32 x 32 results, a row of fp32 sums per lane: bias, fp16, through shared memory (`stage`: 32 rows of GP_OUT_PITCH bytes) to y
__device__ __forceinline__ void gp_store(const GpParams& p, uint32_t (&d)[32], uint32_t stage, int lane, int m0, int n0, int c) {
    if (p.bias) {
#pragma unroll
        for (int i = 0; i < 32; ++i) d[i] = __float_as_uint(__uint_as_float(d[i]) + __half2float(__ldg(p.bias + min(n0 + c + i, p.N - 1))));
    }
    uint32_t h[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const __half2 v = __floats2half2_rn(__uint_as_float(d[2 * i]), __uint_as_float(d[2 * i + 1]));
        h[i] = *reinterpret_cast<const uint32_t*>(&v);
    }
    const uint32_t mine = stage + lane * GP_OUT_PITCH;
#pragma unroll
    for (int i = 0; i < 4; ++i)
        asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(mine + i * 16), "r"(h[4 * i]), "r"(h[4 * i + 1]), "r"(h[4 * i + 2]),
                     "r"(h[4 * i + 3])
                     : "memory");
    __syncwarp();
    const int col = c + (lane & 3) * 8;            // read back: 8 rows of 64 bytes at a time
    const bool on = col < p.n && n0 + col < p.N;   // (both multiples of 16)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        uint4 v;
        asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                     : "r"(stage + ((lane >> 2) + i * 8) * GP_OUT_PITCH + (lane & 3) * 16)
                     : "memory");
        const int m = m0 + i * 8 + (lane >> 2);
        if (on && m < p.M) *reinterpret_cast<uint4*>(p.y + (size_t)m * p.N + n0 + col) = v;
    }
    __syncwarp();
}

// ---------------------------------------------------------------------------------------------
// the GEMM
// ---------------------------------------------------------------------------------------------
template <int S>
__global__ void __launch_bounds__(GP_THREADS, 1) linear_pair_kernel(const __grid_constant__ CUtensorMap xmap, const GpParams p) {
    extern __shared__ __align__(1024) unsigned char smem[];
    const uint32_t sbase = smem_u32(smem);
    const uint32_t a_full = sbase, a_empty = a_full + 8 * GP_ASLOTS, w_full = a_empty + 8 * GP_ASLOTS, w_empty = w_full + 8 * GP_WSLOTS,
                   d_full = w_empty + 8 * GP_WSLOTS, d_empty = d_full + 16, drained = d_empty + 16,       // (two of each d_*)
                   p_full = drained + 8, p_empty = p_full + 8 * GP_PSLOTS;
    volatile int* dead = reinterpret_cast<volatile int*>(smem + 512);
    uint32_t* tmem_base_s = reinterpret_cast<uint32_t*>(smem + 516);
    const uint32_t w_ring = sbase + GP_HDR, a_ring = w_ring + GP_WSLOTS * GP_SLOT, p_ring = a_ring + 2 * GP_ASLOTS * GP_SLOT,
                   out_s = p_ring + gp_pslots(4) * gp_pbytes(4);
    const uint32_t pslots = gp_pslots(p.spg), pbytes = gp_pbytes(p.spg), coef_at = gp_coef_at(p.spg);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = gp_cta_rank();
    const int pair = (int)blockIdx.x >> 1, pairs = (int)gridDim.x >> 1;

    pdl_launch_dependents();
    if (threadIdx.x == 0) {
        for (int i = 0; i < GP_ASLOTS; ++i) {
            mbar_init(reinterpret_cast<uint64_t*>(smem) + i, 1);                     // a_full: the first CTA's producer, and bytes
            mbar_init(reinterpret_cast<uint64_t*>(smem) + GP_ASLOTS + i, 1);         // a_empty: a commit
        }
        uint64_t* w = reinterpret_cast<uint64_t*>(smem) + 2 * GP_ASLOTS;
        for (int i = 0; i < GP_WSLOTS; ++i) {
            mbar_init(w + i, 8);                                                     // w_full: four decoder warps of either CTA
            mbar_init(w + GP_WSLOTS + i, 1);                                         // w_empty: a commit
        }
        uint64_t* d = w + 2 * GP_WSLOTS;
        for (int b = 0; b < 2; ++b) {
            mbar_init(d + b, 1);                                                     // d_full: a commit
            mbar_init(d + 2 + b, 8);                                                 // d_empty: four read-out warps of either CTA
        }
        mbar_init(d + 4, 1);                                                         // drained: a commit, after a time-out only
        for (int i = 0; i < GP_PSLOTS; ++i) {
            mbar_init(d + 5 + i, 1);                                                 // p_full: the fetching warp, and bytes
            mbar_init(d + 5 + GP_PSLOTS + i, 4 * p.spg);                                // p_empty: the four warps of every stage's warpgroup
        }
        *dead = 0;
        fence_mbar_init();
    }
    if (warp == GP_XWARP) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_base_s)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    }
    __syncthreads();
    gp_cluster_sync();                             // both CTAs' barriers are in place
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tbase = *tmem_base_s;
    const int half = p.n >> 1;
    const GpSegs sg(p, pair, pairs);
    const int stages = sg.sg.KBS == 1 ? sg.sg.steps * p.NG * p.spg : sg.sg.steps * p.spg;
    bool ok = tbase == 0;                          // (an allocation of all columns can only start at column 0)

    // blocks of 256 activation rows of an item: the last tile may have one
    auto blocks_of = [&](int item) { return min(2, p.MB - 2 * gp_m(p, item)); };

    if (warp == GP_XWARP) {
        // ------------------------------ activation producer ------------------------------
        pdl_wait();                                // x comes from the previous kernel
        if (lane == 0) {
            int slot = 0;
            uint32_t ph = 1;
            const uint32_t bar0 = gp_mapa(a_full, 0);
            for (int q = 0; q < sg.count() && ok; ++q) {
                const int item = sg.item(q), nb = blocks_of(item), m0 = gp_m(p, item) * 512 + (int)rank * 128, s1 = sg.g1(q) * p.spg;
                for (int ks = sg.g0(q) * p.spg; ks < s1; ++ks) {
                    if (!gp_wait(a_empty + 8 * slot, ph, dead)) {
                        ok = false;
                        break;
                    }
                    if (rank == 0)
                        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(a_full + 8 * slot), "r"(2 * GP_SLOT * nb) : "memory");
                    for (int b = 0; b < nb; ++b) gp_tma(a_ring + (2 * slot + b) * GP_SLOT, &xmap, ks * 64, m0 + b * 256, bar0 + 8 * slot);
                    if (++slot == GP_ASLOTS) slot = 0, ph ^= 1u;
                }
            }
            if (!ok) {                             // the copies that were issued land before the pair leaves
                *dead = 1;
                atomicExch(p.status, 1u);
                atomicExch(p.status + 1, 0x900u + blockIdx.x);
                // (they count at the first CTA, and with the pair out of step no phase may complete: a wait by the clock, 2^22 cycles)
                const long long t0 = clock64();
                while (clock64() - t0 < (1LL << 22)) {}
            }
        }
    } else if (warp == GP_IWARP) {
        // ------------------------------ MMA issuer ------------------------------
        // One lane.  The stages of a turn of the rings are unrolled, so that every operand of an MMA is a constant next to a warp-uniform
        // register.  It waits parked: spinning on the barriers, the next stage's read ahead, took fewer cycles but the power limit gave
        // them back and more (seconds-long loops at 3000 x 28672 x 4096: 600 us parked, 615 spinning; 512 x 28672 x 8192: 205, 219).
        if (rank == 0) {
            if (elect_one()) {
                const uint32_t idesc = (1u << 4) | ((uint32_t)(p.n >> 3) << 17) | ((uint32_t)(256 >> 4) << 24);
                const uint32_t a0 = (a_ring >> 4) | (1u << 16), b0 = (w_ring >> 4) | ((2048u >> 4) << 16);
                int q = 0, left = 0, nb = 0;       // segment, its stages that are left, its blocks
                uint32_t first = 0, wph = 0, dph0 = 1, dph1 = 1;
                for (int it = 0; it < stages && ok; it += GP_TURN, wph ^= (GP_TURN / GP_WSLOTS) & 1) {
#pragma unroll
                    for (int u = 0; u < GP_TURN; ++u) {
                        constexpr uint32_t SLOT4 = GP_SLOT >> 4;
                        const int ws = u % GP_WSLOTS, as = u % GP_ASLOTS;
                        const uint32_t wp = wph ^ ((u / GP_WSLOTS) & 1), aph = (u / GP_ASLOTS) & 1;
                        if (it + u >= stages) break;
                        if (left == 0) {
                            nb = blocks_of(sg.item(q));
                            left = (sg.g1(q) - sg.g0(q)) * p.spg;
                            ++q;
                            first = 1;
                            if (!gp_wait(d_empty, dph0, dead)) ok = false;     // D of block 0 has been read out
                            dph0 ^= 1u;
                        }
                        if (ok && !(gp_wait(w_full + 8 * ws, wp, dead) && gp_wait(a_full + 8 * as, aph, dead))) ok = false;
                        if (!ok) break;
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        --left;
#pragma unroll
                        for (int k = 0; k < 4; ++k) gp_mma(0u, a0 + 2 * as * SLOT4 + k * 2, b0 + ws * SLOT4 + k * 256, idesc, k ? 1u : first ^ 1u);
                        if (left == 0) gp_commit(d_full);
                        if (nb == 2) {
                            if (first) {
                                if (!gp_wait(d_empty + 8, dph1, dead)) ok = false;
                                dph1 ^= 1u;
                                if (!ok) break;
                                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                            }
#pragma unroll
                            for (int k = 0; k < 4; ++k) gp_mma(256u, a0 + (2 * as + 1) * SLOT4 + k * 2, b0 + ws * SLOT4 + k * 256, idesc, k ? 1u : first ^ 1u);
                            if (left == 0) gp_commit(d_full + 8);
                        }
                        gp_commit(a_empty + 8 * as);
                        gp_commit(w_empty + 8 * ws);
                        first = 0;
                    }
                }
                if (!ok) {                         // the MMAs that were issued end before the pair leaves
                    *dead = 1;
                    atomicExch(p.status, 1u);
                    atomicExch(p.status + 1, 0xA00u + blockIdx.x);
                    const long long t0 = clock64();
                    gp_commit(drained);
                    while (!gp_try(drained, 0u) && clock64() - t0 < 200000000LL) {}
                }
            }
            __syncwarp();
        }
    } else if (warp >= GP_EWARP && warp < GP_IWARP) {
        // ------------------------------ read-out ------------------------------
        pdl_wait();                                // y may still be read by the previous kernel
        const int wl = warp - GP_EWARP;
        const uint32_t stage = out_s + (uint32_t)wl * 32 * GP_OUT_PITCH;
        const uint32_t free0 = gp_mapa(d_empty, 0);
        uint32_t ph[2] = {0, 0};
        for (int q = 0; q < sg.count(); ++q) {
            const int item = sg.item(q), nb = blocks_of(item), n0 = gp_n0(p, item), part = sg.part(q);
            for (int b = 0; b < nb; ++b) {
                if (ok && !gp_wait(d_full + 8 * b, ph[b], dead)) ok = false;
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                ph[b] ^= 1u;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const int m0 = gp_m(p, item) * 512 + b * 256 + (int)rank * 128 + wl * 32;
                for (int c = 0; c < p.n; c += 32) {            // (of a last chunk of 16 columns the rest is not stored)
                    uint32_t d[32];
                    gp_ld32(((uint32_t)(wl * 32) << 16) + b * 256 + c, d);
                    if (c + 32 >= p.n) {           // D is read: the next item's MMAs may have it
                        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                        __syncwarp();
                        if (lane == 0) gp_arrive(free0 + 8 * b);
                    }
                    if (part >= 0) {
                        float4* dst = gp_part(p.part, p.n, part, (b * 2 + (int)rank) * 4 + wl, c >> 5) + lane;
#pragma unroll
                        for (int i = 0; i < 8; ++i)
                            __stcg(dst + i * 32, make_float4(__uint_as_float(d[4 * i]), __uint_as_float(d[4 * i + 1]), __uint_as_float(d[4 * i + 2]),
                                                             __uint_as_float(d[4 * i + 3])));
                    } else {
                        gp_store(p, d, stage, lane, m0, n0, c);
                    }
                }
            }
            if (!ok) break;
        }
        if (!ok && lane == 0) {
            *dead = 1;
            atomicExch(p.status, 1u);
            atomicExch(p.status + 1, 0xB00u + blockIdx.x);
        }
    } else if (warp == GP_PWARP) {
        // ------------------------------ packed words and coefficients ------------------------------
        // A group at a time: the words of 32 k are one run of memory, a bulk copy by a lane each; the coefficient lines are gathered by the
        // whole warp, four rows a lane, line numbers two groups ahead, lines one group ahead.  (Loaded by the decoders themselves the words
        // and lines held up the fence in front of every hand-over, 212 us at 512 x 28672 x 8192; fetched stage by stage by one lane they
        // came too late, 188 us.)
        const int N = p.N, spg = p.spg;
        struct Pos {
            int q, g, end, n;                      // segment, group, end of its groups, this lane's first weight row
        };
        auto set_seg = [&](Pos& a) {
            if (a.q >= sg.count()) return;
            a.g = sg.g0(a.q), a.end = sg.g1(a.q);
            a.n = gp_n0(p, sg.item(a.q)) + (int)rank * half + lane;
        };
        auto next_group = [&](Pos& a) {
            if (++a.g >= a.end) {
                ++a.q;
                set_seg(a);
            }
        };
        auto lines_of = [&](const Pos& q, uint32_t (&l)[4]) {
            if (q.q >= sg.count()) return;
            const size_t g = (size_t)q.g * N;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const size_t e = g + min(q.n + 32 * i, N - 1);           // rows past the last (or the tile) repeat some line
                if (p.idx_bytes == 1) l[i] = __ldg(reinterpret_cast<const uint8_t*>(p.idx) + e);
                else if (p.idx_bytes == 2) l[i] = __ldg(reinterpret_cast<const uint16_t*>(p.idx) + e);
                else l[i] = (uint32_t)e;
            }
        };
        auto load_coef = [&](const Pos& q, const uint32_t (&l)[4], uint2 (&c)[4]) {
            if (q.q >= sg.count()) return;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const unsigned short* src = reinterpret_cast<const unsigned short*>(p.coeff) + (size_t)l[i] * S;
                if (S == 4 && p.vec) c[i] = __ldg(reinterpret_cast<const uint2*>(src));
                else if (S == 2 && p.vec) c[i].x = __ldg(reinterpret_cast<const uint32_t*>(src));
                else {
                    c[i].x = __ldg(src) | ((uint32_t)__ldg(src + 1) << 16);
                    if (S > 2) c[i].y = __ldg(src + 2);
                    if (S > 3) c[i].y |= (uint32_t)__ldg(src + 3) << 16;
                }
            }
        };
        Pos ga{0, 0, 0, 0};                        // the group whose lines are in c1; l is of the one after
        set_seg(ga);
        uint2 c0[4] = {}, c1[4] = {};
        uint32_t l[4] = {};
        lines_of(ga, l);
        load_coef(ga, l, c1);
        next_group(ga);
        lines_of(ga, l);
        int slot = 0;
        uint32_t ph = 1;
        for (int q = 0; q < sg.count() && ok; ++q) {
            const int n0 = gp_n0(p, sg.item(q)) + (int)rank * half, rows = min(half, N - n0);
            const uint32_t bytes = rows > 0 ? (uint32_t)(rows * S * 4) : 0u;
            const uint32_t* src = p.bvr + (size_t)n0 * S;
            for (int g = sg.g0(q), g1 = sg.g1(q); g < g1; ++g) {
#pragma unroll
                for (int i = 0; i < 4; ++i) c0[i] = c1[i];
                load_coef(ga, l, c1);
                next_group(ga);
                lines_of(ga, l);
                if (!gp_wait(p_empty + 8 * slot, ph, dead)) ok = false;
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                const uint32_t dst = p_ring + slot * pbytes;
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    asm volatile("st.shared.v2.b32 [%0], {%1,%2};" ::"r"(dst + coef_at + (lane + 32 * i) * 8), "r"(c0[i].x), "r"(c0[i].y) : "memory");
                __syncwarp();
                if (lane == 0)
                    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(p_full + 8 * slot), "r"(2 * spg * bytes) : "memory");
                __syncwarp();
                if (bytes && lane < 2 * spg)
                    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                                     dst + lane * (uint32_t)(half * S * 4)),
                                 "l"(src + (size_t)(2 * g * spg + lane) * N * S), "r"(bytes), "r"(p_full + 8 * slot)
                                 : "memory");
                if (++slot == (int)pslots) slot = 0, ph ^= 1u;
            }
        }
        if (!ok && lane == 0) {                    // copies that were issued land before the pair leaves
            *dead = 1;
            atomicExch(p.status, 1u);
            atomicExch(p.status + 1, 0xD00u + blockIdx.x);
            const long long t0 = clock64();
            while (clock64() - t0 < (1LL << 22)) {}
        }
    } else {
        // ------------------------------ decoder warpgroups ------------------------------
        // The stages of all items of this pair form one sequence; a warpgroup takes every fourth one.
        const int wg = warp >> 2, r = (warp & 3) * 32 + lane;
        const uint32_t full0 = gp_mapa(w_full, 0);
        const int spg_shift = p.spg == 4 ? 2 : 1;
        const bool row_on = r < half;              // (the others only arrive)
        for (int it = wg; it < stages; it += GP_DWGS) {
            const int slot = it % GP_WSLOTS, group = it >> spg_shift, in = it & (p.spg - 1);
            const int turn = p.spg == 4 ? group / 3 : group / 4, pslot = group - turn * (int)pslots;
            const uint32_t dst = w_ring + slot * GP_SLOT + r * 16, src = p_ring + pslot * pbytes;
            if (ok && !gp_wait(p_full + 8 * pslot, (uint32_t)turn & 1u, dead)) ok = false;
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            uint32_t w[2][S];
            unsigned short c[4] = {};
            if (row_on) {
                uint32_t cx, cy;
                asm volatile("ld.shared.v2.b32 {%0,%1}, [%2];" : "=r"(cx), "=r"(cy) : "r"(src + coef_at + r * 8) : "memory");
                c[0] = (unsigned short)cx, c[1] = (unsigned short)(cx >> 16), c[2] = (unsigned short)cy, c[3] = (unsigned short)(cy >> 16);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const uint32_t at = src + (uint32_t)(((2 * in + h) * half + r) * S * 4);
                    if constexpr (S == 4)
                        asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(w[h][0]), "=r"(w[h][1]), "=r"(w[h][2]), "=r"(w[h][3]) : "r"(at) : "memory");
                    else
#pragma unroll
                        for (int s = 0; s < S; ++s) asm volatile("ld.shared.b32 %0, [%1];" : "=r"(w[h][s]) : "r"(at + 4 * s) : "memory");
                }
            } else {
#pragma unroll
                for (int s = 0; s < S; ++s) w[0][s] = w[1][s] = 0u;
            }
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(p_empty + 8 * pslot) : "memory");
            // See linear_gemm.cu: a lone bit at position 10 .. 14 of a half is a power of two; a mask and an HFMA2 add c_s to the
            // pair (j, j + 16) where their bits are set.  |c_s| >= 3.9 takes the sign-flip form.
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
            const bool flip = __any_sync(0xffffffffu, big);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                __half2 acc[16];
                if (!flip) {
#pragma unroll
                    for (int j = 0; j < 16; ++j) acc[j] = __float2half2_rn(0.0f);
#pragma unroll
                    for (int s = 0; s < S; ++s) {
                        const uint32_t v0 = w[h][s] << 10, v1 = w[h][s] << 5, v2 = w[h][s], v3 = w[h][s] >> 1;
#pragma unroll
                        for (int j = 0; j < 16; ++j) {
                            const uint32_t v = (j < 5) ? v0 : (j < 10) ? v1 : (j < 15) ? v2 : v3;
                            const int pos = (j < 15) ? j % 5 : 4;
                            const uint32_t t = v & (0x04000400u << pos);
                            acc[j] = __hfma2(*reinterpret_cast<const __half2*>(&t), mul[s][pos], acc[j]);
                        }
                    }
                } else {
                    uint32_t hc[S];                // (c_s / 2, c_s / 2)
                    float sum = 0.0f;
#pragma unroll
                    for (int s = 0; s < S; ++s) {
                        const float chf = __half2float(__ushort_as_half(c[s])) * 0.5f;
                        sum += chf;
                        const uint32_t hb = (uint32_t)__half_as_ushort(__float2half_rn(chf));
                        hc[s] = hb | (hb << 16);
                    }
                    const __half2 base2 = __half2half2(__float2half_rn(sum));
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        acc[j] = base2;
#pragma unroll
                        for (int s = 0; s < S; ++s) {
                            const uint32_t t = (~(w[h][s] << (15 - j)) & 0x80008000u) ^ hc[s];
                            acc[j] = __hadd2(acc[j], *reinterpret_cast<const __half2*>(&t));
                        }
                    }
                }
                // the slot is waited for with the values in registers
                if (h == 0) {
                    if (ok && !gp_wait(w_empty + 8 * slot, ((uint32_t)(it / GP_WSLOTS) & 1u) ^ 1u, dead)) ok = false;
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;                // (out of the two halves; the stage loop ends below)
                }
                if (row_on) {
                    const uint32_t* a = reinterpret_cast<const uint32_t*>(acc);
#pragma unroll
                    for (int kc = 0; kc < 4; ++kc) {           // eight k each: the lower halves of acc[0 .. 7], [8 .. 15], then the upper ones
                        const uint32_t* f = a + 8 * (kc & 1);
                        const uint32_t sel = kc < 2 ? 0x5410u : 0x7632u;
                        asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(dst + (4 * h + kc) * 2048), "r"(__byte_perm(f[0], f[1], sel)),
                                     "r"(__byte_perm(f[2], f[3], sel)), "r"(__byte_perm(f[4], f[5], sel)), "r"(__byte_perm(f[6], f[7], sel))
                                     : "memory");
                    }
                }
            }
            if (!ok) break;
            fence_proxy_async();                   // the MMAs read through the asynchronous proxy
            __syncwarp();
            if (lane == 0) gp_arrive(full0 + 8 * slot);
        }
        if (!ok && lane == 0) {
            *dead = 1;
            atomicExch(p.status, 1u);
            atomicExch(p.status + 1, 0xC00u + blockIdx.x);
        }
    }
    // ------------------------------ teardown ------------------------------
    // Neither CTA leaves while the other may still arrive at its barriers, read its shared memory or write its tensor memory.
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    gp_cluster_sync();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp == GP_XWARP)
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tbase), "r"(512u) : "memory");
}

// ---------------------------------------------------------------------------------------------
// host
// ---------------------------------------------------------------------------------------------
// The parts of the split items, added in the order of K: a warp has 32 activation rows x 8 weight rows, a row per lane, four parts' loads at a
// time (a warp per 32 x 32, part after part: 3000 x 28672 x 4096, whose six left-over items have thirteen parts each, 514 us, now 509; 2048 x
// 14336 x 4096 187.3, 184.7).
__global__ void __launch_bounds__(128) gp_add_kernel(const GpParams p, int pairs) {
    pdl_launch_dependents();
    pdl_wait();
    const int lane = threadIdx.x & 31, chunks = (p.n + 31) / 32;
    TsSegs sg;
    sg.init(p.items, p.steps, (unsigned int)pairs, 0u);
    const int job = (int)blockIdx.x * 4 + (threadIdx.x >> 5);
    const int quarter = job & 3, chunk = job / 4 % chunks, unit = job / 4 / chunks % 16, rt = job / 4 / chunks / 16;
    const int item = sg.rem_tile0 + rt;
    if (item >= p.items) return;
    const int c0 = sg.cta_of((unsigned int)(rt * sg.KBS)), parts = sg.cta_of((unsigned int)(rt * sg.KBS + sg.KBS - 1)) - c0 + 1;
    const int m = gp_m(p, item) * 512 + (unit >> 3) * 256 + (unit & 7) * 32 + lane, col = chunk * 32 + quarter * 8, n = gp_n0(p, item) + col;
    if (parts == 1 || m - lane >= p.M || col >= p.n || n >= p.N) return;       // one pair has done the item alone; past the last
    const float4* src = gp_part(p.part, p.n, c0 + rt, unit, chunk) + quarter * 64 + lane;
    const size_t step = gp_part(p.part, p.n, 1, 0, 0) - gp_part(p.part, p.n, 0, 0, 0);
    float4 a = make_float4(0.0f, 0.0f, 0.0f, 0.0f), b = a;
    for (int c = 0; c < parts; c += 4) {
        float4 t[4][2];
#pragma unroll
        for (int h = 0; h < 4; ++h) {
            t[h][0] = t[h][1] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (c + h < parts) t[h][0] = __ldcg(src + h * step), t[h][1] = __ldcg(src + h * step + 32);
        }
        src += 4 * step;
#pragma unroll
        for (int h = 0; h < 4; ++h) {
            a.x += t[h][0].x, a.y += t[h][0].y, a.z += t[h][0].z, a.w += t[h][0].w;
            b.x += t[h][1].x, b.y += t[h][1].y, b.z += t[h][1].z, b.w += t[h][1].w;
        }
    }
    if (m >= p.M) return;
    float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    uint32_t h[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        if (p.bias) v[2 * i] += __half2float(__ldg(p.bias + n + 2 * i)), v[2 * i + 1] += __half2float(__ldg(p.bias + n + 2 * i + 1));
        const __half2 r = __floats2half2_rn(v[2 * i], v[2 * i + 1]);
        h[i] = *reinterpret_cast<const uint32_t*>(&r);
    }
    *reinterpret_cast<uint4*>(p.y + (size_t)m * p.N + n) = make_uint4(h[0], h[1], h[2], h[3]);
}

struct GpPlan {
    int n, items, pairs, steps;  // steps: of an item, in the split over the pairs
    size_t part_bytes;
    long long ns;
};

// Weight rows of an item, and whether the items that are left over after whole rounds are split over K: the least time in ns, by these
// figures (see also gm_many_ns, linear_gemm.cu).  A 64-k stage of two blocks takes 160 + 20 S + 2.15 n (790 at n = 256, S = 4), at least 560: the way of
// three stages of activations through L2 and back; runs of 50 to 300 us up to an eighth more (the power limit).  A launch takes 3 100, a round's ends
// 2 000 + 7 n, the last one's 21 n where all pairs have an item.  A split adds a launch, 6 300, and 0.25 per KB of parts out and back.
// The scratch it may count on is what sbvr_workspace_bytes promises, whatever the workspace has grown to for other calls.
static long long gp_run_ns(long long t) { return t + t / 8 * std::min(std::max(t - 50000, 0LL), 250000LL) / 250000; }
static GpPlan gp_plan(const PackedW& w, int M, int sm_count, int device, size_t scratch) {
    size_t promised = 0;
    if (sbvr_workspace_bytes(device, M, w.N, w.K, &promised) != SBVR_OK) promised = SBVR_WS_FIXED_BYTES;
    scratch = std::min(scratch, promised - SBVR_WS_FIXED_BYTES);
    const long long pairs = sm_count / 2, MT = (M + 511) / 512, NG = w.K / w.G, stages = w.K / 64;
    const bool odd = M > 512 && (M - 1) / 256 % 2 == 0;        // the last activation tile has one block
    GpPlan best = {};
    for (int n = 256; n >= 64; n -= 16) {
        const long long stage = std::max(560, 160 + 20 * w.S + 215 * n / 100), half = std::max(stage * 6 / 10, 150LL + 50 * w.S);
        const long long NT = (w.N + n - 1) / n, items = NT * MT, full = odd ? items - NT : items, rounds = (items + pairs - 1) / pairs, left = items % pairs;
        if (items > (1 << 20)) continue;
        const long long long_ones = (full + pairs - 1) / pairs;                // rounds in which the first pair has an item of two blocks
        const long long end = 2000 + 7 * n;
        GpPlan pl = {n, (int)items, (int)std::min(items, pairs), 1, 0, 0};
        pl.ns = gp_run_ns(stages * (long_ones * stage + (rounds - long_ones) * half)) + (rounds - 1) * end +
                21 * n * (items - (rounds - 1) * pairs) / pairs + 3100;
        if (!best.n || pl.ns < best.ns) best = pl;
        if (left * NG < pairs || left * NG * pairs >= (1LL << 32)) continue;
        pl.part_bytes = (size_t)(pairs + left) * 16 * ((n + 31) / 32) * 4096;
        pl.pairs = (int)pairs, pl.steps = (int)NG;
        const long long whole = items / pairs, whole_long = std::min(whole, long_ones);
        pl.ns = gp_run_ns(stages * (whole_long * stage + (whole - whole_long) * half) +
                          (left * stages + pairs - 1) / pairs * (full > whole * pairs ? stage : half)) +  // (cut by steps, long and short)
                whole * end + 9400 + (long long)(pl.part_bytes / 4000);
        if (pl.part_bytes <= scratch && pl.ns < best.ns) best = pl;
    }
    return best;
}

bool linear_pair_supported(const __half* x, int Kin, const PackedW& w, const __half* y, int M) {
    return M > 256 && w.N <= (1 << 24) && w.S >= 2 && w.S <= 4 && (w.G == 256 || w.G == 128) && w.N % 128 == 0 && w.K % 64 == 0 && Kin % 8 == 0 &&
           !((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y)) & 15) &&
           !(reinterpret_cast<uintptr_t>(w.bvr) & 15);
}

long long linear_pair_ns(const PackedW& w, int M, int sm_count, int device, size_t scratch) {
    return gp_plan(w, M, sm_count, device, scratch).ns;
}

template <int S>
static int gp_launch(const CUtensorMap& xmap, const GpParams& p, int pairs, cudaStream_t st) {
    static SmemOnce once;
    const int rc = set_max_smem_once(once, linear_pair_kernel<S>, GP_SMEM);
    if (rc) return rc;
    SBVR_CUDA_TRY(launch_pdl_cluster(linear_pair_kernel<S>, dim3(2 * pairs), dim3(GP_THREADS), 2, (size_t)GP_SMEM, st, xmap, p));
    return SBVR_OK;
}

int launch_linear_pair(const __half* x, int Kin, const PackedW& w, const __half* bias, __half* y, int M, unsigned int* status,
                       char* scratch, size_t scratch_bytes, int sm_count, int device, cudaStream_t st) {
    CUtensorMap xmap;
    int rc = ts_map_2d(&xmap, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, CU_TENSOR_MAP_SWIZZLE_128B, x, (size_t)M, (size_t)Kin, (size_t)Kin * 2, 128, 64);
    if (rc) return rc;
    const GpPlan pl = gp_plan(w, M, sm_count, device, scratch_bytes);
    GpParams p;
    p.bvr = w.bvr, p.idx = w.idx, p.coeff = w.coeff, p.bias = bias, p.y = y, p.status = status;
    p.M = M, p.N = w.N, p.idx_bytes = w.idx_bytes, p.n = pl.n;
    p.vec = !(reinterpret_cast<uintptr_t>(w.coeff) & (2 * w.S - 1));
    p.MB = (M + 255) / 256, p.MT = (p.MB + 1) / 2;
    p.MF = p.MB % 2 && p.MT > 1 ? p.MT - 1 : p.MT;
    p.items = pl.items, p.full = pl.items / p.MT * p.MF;
    p.NG = w.K / w.G, p.spg = w.G / 64, p.steps = pl.steps;
    p.part = reinterpret_cast<float*>(scratch);
    switch (w.S) {
        case 2: rc = gp_launch<2>(xmap, p, pl.pairs, st); break;
        case 3: rc = gp_launch<3>(xmap, p, pl.pairs, st); break;
        default: rc = gp_launch<4>(xmap, p, pl.pairs, st);
    }
    if (rc || !pl.part_bytes) return rc;
    const int jobs = pl.items % pl.pairs * 16 * ((pl.n + 31) / 32) * 4;
    SBVR_CUDA_TRY(launch_pdl(gp_add_kernel, dim3((jobs + 3) / 4), dim3(128), 0, st, p, pl.pairs));
    return SBVR_OK;
}

}  // namespace sbvr
