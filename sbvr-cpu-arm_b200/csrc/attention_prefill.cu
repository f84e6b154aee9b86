// Causal prefill attention on the fifth-generation tensor cores; head_dim 128, the R = n_heads / n_kv query heads of a KV head together.
//
// A CTA takes 128 (query token, query head) pairs that share one KV head (128 / R consecutive tokens of a sequence x its R heads) and walks
// the keys 64 at a time.
//
//   scores   S[128 pairs, 64 keys] = q . k, both from shared memory (128-byte swizzle), fp32 in tensor memory; scaled in fp32
//   weights  a thread per pair: exp2 in fp32 of S less a reference; each weight is split into two fp16 parts (p = hi + lo to 2^-22), so
//            that the probabilities keep their fp32 precision, and stored over S
//   output   O[128 pairs, 128 dims] += hi . V + lo . V, weights from tensor memory, V (keys x dims as it lies in the cache) from shared
//            memory
//
// The reference of a pair is the largest score it has met, but follows it only when that has grown by more than 2^8: then its sums (in
// tensor memory, and the sum of its weights) are scaled.  Weights are at most 2^8 instead of 1, which fp16's exponent holds; every other
// time the output is not touched by the threads.
//
// Seven warps: 0-3 weights, 4 issues the MMAs (one lane), 5 and 6 bring K and V (whole tiles by TMA, the last one by cp.async with zeros past
// the last key).  S and the weights of two
// tiles (64 columns each) and O take 256 columns of tensor memory, 97 KB of shared memory: two CTAs per SM, so that one computes weights while
// the other has the tensor pipe.  Tensor memory is only asked for when the kernel in front has ended, and the kernel behind may start only
// when this one has it: neither can wait for columns that the other holds while the other waits for it to end.  Every wait is bounded; a CTA in
// which one runs out multiplies its pairs out without the tensor cores.
//
// What bounds it: the weights, about 600 instructions and 64 exponentials per thread and tile, on two warps per scheduler; the tensor pipe
// would take 768 cycles a tile, 26 us at 2 x 1500 tokens.  Per layer, 32 query heads, 8 KV heads, us (mma.sync on blocks of 64, in
// brackets): 2 x 1500 tokens 59 (157), 1 x 4000 162 (505), 8 x 256 22 (35), 1 x 512 14 (23).  (With whole tiles by cp.async, too, 63 and 173; with
// K and V on their way before the queries are staged 60 and 164.)
#include "common.cuh"
#include "tc_stream.cuh"

namespace sbvr {

constexpr int AQ_D = 128, AQ_ROWS = 128, AQ_KEYS = 64;
constexpr int AQ_IWARP = 4, AQ_KWARP = 5, AQ_VWARP = 6, AQ_THREADS = 7 * 32;
constexpr uint32_t AQ_QBOX = AQ_ROWS * 128, AQ_KBOX = AQ_KEYS * 128, AQ_TILE = 2 * AQ_KBOX;    // boxes of 64 dims, a tile of K or V
constexpr int AQ_HDR = 1024;
constexpr int AQ_SMEM = AQ_HDR + 2 * (int)AQ_QBOX + 4 * (int)AQ_TILE;
constexpr uint32_t AQ_COLS = 256, AQ_O_COL = 128;

struct AqParams {
    const __half* qkv;
    const __half* kcache;
    const __half* vcache;
    const int* positions;
    __half* out;
    int tokens_per_seq, n_heads, n_kv, max_ctx, r_shift;
    float scale;
};

__device__ __forceinline__ void aq_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void aq_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void aq_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// Descriptors, version 1, 128-byte swizzle, 1024 B between groups of eight rows.  Q and K: rows along M and N, contraction contiguous.  V:
// rows along the contraction; AQ_KBOX between its boxes of 64 dims.
constexpr uint32_t AQ_DESC_HI = (1024u >> 4) | (1u << 14) | (2u << 29);
__device__ __forceinline__ void aq_mma_ss(uint32_t d, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 a, b;\n\tsetp.ne.b32 p, %4, 0;\n\tmov.b64 a, {%1, %5};\n\tmov.b64 b, {%2, %5};\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, p;\n\t}" ::"r"(d),
        "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(accumulate), "r"(AQ_DESC_HI)
        : "memory");
}
__device__ __forceinline__ void aq_mma_ts(uint32_t d, uint32_t a, uint32_t b_lo, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 b;\n\tsetp.ne.b32 p, %4, 0;\n\tmov.b64 b, {%2, %5};\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], b, %3, p;\n\t}" ::"r"(d),
        "r"(a), "r"(b_lo), "r"(idesc), "r"(accumulate), "r"(AQ_DESC_HI)
        : "memory");
}
__device__ __forceinline__ void aq_ld32(uint32_t taddr, uint32_t* r) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
        "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}
// the loads into r[0 .. 31] have come (the registers depend on it)
__device__ __forceinline__ void aq_ld_wait(uint32_t* r) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]), "+r"(r[8]),
                   "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]), "+r"(r[15])
                 :
                 : "memory");
    asm volatile(""
                 : "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]), "+r"(r[22]), "+r"(r[23]), "+r"(r[24]),
                   "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]), "+r"(r[29]), "+r"(r[30]), "+r"(r[31])
                 :
                 : "memory");
}
__device__ __forceinline__ void aq_st32(uint32_t taddr, const uint32_t* a) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
        "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};" ::"r"(taddr),
        "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]), "r"(a[7]), "r"(a[8]), "r"(a[9]),
        "r"(a[10]), "r"(a[11]), "r"(a[12]), "r"(a[13]), "r"(a[14]), "r"(a[15]), "r"(a[16]), "r"(a[17]), "r"(a[18]),
        "r"(a[19]), "r"(a[20]), "r"(a[21]), "r"(a[22]), "r"(a[23]), "r"(a[24]), "r"(a[25]), "r"(a[26]), "r"(a[27]),
        "r"(a[28]), "r"(a[29]), "r"(a[30]), "r"(a[31])
        : "memory");
}
__device__ __forceinline__ void aq_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ float aq_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// A CTA in which a wait has run out, or among whose keys values are not finite that only some of its tokens attend to: all of its pairs (once
// more), a warp each, four dims a lane, key by key as far as the token goes.
__device__ __noinline__ void aq_multiply_out(const AqParams& p, uint32_t q_s, const int* ctx_s, int t0, int nq, int seq, int kvh) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, R = 1 << p.r_shift;
    const float sl2 = (p.scale == 0.0f ? 1.0f : fabsf(p.scale)) * 1.4426950408889634f;
    const size_t at = ((size_t)seq * p.n_kv + kvh) * p.max_ctx * AQ_D + lane * 4;
    auto four = [](const uint2& v, float (&f)[4]) {
        const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&v.x)), b = __half22float2(*reinterpret_cast<const __half2*>(&v.y));
        f[0] = a.x, f[1] = a.y, f[2] = b.x, f[3] = b.y;
    };
    for (int row = warp; row < nq * R; row += AQ_THREADS / 32) {
        const int j = row >> p.r_shift, ctx = ctx_s[j], ch = lane >> 1;
        uint2 v;
        asm volatile("ld.shared.v2.b32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y)
                     : "r"(q_s + (ch >> 3) * AQ_QBOX + row * 128 + (((ch & 7) ^ (row & 7)) << 4) + (lane & 1) * 8)
                     : "memory");
        float q[4], o[4] = {0.0f, 0.0f, 0.0f, 0.0f}, ref = -INFINITY, sum = 0.0f;
        four(v, q);
        for (int key = 0; key < ctx; ++key) {
            float k[4], w[4];
            four(*reinterpret_cast<const uint2*>(p.kcache + at + (size_t)key * AQ_D), k);
            four(*reinterpret_cast<const uint2*>(p.vcache + at + (size_t)key * AQ_D), w);
            float s = q[0] * k[0] + q[1] * k[1] + q[2] * k[2] + q[3] * k[3];
#pragma unroll
            for (int m = 16; m; m >>= 1) s += __shfl_xor_sync(0xffffffffu, s, m);
            const float top = fmaxf(ref, s), base = top == -INFINITY ? 0.0f : top * sl2;
            const float corr = ref == -INFINITY ? 0.0f : aq_exp2(ref * sl2 - base), e = aq_exp2(s * sl2 - base);
            ref = top;
            sum = sum * corr + e;
#pragma unroll
            for (int i = 0; i < 4; ++i) o[i] = o[i] * corr + e * w[i];
        }
        const float inv = sum > 0.0f ? 1.0f / sum : 0.0f;
        const __half2 a = __floats2half2_rn(o[0] * inv, o[1] * inv), b = __floats2half2_rn(o[2] * inv, o[3] * inv);
        *reinterpret_cast<uint2*>(p.out + ((size_t)(t0 + j) * p.n_heads + kvh * R + (row & (R - 1))) * AQ_D + lane * 4) =
            make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
    }
}

__global__ void __launch_bounds__(AQ_THREADS, 2) attention_tc_kernel(const __grid_constant__ CUtensorMap kmap,
                                                                         const __grid_constant__ CUtensorMap vmap, const AqParams p) {
    extern __shared__ __align__(1024) unsigned char smem[];
    uint64_t* k_full = reinterpret_cast<uint64_t*>(smem);        // [2] a tile of K is in shared memory
    uint64_t* v_full = k_full + 2;                               // [2] of V
    uint64_t* s_full = k_full + 4;                               // [2] scores are there, the tile of K is read
    uint64_t* v_empty = k_full + 6;                              // [2] O has a tile's products, the tile of V is read
    uint64_t* p_full = k_full + 8;                               // [2] weights are stored
    uint64_t* drained = k_full + 10;                             // after a time-out
    volatile int* dead_s = reinterpret_cast<volatile int*>(smem + 128);
    uint32_t* tmem_s = reinterpret_cast<uint32_t*>(smem + 132);
    volatile int* odd_s = reinterpret_cast<volatile int*>(smem + 136);
    int* ctx_s = reinterpret_cast<int*>(smem + 256);             // [128 / R]
    const uint32_t q_s = smem_u32(smem) + AQ_HDR, k_s = q_s + 2 * AQ_QBOX, v_s = k_s + 2 * AQ_TILE;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int R = 1 << p.r_shift, QT = AQ_ROWS >> p.r_shift;
    const int nblk = (p.tokens_per_seq + QT - 1) / QT;
    const int per = (int)gridDim.x / nblk;                       // sequences * n_kv
    const int rest = blockIdx.x % per, qblk = nblk - 1 - (int)blockIdx.x / per;      // longest contexts first
    const int kvh = rest % p.n_kv, seq = rest / p.n_kv;
    const int t0 = seq * p.tokens_per_seq + qblk * QT;
    const int nq = min(QT, p.tokens_per_seq - qblk * QT);
    if (threadIdx.x == 0) {
        for (int i = 0; i < 2; ++i) {
            mbar_init(k_full + i, 32);
            mbar_init(v_full + i, 32);
            mbar_init(s_full + i, 1);
            mbar_init(v_empty + i, 1);
            mbar_init(p_full + i, 4);
        }
        mbar_init(drained, 1);
        *dead_s = 0, *odd_s = 0;
        fence_mbar_init();
    }
    pdl_wait();
    if (warp == AQ_IWARP) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_s)), "r"(AQ_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        pdl_launch_dependents();                                 // (one warp's says it for the CTA)
        aq_fence_before();
    }
    for (int j = threadIdx.x; j < QT; j += AQ_THREADS) ctx_s[j] = (j < nq) ? min(p.positions[t0 + j] + 1, p.max_ctx) : 0;
    // queries; their signs as in attention_prefill_kernel: the running maximum is that of the unscaled scores
    const size_t tok_pitch = (size_t)(p.n_heads + 2 * p.n_kv) * AQ_D;
    for (int c = threadIdx.x; c < AQ_ROWS * 16; c += AQ_THREADS) {
        const int row = c >> 4, ch = c & 15, j = row >> p.r_shift, r = row & (R - 1);
        uint4 v = *reinterpret_cast<const uint4*>(p.qkv + (size_t)(t0 + min(j, nq - 1)) * tok_pitch + (size_t)(kvh * R + r) * AQ_D + ch * 8);
        if (p.scale < 0.0f) v.x ^= 0x80008000u, v.y ^= 0x80008000u, v.z ^= 0x80008000u, v.w ^= 0x80008000u;
        if (p.scale == 0.0f) v = make_uint4(0u, 0u, 0u, 0u);
        asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(q_s + (ch >> 3) * AQ_QBOX + row * 128 + (((ch & 7) ^ (row & 7)) << 4)),
                     "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w)
                     : "memory");
    }
    fence_proxy_async();                                         // the MMAs read through the asynchronous proxy
    __syncthreads();
    aq_fence_after();
    const uint32_t tbase = *tmem_s;
    int P = 0, pmin = 0x7fffffff;                                // keys any token of the CTA attends to, and every one
    for (int j = lane; j < nq; j += 32) P = max(P, ctx_s[j]), pmin = min(pmin, ctx_s[j]);
    P = __reduce_max_sync(0xffffffffu, P), pmin = __reduce_min_sync(0xffffffffu, pmin);
    const int ntile = (P + AQ_KEYS - 1) / AQ_KEYS;
    bool ok = true;

    if (warp == AQ_KWARP || warp == AQ_VWARP) {
        // ------------------------------ K, V ------------------------------
        const bool is_k = warp == AQ_KWARP;
        const __half* base = (is_k ? p.kcache : p.vcache) + ((size_t)seq * p.n_kv + kvh) * p.max_ctx * AQ_D + (lane & 15) * 8;
        uint64_t* empty = is_k ? s_full : v_empty;
        uint64_t* full = is_k ? k_full : v_full;
        const uint32_t ring = (is_k ? k_s : v_s) + ((lane & 15) >> 3) * AQ_KBOX;
        for (int t = 0; t < ntile; ++t) {
            const int b = t & 1;
            if (t >= 2 && (*dead_s || !mbar_wait_timed(empty + b, (uint32_t)((t - 2) >> 1) & 1u))) ok = false;
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            if ((t + 1) * AQ_KEYS <= P) {                        // a whole tile
                if (lane == 0) {
                    mbar_arrive_expect_tx(full + b, AQ_TILE);
                    unsigned char* dst = smem + AQ_HDR + 2 * AQ_QBOX + ((is_k ? 0 : 2) + b) * AQ_TILE;
                    const int y = (seq * p.n_kv + kvh) * p.max_ctx + t * AQ_KEYS;
                    ts_tma_2d(dst, is_k ? &kmap : &vmap, 0, y, full + b);
                    ts_tma_2d(dst + AQ_KBOX, is_k ? &kmap : &vmap, 64, y, full + b);
                } else {
                    mbar_arrive(full + b);
                }
            } else {
#pragma unroll 4
                for (int i = 0; i < AQ_KEYS / 2; ++i) {              // two rows at a time, a 16-byte chunk per lane
                    const int row = 2 * i + (lane >> 4), key = t * AQ_KEYS + row;
                    const bool on = key < P;
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(ring + b * AQ_TILE + row * 128 + (((lane & 7) ^ (row & 7)) << 4)),
                                 "l"(base + (size_t)(on ? key : 0) * AQ_D), "r"(on ? 16u : 0u)
                                 : "memory");
                }
                asm volatile("cp.async.wait_all;" ::: "memory");
                fence_proxy_async();
                mbar_arrive(full + b);
            }
            if (!is_k && (t + 1) * AQ_KEYS > pmin) {             // keys that not every token attends to: a weight of zero hides finite values only
                uint32_t any = 0;
                if (!mbar_wait_timed(full + b, (uint32_t)(t >> 1) & 1u)) ok = false;
#pragma unroll 4
                for (int i = 0; i < AQ_KEYS / 2; ++i) {
                    const int row = 2 * i + (lane >> 4);
                    uint32_t v[4];
                    asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3])
                                 : "r"(ring + b * AQ_TILE + row * 128 + (((lane & 7) ^ (row & 7)) << 4))
                                 : "memory");
#pragma unroll
                    for (int e = 0; e < 4; ++e) any |= (v[e] & 0x7c007c00u) + 0x04000400u;     // (an exponent of all ones: bit 15)
                }
                if (any & 0x80008000u) *odd_s = 1;
                fence_proxy_async();                             // read before the next copy writes there
                __syncwarp();
            }
        }
        if (!ok) *dead_s = 1;
    } else if (warp == AQ_IWARP) {
        // ------------------------------ MMA issuer ------------------------------
        if (elect_one()) {
            constexpr uint32_t QK = (1u << 4) | ((AQ_KEYS >> 3) << 17) | ((AQ_ROWS >> 4) << 24);
            constexpr uint32_t PV = (1u << 4) | (1u << 16) | ((AQ_D >> 3) << 17) | ((AQ_ROWS >> 4) << 24);      // (bit 16: B is V as it lies)
            const uint32_t qd = (q_s >> 4) | (1u << 16), kd = (k_s >> 4) | (1u << 16), vd = (v_s >> 4) | ((AQ_KBOX >> 4) << 16);
            auto scores = [&](int t) {
                const int b = t & 1;
                if (*dead_s || !mbar_wait_timed(k_full + b, (uint32_t)(t >> 1) & 1u)) return false;
                aq_fence_after();
#pragma unroll
                for (int k = 0; k < 8; ++k)
                    aq_mma_ss(tbase + b * 64, qd + (k >> 2) * (AQ_QBOX >> 4) + (k & 3) * 2,
                              kd + b * (AQ_TILE >> 4) + (k >> 2) * (AQ_KBOX >> 4) + (k & 3) * 2, QK, k ? 1u : 0u);
                aq_commit(s_full + b);
                return true;
            };
            if (ntile) ok = scores(0);
            for (int t = 0; t < ntile && ok; ++t) {
                const int b = t & 1;
                const uint32_t ph = (uint32_t)(t >> 1) & 1u;
                // (S of the next tile lies over the weights of the tile before: their MMAs are in front of it)
                if (t + 1 < ntile && !scores(t + 1)) ok = false;
                if (ok && !(mbar_wait_timed(v_full + b, ph) && mbar_wait_timed(p_full + b, ph))) ok = false;
                if (!ok) break;
                aq_fence_after();
#pragma unroll
                for (int k = 0; k < 4; ++k) {                    // sixteen keys: 2 KB of V, eight columns of weights
                    const uint32_t v = vd + b * (AQ_TILE >> 4) + k * 128;
                    aq_mma_ts(tbase + AQ_O_COL, tbase + b * 64 + k * 8, v, PV, (t | k) ? 1u : 0u);
                    aq_mma_ts(tbase + AQ_O_COL, tbase + b * 64 + 32 + k * 8, v, PV, 1u);
                }
                aq_commit(v_empty + b);
            }
            if (!ok) {                                           // MMAs that were issued end before the CTA leaves
                *dead_s = 1;
                const long long c0 = clock64();
                aq_commit(drained);
                while (!mbar_test(drained, 0u) && clock64() - c0 < 200000000LL) {}
            }
        }
        __syncwarp();
    } else {
        // ------------------------------ weights ------------------------------
        const int row = warp * 32 + lane, j = row >> p.r_shift;
        const int ctx = ctx_s[j];
        const int wctx = __reduce_min_sync(0xffffffffu, j < nq ? ctx : 0x7fffffff);          // (rows past the last: anything finite)
        const uint32_t mine = tbase + ((uint32_t)(warp * 32) << 16);
        const float sl2 = (p.scale == 0.0f ? 1.0f : fabsf(p.scale)) * 1.4426950408889634f;
        float ref = -INFINITY, sum = 0.0f;
        for (int t = 0; t < ntile; ++t) {
            const int b = t & 1;
            if (*dead_s || !mbar_wait_timed(s_full + b, (uint32_t)(t >> 1) & 1u)) ok = false;
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            aq_fence_after();
            uint32_t u[64];
            aq_ld32(mine + b * 64, u);
            aq_ld32(mine + b * 64 + 32, u + 32);
            aq_ld_wait(u);
            aq_ld_wait(u + 32);
            if ((t + 1) * AQ_KEYS > wctx) {                      // some token's context ends inside or before this tile
#pragma unroll
                for (int i = 0; i < 64; ++i)
                    if (t * AQ_KEYS + i >= ctx) u[i] = 0xff800000u;
            }
            float m4[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) m4[i] = __uint_as_float(u[i]);
#pragma unroll
            for (int i = 4; i < 64; ++i) m4[i & 3] = fmaxf(m4[i & 3], __uint_as_float(u[i]));
            const float m = fmaxf(ref, fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3])));
            if (__any_sync(0xffffffffu, (m - ref) * sl2 > 8.0f)) {
                const float corr = ref == -INFINITY ? 0.0f : aq_exp2((ref - m) * sl2);
                ref = m;
                sum *= corr;
                if (t > 0) {
                    if (!mbar_wait_timed(v_empty + (b ^ 1), (uint32_t)((t - 1) >> 1) & 1u)) ok = false;
                    ok = __all_sync(0xffffffffu, ok);
                    if (!ok) break;
                    aq_fence_after();
#pragma unroll 1
                    for (int c = 0; c < 4; ++c) {
                        uint32_t o[32];
                        aq_ld32(mine + AQ_O_COL + c * 32, o);
                        aq_ld_wait(o);
#pragma unroll
                        for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * corr);
                        aq_st32(mine + AQ_O_COL + c * 32, o);
                    }
                }
            }
            const float base = ref == -INFINITY ? 0.0f : ref * sl2;            // a row without any key so far
            float s4[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            uint32_t hi[32], lo[32];
#pragma unroll
            for (int i = 0; i < 32; ++i) {
                const float a = aq_exp2(fmaf(__uint_as_float(u[2 * i]), sl2, -base)), c = aq_exp2(fmaf(__uint_as_float(u[2 * i + 1]), sl2, -base));
                s4[(2 * i) & 3] += a, s4[(2 * i + 1) & 3] += c;
                const __half2 h = __floats2half2_rn(a, c);
                const float2 f = __half22float2(h);
                const __half2 l = __floats2half2_rn(a - f.x, c - f.y);
                hi[i] = *reinterpret_cast<const uint32_t*>(&h), lo[i] = *reinterpret_cast<const uint32_t*>(&l);
            }
            sum += (s4[0] + s4[1]) + (s4[2] + s4[3]);
            aq_st32(mine + b * 64, hi);
            aq_st32(mine + b * 64 + 32, lo);
            aq_st_wait();
            aq_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(p_full + b);
        }
        if (ok && ntile && !mbar_wait_timed(v_empty + ((ntile - 1) & 1), (uint32_t)((ntile - 1) >> 1) & 1u)) ok = false;
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) *dead_s = 1;
        aq_fence_after();
        const float inv = sum > 0.0f ? 1.0f / sum : 0.0f;
        __half* dst = p.out + ((size_t)(t0 + min(j, nq - 1)) * p.n_heads + kvh * R + (row & (R - 1))) * AQ_D;
#pragma unroll 1
        for (int c = 0; c < 4 && ok; ++c) {
            uint32_t o[32];
            aq_ld32(mine + AQ_O_COL + c * 32, o);
            aq_ld_wait(o);
            if (!ntile) {                                        // no key at all: nothing was written there
#pragma unroll
                for (int i = 0; i < 32; ++i) o[i] = 0u;
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                uint32_t h[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const __half2 v = __floats2half2_rn(__uint_as_float(o[8 * i + 2 * e]) * inv, __uint_as_float(o[8 * i + 2 * e + 1]) * inv);
                    h[e] = *reinterpret_cast<const uint32_t*>(&v);
                }
                if (j < nq) *reinterpret_cast<uint4*>(dst + c * 32 + i * 8) = make_uint4(h[0], h[1], h[2], h[3]);
            }
            __syncwarp();
        }
        aq_fence_before();
    }
    // ------------------------------ teardown ------------------------------
    __syncthreads();
    aq_fence_after();
    if (*dead_s) {                                               // copies that were issued land before the CTA leaves
        const long long c0 = clock64();
        while (clock64() - c0 < (1LL << 22)) {}
    }
    if (*odd_s || *dead_s) aq_multiply_out(p, q_s, ctx_s, t0, nq, seq, kvh);
    if (warp == AQ_IWARP) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tbase), "r"(AQ_COLS) : "memory");
}

bool attention_tc_supported(const void* qkv, const void* out, int tokens, int tokens_per_seq, int n_kv, int R, int sm_count) {
    if ((reinterpret_cast<uintptr_t>(qkv) | reinterpret_cast<uintptr_t>(out)) & 15) return false;
    return attention_tc_faster((long long)(tokens / tokens_per_seq) * n_kv * (((long long)tokens_per_seq * R + 63) / 64), tokens_per_seq, sm_count);
}

int launch_attention_tc(const __half* qkv, const __half* kcache, const __half* vcache, const int* positions, __half* out, int tokens,
                        int tokens_per_seq, int n_heads, int n_kv, int max_ctx, float scale, cudaStream_t st) {
    static SmemOnce once;
    const int rc = set_max_smem_once(once, attention_tc_kernel, AQ_SMEM);
    if (rc) return rc;
    AqParams p{qkv, kcache, vcache, positions, out, tokens_per_seq, n_heads, n_kv, max_ctx, 0, scale};
    while (n_kv << (p.r_shift + 1) <= n_heads) ++p.r_shift;
    CUtensorMap kmap, vmap;
    const size_t rows = (size_t)(tokens / tokens_per_seq) * n_kv * max_ctx;
    int err = ts_map_2d(&kmap, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, CU_TENSOR_MAP_SWIZZLE_128B, kcache, rows, AQ_D, AQ_D * 2, AQ_KEYS, 64);
    if (!err) err = ts_map_2d(&vmap, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, CU_TENSOR_MAP_SWIZZLE_128B, vcache, rows, AQ_D, AQ_D * 2, AQ_KEYS, 64);
    if (err) return err;
    const int QT = AQ_ROWS >> p.r_shift, nblk = (tokens_per_seq + QT - 1) / QT;
    const unsigned blocks = (unsigned)((tokens / tokens_per_seq) * n_kv * nblk);
    SBVR_CUDA_TRY(launch_pdl(attention_tc_kernel, dim3(blocks), dim3(AQ_THREADS), (size_t)AQ_SMEM, st, kmap, vmap, p));
    return SBVR_OK;
}

}  // namespace sbvr
