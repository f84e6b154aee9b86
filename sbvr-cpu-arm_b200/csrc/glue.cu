// The small kernels between the SBVR linears of a Llama decoder layer, each one launch where the reference runs
// a chain of eager PyTorch ops (reference models/sbvr_llama.py): RMSNorm with the residual add folded in
// (:118-123, :395-406), rotary embedding + KV-cache append (:169-224, :330-336), attention over the cache for
// decode and prefill (:243-278), SiLU(gate) * up (:238-240), embedding lookup, greedy argmax.
// Rounding follows the reference where it is visible in fp16: RMSNorm multiplies by the weight after the cast
// to fp16; the rotary products and their sum are separate fp16 operations; SiLU is rounded to fp16 before the
// multiplication.  Attention keeps scores and probabilities in fp32 (the reference rounds the scores and the
// probabilities to fp16), which is inside the 1e-2 tolerance of the layer outputs.
#include <cooperative_groups.h>

#include <algorithm>

#include "common.cuh"

namespace sbvr {

namespace cg = cooperative_groups;

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// ---------------------------------------------------------------------------------------------
// h_out = h_in (+ delta);  y = weight * fp16( h_out * rsqrt(mean(h_out^2) + eps) )        one CTA per row
// ---------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) add_rmsnorm_kernel(const __half* h_in, const __half* __restrict__ delta,
                                                          const __half* __restrict__ weight, __half* h_out,
                                                          __half* __restrict__ y, int hidden, float eps) {
    __shared__ float red[8];
    pdl_launch_dependents();
    pdl_wait();
    const size_t row = (size_t)blockIdx.x * hidden;
    const int nvec = hidden / 8;
    float ss = 0.0f;
    for (int i = threadIdx.x; i < nvec; i += blockDim.x) {
        uint4 a = *reinterpret_cast<const uint4*>(h_in + row + (size_t)i * 8);
        __half2* ah = reinterpret_cast<__half2*>(&a);
        if (delta) {
            const uint4 b = *reinterpret_cast<const uint4*>(delta + row + (size_t)i * 8);
            const __half2* bh = reinterpret_cast<const __half2*>(&b);
#pragma unroll
            for (int e = 0; e < 4; ++e) ah[e] = __hadd2(ah[e], bh[e]);
        }
        if (h_out) *reinterpret_cast<uint4*>(h_out + row + (size_t)i * 8) = a;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float2 f = __half22float2(ah[e]);
            ss += f.x * f.x + f.y * f.y;
        }
    }
    ss = warp_sum(ss);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
    __syncthreads();
    float tot = 0.0f;
#pragma unroll
    for (int w = 0; w < 8; ++w) tot += (w < (int)(blockDim.x >> 5)) ? red[w] : 0.0f;
    const float rs = rsqrtf(tot / (float)hidden + eps);
    const __half* src = h_out ? h_out : h_in;      // written above by this same thread when h_out is set
    for (int i = threadIdx.x; i < nvec; i += blockDim.x) {
        uint4 a = *reinterpret_cast<const uint4*>(src + row + (size_t)i * 8);
        if (!h_out && delta) {
            const uint4 b = *reinterpret_cast<const uint4*>(delta + row + (size_t)i * 8);
            __half2* ah2 = reinterpret_cast<__half2*>(&a);
            const __half2* bh = reinterpret_cast<const __half2*>(&b);
#pragma unroll
            for (int e = 0; e < 4; ++e) ah2[e] = __hadd2(ah2[e], bh[e]);
        }
        const uint4 wv = *reinterpret_cast<const uint4*>(weight + (size_t)i * 8);
        const __half2* ah = reinterpret_cast<const __half2*>(&a);
        const __half2* wh = reinterpret_cast<const __half2*>(&wv);
        uint4 o;
        __half2* oh = reinterpret_cast<__half2*>(&o);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float2 f = __half22float2(ah[e]);
            oh[e] = __hmul2(wh[e], __floats2half2_rn(f.x * rs, f.y * rs));
        }
        *reinterpret_cast<uint4*>(y + (size_t)blockIdx.x * hidden + (size_t)i * 8) = o;
    }
}

// ---------------------------------------------------------------------------------------------
// rotary embedding of q and k in place + append of k, v to the cache            one CTA per token
//   qkv row: [n_heads * d | n_kv * d | n_kv * d];  cache [seq, n_kv, max_ctx, d]
// ---------------------------------------------------------------------------------------------
constexpr int ROPE_HALF = 256;                     // head_dim / 2 at most

__global__ void __launch_bounds__(256) rope_append_kernel(__half* __restrict__ qkv, const int* __restrict__ positions,
                                                          const float* __restrict__ inv_freq, float attn_scaling,
                                                          __half* __restrict__ kcache, __half* __restrict__ vcache,
                                                          int tokens_per_seq, int n_heads, int n_kv, int d, int max_ctx) {
    __shared__ __half cs_s[2][ROPE_HALF];          // cos, sin of this token's position for i < head_dim / 2
    pdl_launch_dependents();
    pdl_wait();
    const int t = blockIdx.x;
    const int pos = positions[t];
    const int seq = t / tokens_per_seq;
    const int half_d = d / 2;
    __half* row = qkv + (size_t)t * (n_heads + 2 * n_kv) * d;
    for (int i = threadIdx.x; i < half_d; i += blockDim.x) {       // the accurate cosf / sinf are the expensive part
        const float ang = (float)pos * inv_freq[i];
        cs_s[0][i] = __float2half_rn(cosf(ang) * attn_scaling);
        cs_s[1][i] = __float2half_rn(sinf(ang) * attn_scaling);
    }
    __syncthreads();
    const int rot_items = (n_heads + n_kv) * half_d;
    for (int it = threadIdx.x; it < rot_items; it += blockDim.x) {
        const int head = it / half_d, i = it - head * half_d;
        const __half c = cs_s[0][i], s = cs_s[1][i];
        __half* hp = row + (size_t)head * d;
        const __half x1 = hp[i], x2 = hp[i + half_d];
        const __half o1 = __hadd(__hmul(x1, c), __hmul(__hneg(x2), s));
        const __half o2 = __hadd(__hmul(x2, c), __hmul(x1, s));
        hp[i] = o1, hp[i + half_d] = o2;
        if (head >= n_heads && pos < max_ctx) {
            __half* kc = kcache + (((size_t)seq * n_kv + (head - n_heads)) * max_ctx + pos) * d;
            kc[i] = o1, kc[i + half_d] = o2;
        }
    }
    if (pos < max_ctx) {
        const __half* vrow = row + (size_t)(n_heads + n_kv) * d;
        for (int it = threadIdx.x; it < n_kv * d; it += blockDim.x) {
            const int head = it / d, i = it - head * d;
            vcache[(((size_t)seq * n_kv + head) * max_ctx + pos) * d + i] = vrow[it];
        }
    }
}

// The same, eight elements at a time (16 bytes of either half of a head), for heads of a multiple of 16 in rows and caches on 16 bytes: the
// first two items of a thread are on their way while the angles are made.  An element at a time a call took 22.2 us at 3000 tokens of 32 + 8 heads of 128 (now 10.9; its
// bytes 9), 5.7 at 16 (now 2.3).
__global__ void __launch_bounds__(256) rope_append_vec_kernel(__half* __restrict__ qkv, const int* __restrict__ positions,
                                                              const float* __restrict__ inv_freq, float attn_scaling,
                                                              __half* __restrict__ kcache, __half* __restrict__ vcache,
                                                              int tokens_per_seq, int n_heads, int n_kv, int d, int max_ctx) {
    __shared__ __align__(16) __half cs_s[2][ROPE_HALF];
    pdl_launch_dependents();
    pdl_wait();
    const int t = blockIdx.x, half_d = d / 2, ch = half_d / 8;
    const int rot = (n_heads + n_kv) * ch, all = rot + n_kv * ch;  // a head's turn, or 16 values of v, per item
    __half* row = qkv + (size_t)t * (n_heads + 2 * n_kv) * d;
    auto load = [&](int it, uint4 (&x)[2]) {
        if (it >= all) return;
        const int head = it / ch;
        const __half* p = row + (size_t)head * d + (it - head * ch) * 8;
        x[0] = *reinterpret_cast<const uint4*>(p), x[1] = *reinterpret_cast<const uint4*>(p + half_d);
    };
    uint4 x[2][2];
    load(threadIdx.x, x[0]);
    load(threadIdx.x + 256, x[1]);
    const int pos = positions[t], seq = t / tokens_per_seq;
    for (int i = threadIdx.x; i < half_d; i += blockDim.x) {
        const float ang = (float)pos * inv_freq[i];
        cs_s[0][i] = __float2half_rn(cosf(ang) * attn_scaling);
        cs_s[1][i] = __float2half_rn(sinf(ang) * attn_scaling);
    }
    __syncthreads();
    auto finish = [&](int it, uint4 (&v)[2]) {
        if (it >= all) return;
        const int head = it / ch, i = (it - head * ch) * 8;
        if (it < rot) {
            const uint4 c = *reinterpret_cast<const uint4*>(&cs_s[0][i]), s = *reinterpret_cast<const uint4*>(&cs_s[1][i]);
            const __half2 *c2 = reinterpret_cast<const __half2*>(&c), *s2 = reinterpret_cast<const __half2*>(&s);
            __half2 *a = reinterpret_cast<__half2*>(&v[0]), *b = reinterpret_cast<__half2*>(&v[1]);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const __half2 x1 = a[e], x2 = b[e];
                a[e] = __hadd2(__hmul2(x1, c2[e]), __hmul2(__hneg2(x2), s2[e]));
                b[e] = __hadd2(__hmul2(x2, c2[e]), __hmul2(x1, s2[e]));
            }
            __half* p = row + (size_t)head * d + i;
            *reinterpret_cast<uint4*>(p) = v[0], *reinterpret_cast<uint4*>(p + half_d) = v[1];
        }
        if (head >= n_heads && pos < max_ctx) {
            const int kv = it < rot ? head - n_heads : head - n_heads - n_kv;
            __half* p = (it < rot ? kcache : vcache) + (((size_t)seq * n_kv + kv) * max_ctx + pos) * d + i;
            *reinterpret_cast<uint4*>(p) = v[0], *reinterpret_cast<uint4*>(p + half_d) = v[1];
        }
    };
    finish(threadIdx.x, x[0]);
    finish(threadIdx.x + 256, x[1]);
    for (int it = threadIdx.x + 512; it < all; it += 256) {
        load(it, x[0]);
        finish(it, x[0]);
    }
}

// ---------------------------------------------------------------------------------------------
// attention of one query token over cache positions [0, pos]; head_dim 128; grouped-query: the R = n_heads / n_kv
// query heads of a KV head are served together.  grid tokens * n_kv * nsplit, 128 threads; the nsplit CTAs of a (token, KV
// head) are a cluster that splits the positions and merges (max, sum, unnormalised sums) through distributed shared memory.
//
// Positions are taken AT_TILE at a time, K and V rows through cp.async, double buffered.  Scores: eight lanes per position,
// sixteen dims each (two 16-byte chunks 128 bytes apart: no bank conflicts).  Weights: a warp per head, running maximum.
// P.V: a thread owns two dims and half of a tile's positions.  It is a chain of latencies (position, rows, three barriers
// per tile, the merge); with a lane per position, a quarter of the positions per warp and a second kernel for the merge it took
// 10.8 + 3.2 us at 576 positions, 32 query heads, 8 KV heads, one token.
// ---------------------------------------------------------------------------------------------
constexpr int AT_D = 128;
constexpr int AT_TILE = 64;
constexpr int AT_MAX_CLUSTER = 16;
constexpr int AT_SMEM = 4 * AT_TILE * AT_D * 2;                // K and V tiles x 2

__device__ __forceinline__ void at_cp16(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}

// `inv_freq` != NULL (decode, one token per sequence): the rotary embedding is applied here -- q on its way into registers;
// the token's own k by the CTA whose positions include it, which also appends k and v to the cache and puts them into its tile
// itself.
template <int R>
__global__ void __launch_bounds__(128) attention_kernel(const __half* __restrict__ qkv, __half* kcache, __half* vcache,
                                                        const int* __restrict__ positions, __half* __restrict__ out,
                                                        int tokens_per_seq, int n_heads, int n_kv, int max_ctx, float scale,
                                                        int nsplit, const float* __restrict__ inv_freq, float attn_scaling) {
    constexpr int RH = R < 4 ? R : 4;              // heads whose queries a thread holds at a time
    extern __shared__ __align__(128) unsigned char at_smem[];
    __shared__ __align__(16) __half qs[R][AT_D];
    __shared__ __align__(16) __half knew[AT_D], vnew[AT_D];
    __shared__ __half cs_s[2][AT_D / 2];
    __shared__ __align__(16) float sc[AT_TILE][R];              // scores, then weights
    __shared__ float corr_s[R];
    __shared__ float wm[R], wl[R];                              // the CTA's maximum and sum
    __shared__ __align__(16) float wacc[2][R][AT_D];            // per half of the threads; [0]: their sum, read by the cluster
    pdl_launch_dependents();
    pdl_wait();
    const int unit = (int)blockIdx.x / nsplit, split = (int)blockIdx.x - unit * nsplit;
    const int t = unit / n_kv, kvh = unit - t * n_kv;
    const int seq = t / tokens_per_seq;
    const int pos = positions[t];
    const int ctx = min(pos + 1, max_ctx);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const __half* tok = qkv + (size_t)t * (n_heads + 2 * n_kv) * AT_D;
    const __half* qrow = tok + (size_t)kvh * R * AT_D;
    const int per = (ctx + nsplit - 1) / nsplit;
    const int p0 = min(ctx, split * per), p1 = min(ctx, p0 + per);
    __half* kb = kcache + ((size_t)seq * n_kv + kvh) * max_ctx * AT_D;
    __half* vb = vcache + ((size_t)seq * n_kv + kvh) * max_ctx * AT_D;
    const bool rope = inv_freq != nullptr;
    // position whose rows do not come from the cache (-1: none)
    const int own = (rope && pos < max_ctx && pos >= p0 && pos < p1) ? pos : -1;
    const uint32_t ks0 = smem_u32(at_smem), vs0 = ks0 + 2 * AT_TILE * AT_D * 2;
    auto load_tile = [&](int base, int buf) {
        const int n = min(AT_TILE, p1 - base);
        for (int c = tid; c < n * 16; c += 128) {
            const int row = c >> 4, ch = c & 15;
            if (base + row == own) continue;
            const size_t src = (size_t)(base + row) * AT_D + ch * 8;
            const uint32_t dst = (uint32_t)(buf * AT_TILE * AT_D * 2 + row * 256 + ch * 16);
            at_cp16(ks0 + dst, kb + src);
            at_cp16(vs0 + dst, vb + src);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    if (p0 < p1) load_tile(p0, 0);
    if (rope) {
        if (tid < AT_D / 2) {
            const float ang = (float)pos * inv_freq[tid];
            cs_s[0][tid] = __float2half_rn(cosf(ang) * attn_scaling);
            cs_s[1][tid] = __float2half_rn(sinf(ang) * attn_scaling);
        }
        __syncthreads();
        auto rot = [&](const __half* row, int dd) {            // products and sum are separate fp16 operations
            const int i2 = dd % (AT_D / 2);
            const __half c = cs_s[0][i2], sn = cs_s[1][i2];
            const __half y = (dd < AT_D / 2) ? __hneg(row[dd + AT_D / 2]) : row[dd - AT_D / 2];
            return __hadd(__hmul(row[dd], c), __hmul(y, sn));
        };
#pragma unroll
        for (int r = 0; r < R; ++r) qs[r][tid] = rot(qrow + r * AT_D, tid);
        if (own >= 0) {                            // this CTA holds the new token's position
            const __half kr = rot(tok + (size_t)(n_heads + kvh) * AT_D, tid);
            const __half vr = tok[(size_t)(n_heads + n_kv + kvh) * AT_D + tid];
            knew[tid] = kr, vnew[tid] = vr;
            kb[(size_t)pos * AT_D + tid] = kr;
            vb[(size_t)pos * AT_D + tid] = vr;
        }
    } else {
#pragma unroll
        for (int r = 0; r < R; ++r) qs[r][tid] = qrow[r * AT_D + tid];
    }
    if (tid < R) wm[tid] = -INFINITY, wl[tid] = 0.0f;

    const int sub = lane & 7;
    const int d2 = tid & 63, hf = tid >> 6;
    float acc[R][2];
#pragma unroll
    for (int r = 0; r < R; ++r) acc[r][0] = acc[r][1] = 0.0f;
    int buf = 0;
#pragma unroll 1
    for (int base = p0; base < p1; base += AT_TILE, buf ^= 1) {
        const int n = min(AT_TILE, p1 - base);
        if (base + AT_TILE < p1) {
            load_tile(base + AT_TILE, buf ^ 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        unsigned char* kt = at_smem + buf * AT_TILE * AT_D * 2;
        unsigned char* vt = kt + 2 * AT_TILE * AT_D * 2;
        if (own >= base && own < base + n) {
            reinterpret_cast<__half*>(kt + (own - base) * 256)[tid] = knew[tid];       // (written by this thread)
            reinterpret_cast<__half*>(vt + (own - base) * 256)[tid] = vnew[tid];
        }
        __syncthreads();                           // tile and queries are in place
#pragma unroll
        for (int r0 = 0; r0 < R; r0 += RH) {
            float q[RH][16];
#pragma unroll
            for (int r = 0; r < RH; ++r)
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    const uint4 v = *reinterpret_cast<const uint4*>(&qs[r0 + r][(sub + 8 * c) * 8]);
                    const __half2* h = reinterpret_cast<const __half2*>(&v);
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const float2 f = __half22float2(h[e]);
                        q[r][c * 8 + 2 * e] = f.x, q[r][c * 8 + 2 * e + 1] = f.y;
                    }
                }
            for (int pb = warp * 4; pb < n; pb += 16) {
                const int p = pb + (lane >> 3), pr = min(p, n - 1);           // (positions past the end are dropped)
                float s[RH];
#pragma unroll
                for (int r = 0; r < RH; ++r) s[r] = 0.0f;
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    const uint4 v = *reinterpret_cast<const uint4*>(kt + pr * 256 + (sub + 8 * c) * 16);
                    const __half2* h = reinterpret_cast<const __half2*>(&v);
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const float2 f = __half22float2(h[e]);
#pragma unroll
                        for (int r = 0; r < RH; ++r) s[r] += f.x * q[r][c * 8 + 2 * e] + f.y * q[r][c * 8 + 2 * e + 1];
                    }
                }
#pragma unroll
                for (int r = 0; r < RH; ++r) {
#pragma unroll
                    for (int o = 4; o; o >>= 1) s[r] += __shfl_xor_sync(0xffffffffu, s[r], o);
                    if (sub == r && p < n) sc[p][r0 + r] = s[r] * scale;
                }
            }
        }
        __syncthreads();                           // scores
        for (int r = warp; r < R; r += 4) {
            const float m0 = wm[r];
            float a = (lane < n) ? sc[lane][r] : -INFINITY, c = (lane + 32 < n) ? sc[lane + 32][r] : -INFINITY;
            float m = fmaxf(a, c);
#pragma unroll
            for (int o = 16; o; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
            m = fmaxf(m, m0);
            const float corr = (m0 == -INFINITY) ? 0.0f : __expf(m0 - m);
            a = (lane < n) ? __expf(a - m) : 0.0f, c = (lane + 32 < n) ? __expf(c - m) : 0.0f;
            sc[lane][r] = a, sc[lane + 32][r] = c;
            const float l = warp_sum(a + c);
            __syncwarp();
            if (lane == 0) wm[r] = m, wl[r] = wl[r] * corr + l, corr_s[r] = corr;
        }
        __syncthreads();                           // weights
#pragma unroll
        for (int r = 0; r < R; ++r) acc[r][0] *= corr_s[r], acc[r][1] *= corr_s[r];
        const int a1 = min(n, (hf + 1) * (AT_TILE / 2));
#pragma unroll 8
        for (int p = hf * (AT_TILE / 2); p < a1; ++p) {
            const float2 v = __half22float2(*reinterpret_cast<const __half2*>(vt + p * 256 + d2 * 4));
#pragma unroll
            for (int r = 0; r < R; ++r) acc[r][0] += sc[p][r] * v.x, acc[r][1] += sc[p][r] * v.y;
        }
        __syncthreads();                           // tile and weights may be overwritten
    }
#pragma unroll
    for (int r = 0; r < R; ++r) *reinterpret_cast<float2*>(&wacc[hf][r][d2 * 2]) = make_float2(acc[r][0], acc[r][1]);
    __syncthreads();
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const float v = wacc[0][r][tid] + wacc[1][r][tid];
        if (nsplit == 1) out[((size_t)t * n_heads + kvh * R + r) * AT_D + tid] = __float2half_rn(wl[r] > 0.0f ? v / wl[r] : 0.0f);
        else wacc[0][r][tid] = v;
    }
    if (nsplit == 1) return;
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    // every CTA of the cluster finishes its share of the (head, dim) pairs, the splits in order
    for (int i = split * 128 + tid; i < R * AT_D; i += nsplit * 128) {
        const int r = i / AT_D, dd = i % AT_D;
        float mv[AT_MAX_CLUSTER], gm = -INFINITY;
#pragma unroll
        for (int k = 0; k < AT_MAX_CLUSTER; ++k) {
            mv[k] = (k < nsplit) ? *cluster.map_shared_rank(&wm[r], k) : -INFINITY;
            gm = fmaxf(gm, mv[k]);
        }
        float gl = 0.0f, ga = 0.0f;
#pragma unroll
        for (int k = 0; k < AT_MAX_CLUSTER; ++k) {
            if (k >= nsplit) break;
            const float c = (mv[k] == -INFINITY) ? 0.0f : __expf(mv[k] - gm);
            gl += *cluster.map_shared_rank(&wl[r], k) * c;
            ga += *cluster.map_shared_rank(&wacc[0][r][dd], k) * c;
        }
        out[((size_t)t * n_heads + kvh * R + r) * AT_D + dd] = __float2half_rn(gl > 0.0f ? ga / gl : 0.0f);
    }
    cluster.sync();                                // nobody leaves while its shared memory is being read
}

// ---------------------------------------------------------------------------------------------
// Causal prefill of short prompts (attention_prefill.cu has the others) on the tensor cores: a CTA takes 64 (query token, query head) pairs that share one KV head (64 / R
// consecutive tokens of a sequence x its R query heads), each of its four warps 16 of them, and walks the keys 64 at a time
// with a running maximum and sum per pair.  grid sequences * n_kv * ceil(tokens / (64 / R)), longest contexts first.
//
//   scores   q . k: mma.sync m16n8k16 on the fp16 values themselves, fp32 accumulation, scaled in fp32
//   weights  exp2 in fp32; for the product with V each is split into two fp16 parts (p = hi + lo to 2^-22), two MMAs per
//            tile, so that the probabilities keep their fp32 precision
//
// K and V tiles come through cp.async, double buffered, rows of 256 bytes with their 16-byte chunks XOR-swizzled by the row
// (ldmatrix without bank conflicts).  What bounds it is the tensor pipe's legacy path and the exponentials.  The CUDA-core
// kernel this replaces read K and V once per 16 pairs and was bound by fp32 FMA issue: 1 790 us per layer at 2 x 1500
// tokens, 32 query heads, 8 KV heads.
// ---------------------------------------------------------------------------------------------
constexpr int AP_ROWS = 64, AP_KEYS = 64, AP_THREADS = 128;
constexpr int AP_TILE = AP_KEYS * AT_D * 2;                    // bytes of a K or V tile
constexpr int AP_SMEM = 4 * AP_TILE;

__device__ __forceinline__ void ap_cp16(uint32_t dst, const void* src, bool on) {
    const uint32_t bytes = on ? 16u : 0u;                      // 0: sixteen zero bytes
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void ap_ldm4(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr)
                 : "memory");
}
__device__ __forceinline__ void ap_ldm4t(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr)
                 : "memory");
}
__device__ __forceinline__ void ap_mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ float ap_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// fp16 pair of (lo, hi) and what the rounding left over, as a second pair
__device__ __forceinline__ uint32_t ap_split(float lo, float hi, uint32_t& rest) {
    const __half2 h = __floats2half2_rn(lo, hi);
    const float2 f = __half22float2(h);
    const __half2 r = __floats2half2_rn(lo - f.x, hi - f.y);
    rest = *reinterpret_cast<const uint32_t*>(&r);
    return *reinterpret_cast<const uint32_t*>(&h);
}

template <int R>
__global__ void __launch_bounds__(AP_THREADS, 2)
    attention_prefill_kernel(const __half* __restrict__ qkv, const __half* __restrict__ kcache, const __half* __restrict__ vcache,
                             const int* __restrict__ positions, __half* __restrict__ out, int tokens_per_seq, int n_heads, int n_kv,
                             int max_ctx, float scale) {
    constexpr int QT = AP_ROWS / R;                            // tokens of a CTA
    extern __shared__ __align__(128) unsigned char ap_smem[];
    __shared__ int ctx_s[QT];
    pdl_launch_dependents();
    pdl_wait();
    const int nblk = (tokens_per_seq + QT - 1) / QT;
    const int per = (int)gridDim.x / nblk;                     // sequences * n_kv
    const int rest = blockIdx.x % per, qblk = nblk - 1 - (int)blockIdx.x / per;
    const int kvh = rest % n_kv, seq = rest / n_kv;
    const int t0 = seq * tokens_per_seq + qblk * QT;
    const int nq = min(QT, tokens_per_seq - qblk * QT);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int gid = lane >> 2, tig = lane & 3;
    for (int j = threadIdx.x; j < QT; j += AP_THREADS) ctx_s[j] = (j < nq) ? min(positions[t0 + j] + 1, max_ctx) : 0;
    __syncthreads();
    int P = 0, pmin = 0x7fffffff;                              // keys any / every live token of the CTA attends to
    for (int j = 0; j < nq; ++j) P = max(P, ctx_s[j]), pmin = min(pmin, ctx_s[j]);
    const __half* kb = kcache + ((size_t)seq * n_kv + kvh) * max_ctx * AT_D;
    const __half* vb = vcache + ((size_t)seq * n_kv + kvh) * max_ctx * AT_D;
    const uint32_t ks0 = smem_u32(ap_smem), vs0 = ks0 + 2 * AP_TILE;

    auto load_tile = [&](int tile, int buf) {
#pragma unroll
        for (int i = 0; i < AP_KEYS * 16 / AP_THREADS; ++i) {
            const int c = i * AP_THREADS + (int)threadIdx.x;
            const int row = c >> 4, ch = c & 15;
            const int key = tile * AP_KEYS + row;
            const bool on = key < P;
            const size_t src = (size_t)(on ? key : 0) * AT_D + ch * 8;
            const uint32_t dst = (uint32_t)(buf * AP_TILE + row * 256 + ((ch ^ (row & 7)) << 4));
            ap_cp16(ks0 + dst, kb + src, on);
            ap_cp16(vs0 + dst, vb + src, on);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    const int ntile = (P + AP_KEYS - 1) / AP_KEYS;
    if (ntile > 0) load_tile(0, 0);

    // this thread's two rows of the warp's sixteen, and their queries as MMA fragments
    int ctx[2];
    uint32_t qf[8][4];
    const size_t tok_pitch = (size_t)(n_heads + 2 * n_kv) * AT_D;
    const bool even = (reinterpret_cast<uintptr_t>(qkv) & 3) == 0;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int row = warp * 16 + gid + 8 * h, j = row / R, r = row % R;
        ctx[h] = ctx_s[j];
        const __half* q = qkv + (size_t)(t0 + min(j, nq - 1)) * tok_pitch + (size_t)(kvh * R + r) * AT_D + tig * 2;
#pragma unroll
        for (int kk = 0; kk < 8; ++kk)
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const __half* e = q + kk * 16 + c * 8;
                uint32_t v;
                if (even) v = *reinterpret_cast<const uint32_t*>(e);
                else v = (uint32_t)__half_as_ushort(e[0]) | ((uint32_t)__half_as_ushort(e[1]) << 16);
                qf[kk][h + 2 * c] = scale > 0.0f ? v : scale < 0.0f ? v ^ 0x80008000u : scale == 0.0f ? 0u : v;
            }
    }
    float o[16][4], mx[2] = {-INFINITY, -INFINITY}, sum[2] = {0.0f, 0.0f};
#pragma unroll
    for (int i = 0; i < 16; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) o[i][e] = 0.0f;
    // Exponentials to base 2.  The running maximum and the mask are those of the unscaled scores, so the factor has to be positive:
    // a negative scale turns the queries' signs, a scale of zero makes every score zero.
    const float sl2 = (scale == 0.0f ? 1.0f : fabsf(scale)) * 1.4426950408889634f;
    const int lrow = lane & 7;
    const uint32_t k_row = (uint32_t)((lrow + ((lane >> 4) & 1) * 8) * 256);
    const uint32_t v_row = (uint32_t)((lrow + ((lane >> 3) & 1) * 8) * 256);
    const int k_ch = (lane >> 3) & 1, v_ch = lane >> 4;

#pragma unroll 1
    for (int t = 0; t < ntile; ++t) {
        const int buf = t & 1;
        if (t + 1 < ntile) {
            load_tile(t + 1, buf ^ 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();
        const uint32_t kt = ks0 + buf * AP_TILE, vt = vs0 + buf * AP_TILE;
        float s[8][4];
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) s[i][e] = 0.0f;
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {
#pragma unroll
            for (int np = 0; np < 4; ++np) {
                uint32_t b[4];
                ap_ldm4(kt + np * 16 * 256 + k_row + (uint32_t)(((kk * 2 + k_ch) ^ lrow) << 4), b);
                ap_mma(s[np * 2], qf[kk], b[0], b[1]);
                ap_mma(s[np * 2 + 1], qf[kk], b[2], b[3]);
            }
        }
        if ((t + 1) * AP_KEYS > pmin) {                        // some token's context ends inside or before this tile
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (t * AP_KEYS + i * 8 + tig * 2 + (e & 1) >= ctx[e >> 1]) s[i][e] = -INFINITY;
        }
        float base[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            float m = mx[h];
#pragma unroll
            for (int i = 0; i < 8; ++i) m = fmaxf(m, fmaxf(s[i][2 * h], s[i][2 * h + 1]));
            m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 1));
            m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 2));
            base[h] = (m == -INFINITY) ? 0.0f : m * sl2;       // a row without any key so far
            const float corr = (mx[h] == -INFINITY) ? 0.0f : ap_exp2(mx[h] * sl2 - base[h]);
            mx[h] = m;
            sum[h] *= corr;
#pragma unroll
            for (int i = 0; i < 16; ++i) o[i][2 * h] *= corr, o[i][2 * h + 1] *= corr;
        }
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                s[i][e] = ap_exp2(fmaf(s[i][e], sl2, -base[e >> 1]));
                sum[e >> 1] += s[i][e];
            }
#pragma unroll
        for (int kq = 0; kq < 4; ++kq) {                       // sixteen keys at a time
            uint32_t ph[4], pl[4];
            ph[0] = ap_split(s[2 * kq][0], s[2 * kq][1], pl[0]);
            ph[1] = ap_split(s[2 * kq][2], s[2 * kq][3], pl[1]);
            ph[2] = ap_split(s[2 * kq + 1][0], s[2 * kq + 1][1], pl[2]);
            ph[3] = ap_split(s[2 * kq + 1][2], s[2 * kq + 1][3], pl[3]);
#pragma unroll
            for (int nd = 0; nd < 8; ++nd) {
                uint32_t b[4];
                ap_ldm4t(vt + kq * 16 * 256 + v_row + (uint32_t)(((nd * 2 + v_ch) ^ lrow) << 4), b);
                ap_mma(o[nd * 2], ph, b[0], b[1]);
                ap_mma(o[nd * 2 + 1], ph, b[2], b[3]);
                ap_mma(o[nd * 2], pl, b[0], b[1]);
                ap_mma(o[nd * 2 + 1], pl, b[2], b[3]);
            }
        }
        __syncthreads();                                       // the buffer may be overwritten
    }
    const bool even_o = (reinterpret_cast<uintptr_t>(out) & 3) == 0;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        float l = sum[h];
        l += __shfl_xor_sync(0xffffffffu, l, 1);
        l += __shfl_xor_sync(0xffffffffu, l, 2);
        const float inv = l > 0.0f ? 1.0f / l : 0.0f;
        const int row = warp * 16 + gid + 8 * h, j = row / R, r = row % R;
        if (j >= nq) continue;
        __half* dst = out + ((size_t)(t0 + j) * n_heads + kvh * R + r) * AT_D + tig * 2;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const __half2 v = __floats2half2_rn(o[i][2 * h] * inv, o[i][2 * h + 1] * inv);
            if (even_o) *reinterpret_cast<__half2*>(dst + i * 8) = v;
            else dst[i * 8] = __low2half(v), dst[i * 8 + 1] = __high2half(v);
        }
    }
}

// ---------------------------------------------------------------------------------------------
// out[t, i] = fp16(silu(gate[t, i])) * up[t, i];   gu row = [gate (inter) | up (inter)]
// ---------------------------------------------------------------------------------------------
__global__ void silu_mul_kernel(const __half* __restrict__ gu, __half* __restrict__ out, int rows, int inter) {
    pdl_launch_dependents();
    pdl_wait();
    const size_t nvec = (size_t)rows * inter / 8;
    for (size_t v = (size_t)blockIdx.x * blockDim.x + threadIdx.x; v < nvec; v += (size_t)gridDim.x * blockDim.x) {
        const size_t e0 = v * 8;
        const size_t t = e0 / inter, i = e0 - t * inter;
        const uint4 g = *reinterpret_cast<const uint4*>(gu + t * 2 * inter + i);
        const uint4 u = *reinterpret_cast<const uint4*>(gu + t * 2 * inter + inter + i);
        const __half2* gh = reinterpret_cast<const __half2*>(&g);
        const __half2* uh = reinterpret_cast<const __half2*>(&u);
        uint4 o;
        __half2* oh = reinterpret_cast<__half2*>(&o);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float2 f = __half22float2(gh[e]);
            const __half2 a = __floats2half2_rn(f.x / (1.0f + expf(-f.x)), f.y / (1.0f + expf(-f.y)));
            oh[e] = __hmul2(a, uh[e]);
        }
        *reinterpret_cast<uint4*>(out + e0) = o;
    }
}

__global__ void embedding_kernel(const int* __restrict__ ids, const __half* __restrict__ table, __half* __restrict__ out,
                                 int hidden) {
    pdl_launch_dependents();
    pdl_wait();
    const size_t src = (size_t)ids[blockIdx.x] * hidden, dst = (size_t)blockIdx.x * hidden;
    for (int i = threadIdx.x; i < hidden / 8; i += blockDim.x)
        *reinterpret_cast<uint4*>(out + dst + (size_t)i * 8) = *reinterpret_cast<const uint4*>(table + src + (size_t)i * 8);
}

// rows of Kin halves -> rows of K (K % 8 == 0), zeros behind; one thread per 8 output elements, any Kin
template <int THREADS>
__global__ void __launch_bounds__(THREADS, 2048 / THREADS) pad_rows_kernel(const __half* __restrict__ in, __half* __restrict__ out, int M, int Kin, int K) {
    pdl_launch_dependents();
    pdl_wait();
    const int kv = K / 8;
    const size_t nvec = (size_t)M * kv;
    for (size_t v = (size_t)blockIdx.x * THREADS + threadIdx.x; v < nvec; v += (size_t)gridDim.x * THREADS) {
        const size_t m = v / kv;
        const int k0 = (int)(v - m * kv) * 8;
        __align__(16) __half o[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) o[e] = (k0 + e < Kin) ? in[m * Kin + k0 + e] : __float2half(0.0f);
        *reinterpret_cast<uint4*>(out + v * 8) = *reinterpret_cast<const uint4*>(o);
    }
}

// Few rows: blocks of 128 threads with 32 registers, which find room beside a CTA of the GEMM in front and leave room for one of the GEMM behind
// (70 x 18945 x 415, S = 3, 25.4 us with blocks of 256, 23.8 so; 300 x 16146 x 415 31.5, 29.7; 64 x 4096 x 4095 20.5, 20.3).  More: blocks of 256, which
// copy faster (2048 x 4096 x 4095 71.1 us, 73.4 with blocks of 128).
constexpr size_t PAD_FEW = 76 * 1024;              // pieces of 16 bytes: four blocks of 128 per SM
int launch_pad_rows(const __half* in, __half* out, int M, int Kin, int K, cudaStream_t st) {
    if (K % 8) return SBVR_ERR_SHAPE;
    const size_t nvec = (size_t)M * (K / 8);
    if (nvec <= PAD_FEW)
        SBVR_CUDA_TRY(launch_pdl(pad_rows_kernel<128>, dim3((unsigned)((nvec + 127) / 128)), dim3(128), 0, st, in, out, M, Kin, K));
    else
        SBVR_CUDA_TRY(launch_pdl(pad_rows_kernel<256>, dim3((unsigned)std::min<size_t>((nvec + 255) / 256, 2368)), dim3(256), 0, st, in, out, M, Kin, K));
    return SBVR_OK;
}

// index of the first maximum of each row (torch.argmax's tie rule); NaN wins like in torch.
// grid (rows, parts): part `blockIdx.y` scans its slice of the row and leaves (value, index) in `partial`
// (or, with one part, writes the result); argmax_final_kernel picks the winner of the parts.
__global__ void __launch_bounds__(1024) argmax_kernel(const __half* __restrict__ logits, int* __restrict__ out, int vocab,
                                                      float* __restrict__ pval, int* __restrict__ pidx) {
    __shared__ float bv[32];
    __shared__ int bi[32];
    pdl_launch_dependents();
    pdl_wait();
    const __half* row = logits + (size_t)blockIdx.x * vocab;
    const int parts = (int)gridDim.y;
    const int per = (vocab + parts - 1) / parts;
    const int i0 = (int)blockIdx.y * per, i1 = min(vocab, i0 + per);
    float best = -INFINITY;
    int idx = 0x7fffffff;
    for (int i = i0 + (int)threadIdx.x; i < i1; i += blockDim.x) {
        float v = __half2float(row[i]);
        if (v != v) v = INFINITY;
        if (v > best || (v == best && i < idx)) best = v, idx = i;
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, idx, o);
        if (ov > best || (ov == best && oi < idx)) best = ov, idx = oi;
    }
    if ((threadIdx.x & 31) == 0) bv[threadIdx.x >> 5] = best, bi[threadIdx.x >> 5] = idx;
    __syncthreads();
    if (threadIdx.x < 32) {
        best = (threadIdx.x < (blockDim.x >> 5)) ? bv[threadIdx.x] : -INFINITY;
        idx = (threadIdx.x < (blockDim.x >> 5)) ? bi[threadIdx.x] : 0x7fffffff;
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, best, o);
            const int oi = __shfl_xor_sync(0xffffffffu, idx, o);
            if (ov > best || (ov == best && oi < idx)) best = ov, idx = oi;
        }
        if (threadIdx.x == 0) {
            if (parts == 1) {
                out[blockIdx.x] = idx;
            } else {
                pval[(size_t)blockIdx.x * parts + blockIdx.y] = best;
                pidx[(size_t)blockIdx.x * parts + blockIdx.y] = idx;
            }
        }
    }
}

__global__ void __launch_bounds__(32) argmax_final_kernel(const float* __restrict__ pval, const int* __restrict__ pidx,
                                                          int* __restrict__ out, int parts) {
    pdl_launch_dependents();
    pdl_wait();
    float best = -INFINITY;
    int idx = 0x7fffffff;
    for (int i = threadIdx.x; i < parts; i += 32) {
        const float v = pval[(size_t)blockIdx.x * parts + i];
        const int j = pidx[(size_t)blockIdx.x * parts + i];
        if (v > best || (v == best && j < idx)) best = v, idx = j;
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, idx, o);
        if (ov > best || (ov == best && oi < idx)) best = ov, idx = oi;
    }
    if (threadIdx.x == 0) out[blockIdx.x] = idx;
}

// Tiles beyond the default shared memory, clusters beyond the portable eight CTAs; once per device.
template <typename Kernel>
static int at_setup(SmemOnce& once, Kernel kernel) {
    int dev = 0;
    SBVR_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return SBVR_ERR_BAD_ARG;
    std::lock_guard<std::mutex> lock(once.mu);
    if (!once.done[dev]) {
        SBVR_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, AT_SMEM));
        SBVR_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        once.done[dev] = true;
    }
    return SBVR_OK;
}

}  // namespace sbvr

using namespace sbvr;

extern "C" {

int sbvr_add_rmsnorm_f16(const void* h_in, const void* delta, const void* weight, void* h_out, void* y, int rows,
                         int hidden, float eps, sbvr_stream_t stream) {
    if (!h_in || !weight || !y || rows < 1 || hidden < 8) return SBVR_ERR_BAD_ARG;
    if (hidden % 8) return SBVR_ERR_SHAPE;
    if ((reinterpret_cast<uintptr_t>(h_in) | reinterpret_cast<uintptr_t>(delta) | reinterpret_cast<uintptr_t>(weight) |
         reinterpret_cast<uintptr_t>(h_out) | reinterpret_cast<uintptr_t>(y)) & 15)
        return SBVR_ERR_ALIGN;
    SBVR_CUDA_TRY(launch_pdl(add_rmsnorm_kernel, dim3(rows), dim3(256), 0, reinterpret_cast<cudaStream_t>(stream),
                             reinterpret_cast<const __half*>(h_in), reinterpret_cast<const __half*>(delta),
                             reinterpret_cast<const __half*>(weight), reinterpret_cast<__half*>(h_out),
                             reinterpret_cast<__half*>(y), hidden, eps));
    return SBVR_OK;
}

int sbvr_rope_append_f16(void* qkv, const int* positions, const float* inv_freq, float attn_scaling, void* kcache,
                         void* vcache, int tokens, int tokens_per_seq, int n_heads, int n_kv, int head_dim, int max_ctx,
                         sbvr_stream_t stream) {
    if (!qkv || !positions || !inv_freq || !kcache || !vcache) return SBVR_ERR_BAD_ARG;
    if (tokens < 1 || tokens_per_seq < 1 || tokens % tokens_per_seq || n_heads < 1 || n_kv < 1 || head_dim < 2 ||
        head_dim % 2 || max_ctx < 1)
        return SBVR_ERR_BAD_ARG;
    if (head_dim > 2 * ROPE_HALF) return SBVR_ERR_UNSUPPORTED;
    const bool vec = head_dim % 16 == 0 && !((reinterpret_cast<uintptr_t>(qkv) | reinterpret_cast<uintptr_t>(kcache) |
                                              reinterpret_cast<uintptr_t>(vcache)) & 15);
    SBVR_CUDA_TRY(launch_pdl(vec ? rope_append_vec_kernel : rope_append_kernel, dim3(tokens), dim3(256), 0, reinterpret_cast<cudaStream_t>(stream),
                             reinterpret_cast<__half*>(qkv), positions, inv_freq, attn_scaling,
                             reinterpret_cast<__half*>(kcache), reinterpret_cast<__half*>(vcache), tokens_per_seq, n_heads,
                             n_kv, head_dim, max_ctx));
    return SBVR_OK;
}

static int attention_launch(const void* qkv, void* kcache, void* vcache, const int* positions, void* out, float* scratch,
                            int tokens, int tokens_per_seq, int n_heads, int n_kv, int head_dim, int max_ctx, float scale,
                            int nsplit, const float* inv_freq, float attn_scaling, sbvr_stream_t stream) {
    if (!qkv || !kcache || !vcache || !positions || !out) return SBVR_ERR_BAD_ARG;
    if (tokens < 1 || tokens_per_seq < 1 || tokens % tokens_per_seq || n_kv < 1 || n_heads % n_kv || max_ctx < 1 ||
        nsplit < 1 || nsplit > 64)
        return SBVR_ERR_BAD_ARG;
    if (head_dim != AT_D) return SBVR_ERR_UNSUPPORTED;
    if (nsplit > 1 && !scratch) return SBVR_ERR_WORKSPACE;
    if ((reinterpret_cast<uintptr_t>(kcache) | reinterpret_cast<uintptr_t>(vcache)) & 15) return SBVR_ERR_ALIGN;
    const int R = n_heads / n_kv;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const __half* q = reinterpret_cast<const __half*>(qkv);
    __half* kc = reinterpret_cast<__half*>(kcache);
    __half* vc = reinterpret_cast<__half*>(vcache);
    __half* o = reinterpret_cast<__half*>(out);
    if (!inv_freq && nsplit == 1 && tokens_per_seq >= 8) {      // prefill: tokens of a sequence share K / V fetches
        if (R != 1 && R != 2 && R != 4 && R != 8) return SBVR_ERR_UNSUPPORTED;
        DeviceInfo di;
        int dev = 0;
        SBVR_CUDA_TRY(cudaGetDevice(&dev));
        const int rc = device_info(dev, &di);
        if (rc) return rc;
        if (attention_tc_supported(qkv, out, tokens, tokens_per_seq, n_kv, R, di.sm_count))
            return launch_attention_tc(q, kc, vc, positions, o, tokens, tokens_per_seq, n_heads, n_kv, max_ctx, scale, st);
        const int QT = AP_ROWS / R, nblk = (tokens_per_seq + QT - 1) / QT;
        const dim3 bgrid((unsigned)((tokens / tokens_per_seq) * n_kv * nblk));
#define SBVR_ATTP(RR)                                                                                                       \
    do {                                                                                                                    \
        static SmemOnce once;                                                                                               \
        const int rc = set_max_smem_once(once, attention_prefill_kernel<RR>, AP_SMEM);                                      \
        if (rc) return rc;                                                                                                  \
        SBVR_CUDA_TRY(launch_pdl(attention_prefill_kernel<RR>, bgrid, dim3(AP_THREADS), (size_t)AP_SMEM, st, q,             \
                                 static_cast<const __half*>(kc), static_cast<const __half*>(vc), positions, o, tokens_per_seq, \
                                 n_heads, n_kv, max_ctx, scale));                                                           \
    } while (0)
        switch (R) {
            case 1: SBVR_ATTP(1); break;
            case 2: SBVR_ATTP(2); break;
            case 4: SBVR_ATTP(4); break;
            default: SBVR_ATTP(8); break;
        }
#undef SBVR_ATTP
        return SBVR_OK;
    }
    int cs = 1;                                    // splits: a power of two of at most 16
    while (cs * 2 <= nsplit && cs * 2 <= AT_MAX_CLUSTER) cs *= 2;
    nsplit = cs;
#define SBVR_ATT(RR)                                                                                                        \
    do {                                                                                                                    \
        static SmemOnce once;                                                                                               \
        const int rc = at_setup(once, attention_kernel<RR>);                                                                \
        if (rc) return rc;                                                                                                  \
        SBVR_CUDA_TRY(launch_pdl_cluster(attention_kernel<RR>, dim3((unsigned)(tokens * n_kv * nsplit)), dim3(128), nsplit, \
                                         (size_t)AT_SMEM, st, q, kc, vc, positions, o, tokens_per_seq, n_heads, n_kv, max_ctx, \
                                         scale, nsplit, inv_freq, attn_scaling));                                           \
    } while (0)
    switch (R) {
        case 1: SBVR_ATT(1); break;
        case 2: SBVR_ATT(2); break;
        case 4: SBVR_ATT(4); break;
        case 8: SBVR_ATT(8); break;
        default: return SBVR_ERR_UNSUPPORTED;
    }
#undef SBVR_ATT
    return SBVR_OK;
}

int sbvr_attention_f16(const void* qkv, const void* kcache, const void* vcache, const int* positions, void* out,
                       float* scratch, int tokens, int tokens_per_seq, int n_heads, int n_kv, int head_dim, int max_ctx,
                       float scale, int nsplit, sbvr_stream_t stream) {
    return attention_launch(qkv, const_cast<void*>(kcache), const_cast<void*>(vcache), positions, out, scratch, tokens,
                            tokens_per_seq, n_heads, n_kv, head_dim, max_ctx, scale, nsplit, nullptr, 1.0f, stream);
}

int sbvr_rope_attention_f16(const void* qkv, const int* positions, const float* inv_freq, float attn_scaling, void* kcache,
                            void* vcache, void* out, float* scratch, int tokens, int n_heads, int n_kv, int head_dim,
                            int max_ctx, float scale, int nsplit, sbvr_stream_t stream) {
    if (!inv_freq) return SBVR_ERR_BAD_ARG;
    return attention_launch(qkv, kcache, vcache, positions, out, scratch, tokens, 1, n_heads, n_kv, head_dim, max_ctx, scale,
                            nsplit, inv_freq, attn_scaling, stream);
}

int sbvr_silu_mul_f16(const void* gate_up, void* out, int rows, int inter, sbvr_stream_t stream) {
    if (!gate_up || !out || rows < 1 || inter < 8) return SBVR_ERR_BAD_ARG;
    if (inter % 8) return SBVR_ERR_SHAPE;
    if ((reinterpret_cast<uintptr_t>(gate_up) | reinterpret_cast<uintptr_t>(out)) & 15) return SBVR_ERR_ALIGN;
    const size_t nvec = (size_t)rows * inter / 8;
    const int blocks = (int)((nvec + 255) / 256 < 4096 ? (nvec + 255) / 256 : 4096);
    SBVR_CUDA_TRY(launch_pdl(silu_mul_kernel, dim3(blocks), dim3(256), 0, reinterpret_cast<cudaStream_t>(stream),
                             reinterpret_cast<const __half*>(gate_up), reinterpret_cast<__half*>(out), rows, inter));
    return SBVR_OK;
}

int sbvr_embedding_f16(const int* ids, const void* table, void* out, int tokens, int hidden, sbvr_stream_t stream) {
    if (!ids || !table || !out || tokens < 1 || hidden < 8) return SBVR_ERR_BAD_ARG;
    if (hidden % 8) return SBVR_ERR_SHAPE;
    if ((reinterpret_cast<uintptr_t>(table) | reinterpret_cast<uintptr_t>(out)) & 15) return SBVR_ERR_ALIGN;
    SBVR_CUDA_TRY(launch_pdl(embedding_kernel, dim3(tokens), dim3(256), 0, reinterpret_cast<cudaStream_t>(stream), ids,
                             reinterpret_cast<const __half*>(table), reinterpret_cast<__half*>(out), hidden));
    return SBVR_OK;
}

int sbvr_argmax_f16(const void* logits, int* out, float* scratch, int rows, int vocab, sbvr_stream_t stream) {
    if (!logits || !out || rows < 1 || vocab < 1) return SBVR_ERR_BAD_ARG;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    // few rows of a large vocabulary: cut every row into up to 64 parts so that more than one SM scans it
    int parts = 1;
    if (scratch && vocab >= 16384) {
        parts = 128 / rows;
        if (parts > 64) parts = 64;
        if (parts < 1) parts = 1;
    }
    float* pval = scratch;
    int* pidx = reinterpret_cast<int*>(scratch) + (size_t)rows * parts;
    SBVR_CUDA_TRY(launch_pdl(argmax_kernel, dim3((unsigned)rows, (unsigned)parts), dim3(1024), 0, st,
                             reinterpret_cast<const __half*>(logits), out, vocab, pval, pidx));
    if (parts > 1)
        SBVR_CUDA_TRY(launch_pdl(argmax_final_kernel, dim3(rows), dim3(32), 0, st, static_cast<const float*>(pval),
                                 static_cast<const int*>(pidx), out, parts));
    return SBVR_OK;
}

}  // extern "C"
