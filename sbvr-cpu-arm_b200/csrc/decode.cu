// sbvr_decode_f16: packed bit-planes + coefficients -> dense fp16 weight, bit-exact with the
// reference decoder (`sbvr.decode`, reference sbvr/core.py:926-949): for every element the
// coefficients of its set planes are summed in fp32 in plane order (products with 0/1 are exact)
// and rounded to fp16 once (round-to-nearest-even).  No fast-math, no flush-to-zero: about 0.5 %
// of N(0, 0.01) coefficients are fp16 subnormals and must survive.
//
// HBM-bound: reads S/8 + idx bytes per element, writes 2 bytes per element.  Two kernels:
//
// decode_table_kernel (two to four planes, rows that can be stored 16 bytes at a time).  A (row, group) has only 2^S different values:
// a thread forms them once for 64 k of a row, as two tables of bytes in registers, and looks them up four at a time with byte permutes: about
// 135 instructions per 32 values at S = 4 where a test and a predicated add per plane bit were 290, which in blocks that decode, wait and store
// added up with the bytes.  14336 x 4096: S = 4 35.5 -> 27.5 us (5.3 TB/s), S = 3 35.3 -> 26.2, S = 2 29.1 -> 24.0; 28672 x 8192, S = 4:
// 128 -> 104.  (One persistent block of 24 warps per SM, each with a run of units of its own, took 43.7: nothing is stored for the first
// microseconds, and the codebook has no room in L1.)
//
// decode_kernel (other shapes, pointers and plane counts).  A block decodes 32 rows x 256 k.  A warp takes 32 consecutive rows at one word
// position, so its plane loads are one contiguous run of 32*S words, and a thread the 32 elements of one (row, word) pair.  The values go
// through shared memory and leave as whole 512-byte row segments: written straight from the decoding threads (16 bytes per lane, one
// row per lane) they made half-filled 32-byte sectors and the kernel took 87 us at 14336 x 4096, S = 4, 1.7 TB/s.
#include "common.cuh"

namespace sbvr {

constexpr int DEC_ROWS = 32, DEC_K = 256;
constexpr int DEC_PITCH = DEC_K * 2 + 16;          // bytes; 33 16-byte units: lanes one row apart hit different banks

template <int S>
__global__ void __launch_bounds__(256) decode_kernel(const uint32_t* __restrict__ bvr, const void* __restrict__ idx,
                                                     int idx_bytes, const __half* __restrict__ coeff,
                                                     __half* __restrict__ W, int ldw, int N, int K, int Kout, int G) {
    __shared__ __align__(16) unsigned char tile[DEC_ROWS * DEC_PITCH];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int n0 = blockIdx.x * DEC_ROWS, k0 = blockIdx.y * DEC_K;
    const int n = n0 + lane, kw = k0 / 32 + warp;

    if (n < N && kw * 32 < K && kw * 32 < Kout) {
        uint32_t w[S];
        const uint32_t* src = bvr + ((size_t)kw * N + n) * S;
        if constexpr (S == 4) {
            if ((reinterpret_cast<uintptr_t>(bvr) & 15) == 0) {
                const uint4 v = __ldcs(reinterpret_cast<const uint4*>(src));
                w[0] = v.x, w[1] = v.y, w[2] = v.z, w[3] = v.w;
            } else {
#pragma unroll
                for (int s = 0; s < S; ++s) w[s] = __ldg(src + s);
            }
        } else {
#pragma unroll
            for (int s = 0; s < S; ++s) w[s] = __ldg(src + s);
        }
        const __half* line = coeff_line(idx, idx_bytes, coeff, (kw * 32) / G, n, N, S);
        float c[S];
#pragma unroll
        for (int s = 0; s < S; ++s) c[s] = __half2float(line[s]);   // exact, subnormals included
        uint4* dst = reinterpret_cast<uint4*>(tile + lane * DEC_PITCH + warp * 64);
#pragma unroll
        for (int j8 = 0; j8 < 4; ++j8) {
            __align__(16) __half2 out[4];
#pragma unroll
            for (int jj = 0; jj < 4; ++jj) {
                float v[2];
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const uint32_t bit = 1u << (j8 * 8 + jj * 2 + e);
                    float acc = 0.0f;
#pragma unroll
                    for (int s = 0; s < S; ++s)
                        if (w[s] & bit) acc = __fadd_rn(acc, c[s]);
                    v[e] = acc;
                }
                out[jj] = __floats2half2_rn(v[0], v[1]);
            }
            dst[j8] = *reinterpret_cast<const uint4*>(out);
        }
    }
    __syncthreads();
    // row segments: a warp writes one row's 256 values at a time
    const int kn = min(DEC_K, Kout - k0);
    const bool vec = (ldw % 8 == 0) && ((reinterpret_cast<uintptr_t>(W) & 15) == 0);
#pragma unroll
    for (int r = warp; r < DEC_ROWS; r += 8) {
        if (n0 + r >= N) break;
        __half* dst = W + (size_t)(n0 + r) * ldw + k0;
        const unsigned char* src = tile + r * DEC_PITCH;
        if (vec && lane * 8 + 8 <= kn) {
            __stcs(reinterpret_cast<uint4*>(dst) + lane, reinterpret_cast<const uint4*>(src)[lane]);
        } else if (!vec || lane * 8 < kn) {
            // rows that start off a 16-byte boundary, or the end of a row: one element per lane and step
            const int b = vec ? lane * 8 : lane, step = vec ? 1 : 32, e1 = vec ? min(kn, lane * 8 + 8) : kn;
            for (int e = b; e < e1; e += step) dst[e] = reinterpret_cast<const __half*>(src)[e];
        }
    }
}

// ---------------------------------------------------------------------------------------------
// values by table
// ---------------------------------------------------------------------------------------------
constexpr int DT_THREADS = 128;                    // a block decodes 32 rows x 256 k, a thread 64 k of a row

// The planes of 32 elements as one code of S bits per element, eight in a word: code of element 8 m + i in the low half of byte i of x[m],
// of element 8 m + 4 + i in its high half.
template <int S>
__device__ __forceinline__ void dt_codes(const uint32_t (&w)[S], uint32_t (&x)[4]) {
    constexpr uint32_t M1 = 0x55555555u, M2 = 0x33333333u, M4 = 0x44444444u;
    const uint32_t a = (w[0] & M1) | ((w[1] << 1) & ~M1), b = ((w[0] >> 1) & M1) | (w[1] & ~M1);         // elements 2 i, 2 i + 1: two bits each
    uint32_t e0 = a & M2, e1 = b & M2, e2 = (a >> 2) & M2, e3 = (b >> 2) & M2;                           // elements 4 i, .. 4 i + 3
    if constexpr (S == 3) e0 |= (w[2] << 2) & M4, e1 |= (w[2] << 1) & M4, e2 |= w[2] & M4, e3 |= (w[2] >> 1) & M4;
    if constexpr (S == 4) {
        const uint32_t c = (w[2] & M1) | ((w[3] << 1) & ~M1), d = ((w[2] >> 1) & M1) | (w[3] & ~M1);
        e0 |= (c << 2) & ~M2, e1 |= (d << 2) & ~M2, e2 |= c & ~M2, e3 |= d & ~M2;
    }
    const uint32_t t0 = __byte_perm(e0, e1, 0x5140), t1 = __byte_perm(e0, e1, 0x7362), u0 = __byte_perm(e2, e3, 0x5140),
                   u1 = __byte_perm(e2, e3, 0x7362);
    x[0] = __byte_perm(t0, u0, 0x5410), x[1] = __byte_perm(t0, u0, 0x7632);
    x[2] = __byte_perm(t1, u1, 0x5410), x[3] = __byte_perm(t1, u1, 0x7632);
}
// Four values, lower and upper bytes apart, by four codes (the lower half of `sel`); `hi`: 1 where a code has its fourth bit set.
template <int S>
__device__ __forceinline__ void dt_look_up(const uint32_t (&lo)[4], const uint32_t (&up)[4], uint32_t sel, uint32_t hi, uint32_t& l, uint32_t& u) {
    l = __byte_perm(lo[0], lo[1], sel), u = __byte_perm(up[0], up[1], sel);
    if constexpr (S == 4) {
        const uint32_t l2 = __byte_perm(lo[2], lo[3], sel), u2 = __byte_perm(up[2], up[3], sel), m = __byte_perm(0x0000ff00u, 0u, hi);
        l = (l & ~m) | (l2 & m), u = (u & ~m) | (u2 & m);
    }
}

template <int S>
__global__ void __launch_bounds__(DT_THREADS) decode_table_kernel(const uint32_t* __restrict__ bvr, const void* __restrict__ idx, int idx_bytes,
                                                                  const __half* __restrict__ coeff, int vec, __half* __restrict__ W, int ldw, int N,
                                                                  int KW, int Kout, int G) {
    __shared__ __align__(16) unsigned char tile[DEC_ROWS * DEC_PITCH];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int n0 = blockIdx.x * DEC_ROWS, k0 = blockIdx.y * DEC_K;
    const int n = min(n0 + lane, N - 1), kw = k0 / 32 + 2 * warp;          // rows past the last repeat it and are not stored
    pdl_launch_dependents();
    if (kw < KW) {
        uint32_t w[2][S];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const uint32_t* src = bvr + ((size_t)min(kw + j, KW - 1) * N + n) * S;
            if constexpr (S == 4) {
                const uint4 v = __ldcs(reinterpret_cast<const uint4*>(src));
                w[j][0] = v.x, w[j][1] = v.y, w[j][2] = v.z, w[j][3] = v.w;
            } else if constexpr (S == 2) {
                const uint2 v = __ldcs(reinterpret_cast<const uint2*>(src));
                w[j][0] = v.x, w[j][1] = v.y;
            } else {
#pragma unroll
                for (int s = 0; s < S; ++s) w[j][s] = __ldcs(src + s);
            }
        }
        // the 2^S values of this (row, group): sums in fp32 in plane order, rounded once
        const unsigned short* line = reinterpret_cast<const unsigned short*>(coeff_line(idx, idx_bytes, coeff, kw * 32 / G, n, N, S));
        unsigned short h[S];
        if (S == 4 && vec) {
            const uint2 v = __ldg(reinterpret_cast<const uint2*>(line));
            h[0] = v.x & 0xffff, h[1] = v.x >> 16, h[2] = v.y & 0xffff, h[S - 1] = v.y >> 16;
        } else if (S == 2 && vec) {
            const uint32_t v = __ldg(reinterpret_cast<const uint32_t*>(line));
            h[0] = v & 0xffff, h[1] = v >> 16;
        } else {
#pragma unroll
            for (int s = 0; s < S; ++s) h[s] = __ldg(line + s);
        }
        uint32_t lo[4], up[4];
        {
            float v[1 << S];
            v[0] = 0.0f;
#pragma unroll
            for (int s = 0; s < S; ++s) {
                const float c = __half2float(__ushort_as_half(h[s]));          // exact, subnormals included
#pragma unroll
                for (int j = 0; j < (1 << s); ++j) v[(1 << s) + j] = __fadd_rn(v[j], c);
            }
#pragma unroll
            for (int q = 0; q < (1 << S) / 4; ++q) {
                const __half2 a = __floats2half2_rn(v[4 * q], v[4 * q + 1]), b = __floats2half2_rn(v[4 * q + 2], v[4 * q + 3]);
                const uint32_t ab = *reinterpret_cast<const uint32_t*>(&a), bb = *reinterpret_cast<const uint32_t*>(&b);
                lo[q] = __byte_perm(ab, bb, 0x6420), up[q] = __byte_perm(ab, bb, 0x7531);
            }
            if constexpr (S == 2) lo[1] = up[1] = 0u;
        }
        uint4* mine = reinterpret_cast<uint4*>(tile + lane * DEC_PITCH + warp * 128);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            uint32_t x[4];
            dt_codes<S>(w[j], x);
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                const uint32_t sel = S == 4 ? x[m] & 0x77777777u : x[m], hi = S == 4 ? (x[m] >> 3) & 0x11111111u : 0u;
                uint32_t la, ua, lb, ub;           // elements 0, 4, 1, 5 and 2, 6, 3, 7 of the eight
                dt_look_up<S>(lo, up, sel, hi, la, ua);
                dt_look_up<S>(lo, up, sel >> 16, hi >> 16, lb, ub);
                mine[j * 4 + m] = make_uint4(__byte_perm(la, ua, 0x6240), __byte_perm(lb, ub, 0x6240), __byte_perm(la, ua, 0x7351),
                                             __byte_perm(lb, ub, 0x7351));
            }
        }
    }
    pdl_wait();                                    // W may still be in use by the kernel in front
    __syncthreads();
    // row segments: a warp writes one row's 256 values at a time, 16 bytes per lane
    const int kn = min(DEC_K, Kout - k0);
#pragma unroll
    for (int r = warp; r < DEC_ROWS; r += DT_THREADS / 32) {
        if (n0 + r >= N) break;
        __half* dst = W + (size_t)(n0 + r) * ldw + k0;
        const unsigned char* src = tile + r * DEC_PITCH;
        if (lane * 8 + 8 <= kn) {
            __stcs(reinterpret_cast<uint4*>(dst) + lane, reinterpret_cast<const uint4*>(src)[lane]);
        } else {
            for (int e = lane * 8; e < min(kn, lane * 8 + 8); ++e) dst[e] = reinterpret_cast<const __half*>(src)[e];
        }
    }
}

template <int S>
static int dt_launch(const PackedW& w, __half* W, int ldw, int Kout, cudaStream_t st) {
    const dim3 grid((w.N + DEC_ROWS - 1) / DEC_ROWS, (Kout + DEC_K - 1) / DEC_K);
    const int vec = !(reinterpret_cast<uintptr_t>(w.coeff) & (2 * S - 1)), KW = (Kout + 31) / 32;
    // Three quarters of the SM's memory for the blocks' rows (ten blocks): with all of it the codebook does not stay in L1 (30.2 -> 27.5 us)
    static SmemOnce once;
    const int rc = set_attribute_once(once, decode_table_kernel<S>, cudaFuncAttributePreferredSharedMemoryCarveout, 75);
    if (rc) return rc;
    SBVR_CUDA_TRY(launch_pdl(decode_table_kernel<S>, grid, dim3(DT_THREADS), 0, st, w.bvr, w.idx, w.idx_bytes, w.coeff, vec, W, ldw, w.N, KW, Kout,
                             w.G));
    return SBVR_OK;
}

int launch_decode(const PackedW& w, __half* W, int ldw, int Kout, cudaStream_t st) {
    // rows stored and words loaded in vectors, two neighbouring words in one group
    if (w.S >= 2 && w.S <= 4 && w.G % 64 == 0 && ldw % 8 == 0 && !(reinterpret_cast<uintptr_t>(W) & 15) &&
        (w.S == 3 || !(reinterpret_cast<uintptr_t>(w.bvr) & (4 * w.S - 1)))) {
        switch (w.S) {
            case 2: return dt_launch<2>(w, W, ldw, Kout, st);
            case 3: return dt_launch<3>(w, W, ldw, Kout, st);
            default: return dt_launch<4>(w, W, ldw, Kout, st);
        }
    }
    dim3 grid((w.N + DEC_ROWS - 1) / DEC_ROWS, (Kout + DEC_K - 1) / DEC_K);
    dim3 block(256);
#define SBVR_DECODE_CASE(SS)                                                                                        \
    case SS:                                                                                                         \
        decode_kernel<SS><<<grid, block, 0, st>>>(w.bvr, w.idx, w.idx_bytes, w.coeff, W, ldw, w.N, w.K, Kout,  \
                                                  w.G);        \
        break;
    switch (w.S) {
        SBVR_DECODE_CASE(1)
        SBVR_DECODE_CASE(2)
        SBVR_DECODE_CASE(3)
        SBVR_DECODE_CASE(4)
        SBVR_DECODE_CASE(5)
        SBVR_DECODE_CASE(6)
        SBVR_DECODE_CASE(7)
        SBVR_DECODE_CASE(8)
        default:
            return SBVR_ERR_UNSUPPORTED;
    }
#undef SBVR_DECODE_CASE
    SBVR_CUDA_TRY(cudaGetLastError());
    return SBVR_OK;
}

}  // namespace sbvr
