// sbvr_decode_f16: packed bit-planes + coefficients -> dense fp16 weight, bit-exact with the
// reference decoder (`sbvr.decode`, reference sbvr/core.py:926-949): for every element the
// coefficients of its set planes are summed in fp32 in plane order (products with 0/1 are exact)
// and rounded to fp16 once (round-to-nearest-even).  No fast-math, no flush-to-zero: about 0.5 %
// of N(0, 0.01) coefficients are fp16 subnormals and must survive.
//
// HBM-bound: reads S/8 + idx bytes per element, writes 2 bytes per element.
// A block decodes 32 rows x 256 k.  A warp takes 32 consecutive rows at one word position, so its plane loads are one
// contiguous run of 32*S words, and a thread the 32 elements of one (row, word) pair.  The values go through shared memory
// and leave as whole 512-byte row segments: written straight from the decoding threads (16 bytes per lane, one row per lane)
// they made half-filled 32-byte sectors and the kernel took 87 us at 14336 x 4096, S = 4, 1.7 TB/s.
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

int launch_decode(const PackedW& w, __half* W, int ldw, int Kout, cudaStream_t st) {
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
