// Activation rows as the exact-class GEMM takes them (gemm_dq.cu): row m scaled by the power of two that brings it into (-1, 1),
// xh[m] = fp16 leading parts, xh[m_rows + m] = fp16 of what the first rounding dropped, columns in the order 0 2 1 3 within groups of
// four; xscale[m] = the inverse of the scale; xsum = sums of 32 columns, leading part and remainder:
// [k / 256][m][t]{hi of sub-blocks 2 t, 2 t + 1, lo of both}, the B fragment of the GEMM's minimum term.
//
// What produces the row is part of the kernel: a norm, SwiGLU or GELU. One block per row keeps it in registers from the first
// read to the store, so a norm reads and writes 8 bytes per value (it took two launches and 24: norm to f32, maximum, split),
// SwiGLU 12 (28). Norms, activations and splits of 16 layers of the 8B shape: 512 rows 1.89 ms in 114 launches before, 0.92 in
// 66 now; 32 rows 0.47 and 0.22.
#include <cuda_fp16.h>

#include <algorithm>

#include "kernels.h"
#include "pdl.cuh"
#include "sp_common.cuh"

namespace sp {

cudaError_t count_launch_and_check();  // kernels.cu

constexpr int DR_THREADS = 512;
// Threads of a row's block, at most: twice as many where they have two pieces of eight columns.
__host__ __device__ constexpr int dr_threads(int nc) { return nc == 2 ? 2 * DR_THREADS : DR_THREADS; }

struct DqRowsArgs {
    const float* x;
    int ldx, k, m_rows;
    const float* w;      // norms: weight and bias [k], either may be null
    const float* b;
    float eps;
    int up;              // SwiGLU: columns from gate to up
    __half* xh;
    float* xscale;
    __half* xsum;
};

__device__ __forceinline__ void dr_load8(const float* p, float (&v)[8]) {
    const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}

template <bool MAX>
__device__ __forceinline__ float dr_block(float v, float* sh) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float u = __shfl_xor_sync(0xFFFFFFFFu, v, o);
        v = MAX ? fmaxf(v, u) : v + u;
    }
    __syncthreads();
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    float t = sh[0];
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) t = MAX ? fmaxf(t, sh[w]) : t + sh[w];
    return t;
}

// Power of two that brings a row of this maximum into (-1, 1), and its inverse.
__device__ __forceinline__ float2 dr_scale(float amax) {
    if (!(amax > 0.f && amax < INFINITY)) return make_float2(1.f, 1.f);
    const int e = max(-100, min(100, (__float_as_int(amax) >> 23) - 126));  // amax < 2^e (subnormal maxima end at -100)
    return make_float2(__int_as_float((127 - e) << 23), __int_as_float((127 + e) << 23));
}

// Columns c .. c + 7 (v, in their order) of row m; every lane of the warp calls.
__device__ __forceinline__ void dr_split(const DqRowsArgs& a, int m, int c, bool live, const float (&v)[8], float up) {
    const int lane = threadIdx.x & 31;
    float x[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) x[i] = v[(i & 4) | ((i & 1) << 1) | ((i >> 1) & 1)] * up;
    uint32_t hi[4], lo[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const __half2 h = __floats2half2_rn(x[2 * j], x[2 * j + 1]);
        const __half2 l = __floats2half2_rn(x[2 * j] - __low2float(h), x[2 * j + 1] - __high2float(h));
        hi[j] = *reinterpret_cast<const uint32_t*>(&h);
        lo[j] = *reinterpret_cast<const uint32_t*>(&l);
    }
    float s = ((x[0] + x[1]) + (x[2] + x[3])) + ((x[4] + x[5]) + (x[6] + x[7]));
    s += __shfl_xor_sync(0xFFFFFFFFu, s, 1);
    s += __shfl_xor_sync(0xFFFFFFFFu, s, 2);
    if (!live) return;
    *reinterpret_cast<uint4*>(a.xh + (int64_t)m * a.k + c) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
    *reinterpret_cast<uint4*>(a.xh + ((int64_t)m + a.m_rows) * a.k + c) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
    if ((lane & 3) == 0 && (a.k & 255) == 0) {
        const int sub = (c >> 5) & 7;
        __half* d = a.xsum + ((int64_t)(c >> 8) * a.m_rows + m) * 16 + (sub >> 1) * 4 + (sub & 1);
        const __half h = __float2half_rn(s);
        d[0] = h;
        d[2] = __float2half_rn(s - __half2float(h));
    }
}

// One row per block, up to 8 NC columns per thread in registers. Formulas: kernels/layernorm.rs:17-105, elementwise.rs:120-143.
template <int SRC, int NC>
__global__ void __launch_bounds__(dr_threads(NC)) dq_rows_kernel(const DqRowsArgs a) {
    __shared__ float sh[dr_threads(NC) / 32];
    const int m = blockIdx.x;
    const float* row = a.x + (int64_t)m * a.ldx;
    // (a short row's norm weights, which no kernel writes, are here when the row comes)
    constexpr bool AHEAD = NC == 1 && (SRC == DQ_RMS || SRC == DQ_LN);
    float wa[8], ba[8];
    if (AHEAD && threadIdx.x * 8 < a.k) {
        if (a.w) dr_load8(a.w + threadIdx.x * 8, wa);
        if (SRC == DQ_LN && a.b) dr_load8(a.b + threadIdx.x * 8, ba);
    }
    pdl_wait();
    pdl_trigger();
    float v[NC][8];
    float amax = 0.f;
    auto each = [&](auto f) {
#pragma unroll
        for (int i = 0; i < NC; ++i) {
            const int c = (threadIdx.x + i * blockDim.x) * 8;
            if (c < a.k) f(v[i], c);
        }
    };
#pragma unroll
    for (int i = 0; i < 8 * NC; ++i) v[i >> 3][i & 7] = 0.f;
    each([&](float (&x)[8], int c) {
        dr_load8(row + c, x);
        if (SRC == DQ_SWIGLU) {
            float u[8];
            dr_load8(row + a.up + c, u);
#pragma unroll
            for (int i = 0; i < 8; ++i) x[i] = __fmul_rn(x[i] / (1.0f + expf(-x[i])), u[i]);
        } else if (SRC == DQ_GELU) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float t = x[i];
                const float inner = __fmul_rn(0.79788456f, __fadd_rn(t, __fmul_rn(__fmul_rn(__fmul_rn(0.044715f, t), t), t)));
                x[i] = __fmul_rn(__fmul_rn(0.5f, t), __fadd_rn(1.0f, tanhf(inner)));
            }
        }
    });
    if (SRC == DQ_RMS || SRC == DQ_LN) {
        float mean = 0.f, s = 0.f;
        if (SRC == DQ_LN) {
            each([&](float (&x)[8], int) { s += ((x[0] + x[1]) + (x[2] + x[3])) + ((x[4] + x[5]) + (x[6] + x[7])); });
            mean = dr_block<false>(s, sh) / (float)a.k;
            s = 0.f;
        }
        each([&](float (&x)[8], int) {
#pragma unroll
            for (int i = 0; i < 8; ++i) { const float d = x[i] - mean; s = fmaf(d, d, s); }
        });
        const float inv = 1.0f / sqrtf(dr_block<false>(s, sh) / (float)a.k + a.eps);
        each([&](float (&x)[8], int c) {
            float w[8], b[8];
            if (!AHEAD && a.w) dr_load8(a.w + c, w);
            if (!AHEAD && SRC == DQ_LN && a.b) dr_load8(a.b + c, b);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                if (AHEAD) { w[i] = wa[i]; b[i] = ba[i]; }
                x[i] = __fmul_rn(x[i] - mean, inv);
                if (a.w) x[i] = __fmul_rn(x[i], w[i]);
                if (SRC == DQ_LN && a.b) x[i] = __fadd_rn(x[i], b[i]);
            }
        });
    }
    each([&](float (&x)[8], int) {
#pragma unroll
        for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(x[i]));
    });
    const float2 sc = dr_scale(dr_block<true>(amax, sh));
    if (threadIdx.x == 0) a.xscale[m] = sc.y;
#pragma unroll
    for (int i = 0; i < NC; ++i) {
        const int c = (threadIdx.x + i * blockDim.x) * 8;
        dr_split(a, m, c, c < a.k, v[i], sc.x);
    }
}

// Rows as they are, of any length: read twice.
__global__ void __launch_bounds__(DR_THREADS) dq_long_rows_kernel(const DqRowsArgs a) {
    __shared__ float sh[DR_THREADS / 32];
    pdl_wait();
    pdl_trigger();
    const int m = blockIdx.x;
    const float* row = a.x + (int64_t)m * a.ldx;
    float amax = 0.f, v[8];
    for (int c = threadIdx.x * 8; c < a.k; c += blockDim.x * 8) {
        dr_load8(row + c, v);
#pragma unroll
        for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(v[i]));
    }
    const float2 sc = dr_scale(dr_block<true>(amax, sh));
    if (threadIdx.x == 0) a.xscale[m] = sc.y;
    for (int c0 = (threadIdx.x & ~31) * 8; c0 < a.k; c0 += blockDim.x * 8) {
        const int c = c0 + (threadIdx.x & 31) * 8;
        if (c < a.k) dr_load8(row + c, v);
        else
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = 0.f;
        dr_split(a, m, c, c < a.k, v, sc.x);
    }
}

bool dq_rows_fit(int k) { return k <= 4 * 8 * DR_THREADS; }

cudaError_t launch_dq_rows(int src, const float* x, int ldx, const float* w, const float* b, float eps, int m, int k, const DqInput& in, cudaStream_t st) {
    if (m <= 0) return cudaSuccess;
    if (k % 128 != 0 || !in.xscale || (src != DQ_PLAIN && !dq_rows_fit(k))) return cudaErrorInvalidValue;
    DqRowsArgs a{};
    a.x = x; a.ldx = ldx; a.k = k; a.m_rows = m; a.w = w; a.b = b; a.eps = eps; a.up = k;
    a.xh = in.xh; a.xscale = in.xscale; a.xsum = in.xsum;
    // Threads for eight columns each, or, above 4096 columns, for two or four such pieces. While rows are few a block has an SM nearly for
    // itself, and with more warps hides its loads better: SwiGLU of 32 rows of 14336, two pieces 5.4 us and four 8.4, of 192 rows of 8960 6.3
    // and 7.0, GELU of 389 rows of 10240 8.3 and 10.0; but 512 rows of 14336 23.5 and 18.3.
    const int pieces = k / 8, nc = pieces <= DR_THREADS ? 1 : pieces <= 2 * DR_THREADS || m <= 3 * device_sm_count() ? 2 : 4;
    const int threads = std::min(dr_threads(nc), ((pieces + nc - 1) / nc + 31) / 32 * 32);
    const dim3 grid((unsigned)m), block((unsigned)(dq_rows_fit(k) ? threads : DR_THREADS));
    cudaError_t le = cudaErrorInvalidValue;
#define SP_DR(S)                                                                                  \
    if (src == S) {                                                                               \
        if (nc == 1) le = launch_pdl(dq_rows_kernel<S, 1>, grid, block, 0, st, a);                \
        else if (nc == 2) le = launch_pdl(dq_rows_kernel<S, 2>, grid, block, 0, st, a);           \
        else le = launch_pdl(dq_rows_kernel<S, 4>, grid, block, 0, st, a);                        \
    }
    if (!dq_rows_fit(k)) le = launch_pdl(dq_long_rows_kernel, grid, block, 0, st, a);
    else { SP_DR(DQ_PLAIN) SP_DR(DQ_RMS) SP_DR(DQ_LN) SP_DR(DQ_SWIGLU) SP_DR(DQ_GELU) }
#undef SP_DR
    if (le != cudaSuccess) return le;
    return count_launch_and_check();
}

}  // namespace sp
