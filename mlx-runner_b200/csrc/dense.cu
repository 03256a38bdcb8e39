// The dense matvec / small-batch kernel (dense.cuh).
#include "dense.cuh"

namespace mlxq {

namespace {

constexpr int DENSE_WARPS = 8;
constexpr int DENSE_TOKENS = 8;      // tokens per pass over a row

// eight consecutive elements as fp32; `vec`: the address is 16-byte aligned (32 for fp32) and may be read in one piece
__device__ __forceinline__ void load8_any(const void* p, int dt, size_t idx, bool vec, float (&o)[8]) {
    if (vec) {
        if (dt == DT_F32) {
            const float4 a = *reinterpret_cast<const float4*>(static_cast<const float*>(p) + idx);
            const float4 b = *reinterpret_cast<const float4*>(static_cast<const float*>(p) + idx + 4);
            o[0] = a.x; o[1] = a.y; o[2] = a.z; o[3] = a.w; o[4] = b.x; o[5] = b.y; o[6] = b.z; o[7] = b.w;
            return;
        }
        const uint4 v = *reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(p) + idx);
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int i = 0; i < 4; i++) {
            if (dt == DT_F16) {
                const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[i]));
                o[2 * i] = f.x; o[2 * i + 1] = f.y;
            } else {
                o[2 * i] = __uint_as_float(w[i] << 16);
                o[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
            }
        }
        return;
    }
#pragma unroll
    for (int i = 0; i < 8; i++) o[i] = load_scalar(p, dt, idx + i);
}

// A warp takes ROWS rows: their weights are streamed once, and every activation it loads serves all of them.  (With
// a row per warp the activations, read again for every row through L1, were the larger stream: 32000 x 4096 bf16 took
// 86 / 105 / 164 / 310 us with 1 / 2 / 4 / 8 fp32 tokens.)  NT: tokens of the call, compiled in so that the accumulators
// of absent tokens cost nothing.
template <int NT, int ROWS>
__global__ void __launch_bounds__(DENSE_WARPS * 32)
dense_mv_kernel(const void* __restrict__ w, int w_dtype, const void* __restrict__ bias, int bias_dtype, const void* __restrict__ x,
                int x_dtype, long long x_stride, void* __restrict__ y, int y_dtype, long long y_stride, int O, int K,
                int w_vec, int x_vec) {
    const int lane = threadIdx.x & 31;
    const int row0 = (blockIdx.x * DENSE_WARPS + (threadIdx.x >> 5)) * ROWS;
    if (row0 >= O) return;
    float acc[ROWS][NT];
    size_t wrow[ROWS];
#pragma unroll
    for (int r = 0; r < ROWS; r++) {
        wrow[r] = static_cast<size_t>(min(row0 + r, O - 1)) * K;      // (rows past the end read the last row; never stored)
#pragma unroll
        for (int t = 0; t < NT; t++) acc[r][t] = 0.0f;
    }
    const int K8 = K & ~7;
#pragma unroll 1
    for (int k = lane * 8; k < K8; k += 256) {
        float wv[ROWS][8];
#pragma unroll
        for (int r = 0; r < ROWS; r++) load8_any(w, w_dtype, wrow[r] + k, w_vec != 0, wv[r]);
#pragma unroll
        for (int t = 0; t < NT; t++) {
            float xv[8];
            load8_any(x, x_dtype, static_cast<size_t>(t) * x_stride + k, x_vec != 0, xv);
#pragma unroll
            for (int r = 0; r < ROWS; r++)
#pragma unroll
                for (int i = 0; i < 8; i++) acc[r][t] = fmaf(wv[r][i], xv[i], acc[r][t]);
        }
    }
    for (int k = K8 + lane; k < K; k += 32) {
#pragma unroll
        for (int r = 0; r < ROWS; r++) {
            const float wv = load_scalar(w, w_dtype, wrow[r] + k);
#pragma unroll
            for (int t = 0; t < NT; t++) acc[r][t] = fmaf(wv, load_scalar(x, x_dtype, static_cast<size_t>(t) * x_stride + k), acc[r][t]);
        }
    }
#pragma unroll
    for (int r = 0; r < ROWS; r++)
#pragma unroll
        for (int t = 0; t < NT; t++) {
            float v = acc[r][t];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            const int row = row0 + r;
            if (lane == 0 && row < O) {
                if (bias != nullptr) v += load_scalar(bias, bias_dtype, row);
                store_scalar(y, y_dtype, static_cast<size_t>(t) * y_stride + row, v);
            }
        }
}

template <int NT, int ROWS>
void launch_tokens(int nt, unsigned grid, cudaStream_t st, const void* w, int w_dtype, const void* bias, int bias_dtype, const void* x, int x_dtype,
                   long long x_stride, void* y, int y_dtype, long long y_stride, int O, int K, int w_vec, int x_vec) {
    if constexpr (NT > 1)
        if (nt < NT) return launch_tokens<NT - 1, ROWS>(nt, grid, st, w, w_dtype, bias, bias_dtype, x, x_dtype, x_stride, y, y_dtype, y_stride, O, K, w_vec, x_vec);
    dense_mv_kernel<NT, ROWS><<<grid, DENSE_WARPS * 32, 0, st>>>(w, w_dtype, bias, bias_dtype, x, x_dtype, x_stride, y, y_dtype, y_stride, O, K, w_vec, x_vec);
}

// Rows per warp.  Two save activation reads but leave half as many warps, which few rows or few tokens do not pay for.
// Times over those of a row per warp with the tokens not compiled in (bf16 weights, 512 ... 8192 columns, geometric mean):
//   fp32 tokens, 1 / 2 rows per warp:  2 tokens  4096 rows 0.90 / 1.03, 32000 0.83 / 0.85;  8 tokens  0.98 / 0.98, 0.94 / 0.75
//   bf16 tokens:                       2 tokens  4096 rows 0.86 / 1.09, 32000 0.72 / 0.88;  8 tokens  0.91 / 1.05, 0.86 / 0.83
// and from 6144 rows on two win from 3 fp32 or 4 bf16 tokens on (3 bf16 tokens 0.64 ... 0.84 / 0.72 ... 0.91).  Four rows per
// warp, and two turns of the loop in flight, cost registers and with them warps: 8 bf16 tokens with either 1.06 ... 1.35.
int rows_per_warp(int tokens, int O) { return tokens >= 3 && O >= 6144 ? 2 : 1; }

}  // namespace

cudaError_t launch_dense(const void* w, int w_dtype, const void* bias, int bias_dtype, const void* x, int x_dtype, long long x_stride,
                         void* y, int y_dtype, long long y_stride, long long T, int O, int K, cudaStream_t st) {
    const size_t wsz = dtype_size(w_dtype), xsz = dtype_size(x_dtype);
    const int w_vec = (reinterpret_cast<uintptr_t>(w) % 16 == 0 && (static_cast<size_t>(K) * wsz) % 16 == 0) ? 1 : 0;
    const int x_vec = (reinterpret_cast<uintptr_t>(x) % 16 == 0 && (static_cast<size_t>(x_stride) * xsz) % 16 == 0) ? 1 : 0;
    for (long long t0 = 0; t0 < T; t0 += DENSE_TOKENS) {
        const int tt = static_cast<int>(T - t0 < DENSE_TOKENS ? T - t0 : DENSE_TOKENS);
        const int rows = rows_per_warp(tt, O);
        const unsigned grid = static_cast<unsigned>((O + DENSE_WARPS * rows - 1) / (DENSE_WARPS * rows));
        const auto launch = rows == 2 ? launch_tokens<DENSE_TOKENS, 2> : launch_tokens<DENSE_TOKENS, 1>;
        launch(tt, grid, st, w, w_dtype, bias, bias_dtype, static_cast<const char*>(x) + static_cast<size_t>(t0) * x_stride * xsz, x_dtype, x_stride,
               static_cast<char*>(y) + static_cast<size_t>(t0) * y_stride * dtype_size(y_dtype), y_dtype, y_stride, O, K, w_vec, x_vec);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace mlxq
