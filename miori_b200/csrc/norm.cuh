// Row arithmetic shared by the stand-alone norm kernels and the GEMV epilogue that applies
// post_norm_add (shaders/ops.metal:605-631) to the rows it has just produced: the same 256 threads
// in the same order, so both give the same bits.
#pragma once
#include "common.cuh"

namespace miori_b200 {
namespace neighbors {

constexpr int NORM_THREADS = 256;

// Meeting point of the NORM_THREADS threads that work on a row.  BAR == 0: they are the whole CTA;
// otherwise the CTA's first NORM_THREADS threads, on named barrier BAR.
template <int BAR>
__device__ __forceinline__ void norm_sync() {
    if constexpr (BAR == 0) __syncthreads();
    else asm volatile("bar.sync %0, %1;" ::"n"(BAR), "n"(NORM_THREADS) : "memory");
}

// Element i of a row another CTA of this launch may have written (L2 is the point of coherence).
template <bool FRESH>
__device__ __forceinline__ float norm_load(const float* row, uint32_t i) {
    if constexpr (FRESH) return __ldcg(row + i);
    else return ld_fresh(row + i);
}

// Sum of squares of a row, in a fixed order: every thread adds its strided elements, warps reduce
// by shuffles, every thread then adds the eight warp sums.  Called by threads 0 .. NORM_THREADS-1.
template <int BAR, bool FRESH>
__device__ __forceinline__ float row_sum_squares(const float* row, uint32_t n, float* part) {
    float ss = 0.0f;
    for (uint32_t i = threadIdx.x; i < n; i += NORM_THREADS) {
        const float v = norm_load<FRESH>(row, i);
        ss = __fmaf_rn(v, v, ss);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xFFFFFFFFu, ss, o);
    if ((threadIdx.x & 31u) == 0) part[threadIdx.x >> 5] = ss;
    norm_sync<BAR>();
    float tot = 0.0f;
#pragma unroll
    for (int i = 0; i < NORM_THREADS / 32; ++i) tot += part[i];
    return tot;
}

// The same for a row held in registers as 16-byte pieces.
template <int BAR, int PIECES>
__device__ __forceinline__ float row_sum_of_pieces(const float4 (&v)[PIECES], float* part) {
    float ss = 0.0f;
#pragma unroll
    for (int j = 0; j < PIECES; ++j) {
        ss = __fmaf_rn(v[j].x, v[j].x, ss), ss = __fmaf_rn(v[j].y, v[j].y, ss);
        ss = __fmaf_rn(v[j].z, v[j].z, ss), ss = __fmaf_rn(v[j].w, v[j].w, ss);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xFFFFFFFFu, ss, o);
    if ((threadIdx.x & 31u) == 0) part[threadIdx.x >> 5] = ss;
    norm_sync<BAR>();
    float tot = 0.0f;
#pragma unroll
    for (int i = 0; i < NORM_THREADS / 32; ++i) tot += part[i];
    return tot;
}

// out = x + src * rsqrt(mean(src^2) + eps) * w for one row of n elements; out may be src.
template <int BAR, bool FRESH>
__device__ __forceinline__ void post_norm_add_row(const float* x, const float* src, const uint16_t* w, float* out,
                                                  uint32_t n, float eps, float* part) {
    const float inv = rsqrtf(row_sum_squares<BAR, FRESH>(src, n, part) / (float)n + eps);
    for (uint32_t i = threadIdx.x; i < n; i += NORM_THREADS)
        out[i] = ld_fresh(x + i) + norm_load<FRESH>(src, i) * inv * bf16_bits_to_float(w[i]);
}

// The same for rows that divide into 16-byte pieces, at most PIECES of them per thread: every load of the
// row is issued before the first use -- one trip to memory instead of two dependent ones -- and a thread
// owns pieces, four neighbouring elements, so that loads and stores are 16 bytes wide.
template <int BAR, bool FRESH, int PIECES>
__device__ __forceinline__ void post_norm_add_row_vec(const float* x, const float* src, const uint16_t* w, float* out,
                                                      uint32_t n, float eps, float* part) {
    float4 v[PIECES], r[PIECES];
    uint2 g[PIECES];
#pragma unroll
    for (int j = 0; j < PIECES; ++j) {
        const uint32_t i = threadIdx.x + (uint32_t)j * NORM_THREADS;
        v[j] = r[j] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        g[j] = make_uint2(0u, 0u);
        if (i < n / 4u) {
            if constexpr (FRESH) v[j] = __ldcg(reinterpret_cast<const float4*>(src) + i);
            else v[j] = ld_fresh(reinterpret_cast<const float4*>(src) + i);
            r[j] = ld_fresh(reinterpret_cast<const float4*>(x) + i);
            g[j] = reinterpret_cast<const uint2*>(w)[i];
        }
    }
    const float inv = rsqrtf(row_sum_of_pieces<BAR, PIECES>(v, part) / (float)n + eps);
#pragma unroll
    for (int j = 0; j < PIECES; ++j) {
        const uint32_t i = threadIdx.x + (uint32_t)j * NORM_THREADS;
        if (i < n / 4u)
            reinterpret_cast<float4*>(out)[i] =
                make_float4(r[j].x + v[j].x * inv * bf16lo(g[j].x), r[j].y + v[j].y * inv * bf16hi(g[j].x),
                            r[j].z + v[j].z * inv * bf16lo(g[j].y), r[j].w + v[j].w * inv * bf16hi(g[j].y));
    }
}

// y = bf16(x * rsqrt(mean(x^2) + eps) * w) for such a row.
// Waits for the preceding kernel itself: the norm weights are immutable and travel before that.
template <int PIECES>
__device__ __forceinline__ void rmsnorm_row_vec(const float* x, const uint16_t* w, uint16_t* y, uint32_t n, float eps,
                                                float* part) {
    float4 v[PIECES];
    uint2 g[PIECES];
#pragma unroll
    for (int j = 0; j < PIECES; ++j) {
        const uint32_t i = threadIdx.x + (uint32_t)j * NORM_THREADS;
        g[j] = make_uint2(0u, 0u);
        if (i < n / 4u) g[j] = __ldg(reinterpret_cast<const uint2*>(w) + i);
    }
    pdl_wait_prior();
#pragma unroll
    for (int j = 0; j < PIECES; ++j) {
        const uint32_t i = threadIdx.x + (uint32_t)j * NORM_THREADS;
        v[j] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (i < n / 4u) v[j] = ld_fresh(reinterpret_cast<const float4*>(x) + i);
    }
    const float inv = rsqrtf(row_sum_of_pieces<0, PIECES>(v, part) / (float)n + eps);
#pragma unroll
    for (int j = 0; j < PIECES; ++j) {
        const uint32_t i = threadIdx.x + (uint32_t)j * NORM_THREADS;
        if (i < n / 4u)
            reinterpret_cast<uint2*>(y)[i] =
                make_uint2(float_to_bf16_bits(v[j].x * inv * bf16lo(g[j].x)) | (float_to_bf16_bits(v[j].y * inv * bf16hi(g[j].x)) << 16),
                           float_to_bf16_bits(v[j].z * inv * bf16lo(g[j].y)) | (float_to_bf16_bits(v[j].w * inv * bf16hi(g[j].y)) << 16));
    }
}

constexpr int NORM_PIECES = 2;  // pieces per thread: rows of up to 2048 elements

// post_norm_add of one row by whichever form takes it: the stand-alone kernel and the GEMV's epilogue both
// come here, so that they give the same bits.
template <int BAR, bool FRESH>
__device__ __forceinline__ void post_norm_add_any(const float* x, const float* src, const uint16_t* w, float* out,
                                                  uint32_t n, float eps, float* part, bool vec) {
    if (vec) post_norm_add_row_vec<BAR, FRESH, NORM_PIECES>(x, src, w, out, n, eps, part);
    else post_norm_add_row<BAR, FRESH>(x, src, w, out, n, eps, part);
}
// Host: rows of n elements divide into pieces a CTA can hold (all pointers given).
inline bool norm_vec(uint32_t n, const void* a, const void* b, const void* c, const void* w) {
    return n % 4u == 0u && n <= 4u * NORM_THREADS * NORM_PIECES && aligned16(a) && aligned16(b) && aligned16(c) &&
           (reinterpret_cast<uintptr_t>(w) & 7u) == 0;
}

}  // namespace neighbors
}  // namespace miori_b200
