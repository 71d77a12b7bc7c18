// The steps either side of a projection in the reference's decode graph (src/engine.cpp:389-413,
// 484-502): RMSNorm in front of it, SiLU x up or post-norm + residual behind it, and the 8-bit
// embedding gather that shares its table with the LM head.  Each is a small HBM- or latency-bound
// kernel; the RMSNorm also exists fused into the GEMV's activation staging (gemv_digits.cuh, gemv_tma.cuh).
//   rmsnorm        shaders/ops.metal:86-115   y = bf16(x * rsqrt(mean(x^2) + eps) * w)
//   silu_mul       shaders/ops.metal:129-139  out = bf16(g / (1 + exp(-g)) * up)
//   post_norm_add  shaders/ops.metal:605-631  out = x + src * rsqrt(mean(src^2) + eps) * w
//   embed8         shaders/ops.metal:170-197  out[t][k] = bf16(code * scale + bias) of row tokens[t]
#include "common.cuh"
#include "norm.cuh"
#include "peers.cuh"

namespace miori_b200 {
namespace neighbors {

// PIECES > 0: rows of at most 4 * NORM_THREADS * PIECES elements in 16-byte pieces, read once (norm.cuh).
// SPLIT: copies of the norm kernels for a few rows between the projections of a decode step (common.cuh: set_up_kernel).
template <int PIECES, Split SPLIT>
__global__ void __launch_bounds__(NORM_THREADS)
rmsnorm_kernel(const float* __restrict__ x, const uint16_t* __restrict__ w, uint16_t* __restrict__ y,
               uint32_t n, float eps) {
    __shared__ float part[NORM_THREADS / 32];
    pdl_launch_dependents();
    const float* row = x + (size_t)blockIdx.x * n;
    uint16_t* to = y + (size_t)blockIdx.x * n;
    if constexpr (PIECES > 0) {
        rmsnorm_row_vec<PIECES>(row, w, to, n, eps, part);
    } else {
        pdl_wait_prior();
        const float inv = rsqrtf(row_sum_squares<0, false>(row, n, part) / (float)n + eps);
        for (uint32_t i = threadIdx.x; i < n; i += NORM_THREADS)
            to[i] = (uint16_t)float_to_bf16_bits(ld_fresh(row + i) * inv * bf16_bits_to_float(w[i]));
    }
}

template <Split SPLIT>
__global__ void __launch_bounds__(NORM_THREADS)
post_norm_add_kernel(const float* __restrict__ x, const float* __restrict__ src,
                     const uint16_t* __restrict__ w, float* __restrict__ out, uint32_t n, float eps, bool vec) {
    __shared__ float part[NORM_THREADS / 32];
    pdl_launch_dependents();
    pdl_wait_prior();
    const size_t at = (size_t)blockIdx.x * n;
    post_norm_add_any<0, false>(x + at, src + at, w, out + at, n, eps, part, vec);
}

__device__ __forceinline__ uint32_t silu_mul_bits(float g, float u) {
    const float s = g / (1.0f + expf(-g));
    return float_to_bf16_bits(s * u);
}
// HBM-bound (8 B read, 2 B written per element): four elements per thread and 16-byte loads where the
// pointers allow it (1024 x 8192, from L2: 24.5 us one element at a time, 10.2 now).
template <bool VEC>
__global__ void __launch_bounds__(256)
silu_mul_kernel(const float* __restrict__ gate, const float* __restrict__ up, uint16_t* __restrict__ out,
                size_t n) {
    pdl_launch_dependents();
    pdl_wait_prior();
    const size_t first = (size_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (size_t)gridDim.x * blockDim.x;
    if constexpr (VEC) {
        for (size_t i = first; i < n / 4u; i += stride) {
            const float4 g = ld_fresh(reinterpret_cast<const float4*>(gate) + i), u = ld_fresh(reinterpret_cast<const float4*>(up) + i);
            reinterpret_cast<uint2*>(out)[i] =
                make_uint2(silu_mul_bits(g.x, u.x) | (silu_mul_bits(g.y, u.y) << 16), silu_mul_bits(g.z, u.z) | (silu_mul_bits(g.w, u.w) << 16));
        }
    } else {
        for (size_t i = first; i < n; i += stride) out[i] = (uint16_t)silu_mul_bits(ld_fresh(gate + i), ld_fresh(up + i));
    }
}

// One CTA per token: dequantize row tokens[t] of the 8-bit table.  A thread handles 16 codes (one
// 16-byte load), so a warp reads 512 contiguous bytes; fp32 multiply then add (unfused, like the
// cache build), integer round-to-nearest-even to bf16: bit-exact with src/cpu_ref.h:16-23,36-45.
__global__ void __launch_bounds__(128)
embed8_kernel(const uint4* __restrict__ q, const uint16_t* __restrict__ s, const uint16_t* __restrict__ b,
              const uint32_t* __restrict__ tokens, uint16_t* __restrict__ out, uint32_t K, uint32_t gshift,
              uint32_t rows) {
    pdl_launch_dependents();
    pdl_wait_prior();
    const uint32_t tok = ld_fresh(tokens + blockIdx.x);
    if (tok >= rows) return;  // an id outside the table leaves its output row untouched
    const uint32_t ng = K >> gshift;
    const uint4* qrow = q + (size_t)tok * (K / 16u);
    for (uint32_t c = threadIdx.x; c < K / 16u; c += blockDim.x) {
        const uint4 w = __ldg(qrow + c);
        const uint32_t g = (c * 16u) >> gshift;
        const float sc = bf16_bits_to_float(s[(size_t)tok * ng + g]);
        const float bi = bf16_bits_to_float(b[(size_t)tok * ng + g]);
        const uint32_t ww[4] = {w.x, w.y, w.z, w.w};
        uint32_t o[8];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
#pragma unroll
            for (int j = 0; j < 4; j += 2) {
                const float v0 = __fadd_rn(__fmul_rn((float)((ww[i] >> (8 * j)) & 0xFFu), sc), bi);
                const float v1 = __fadd_rn(__fmul_rn((float)((ww[i] >> (8 * j + 8)) & 0xFFu), sc), bi);
                o[i * 2 + j / 2] = float_to_bf16_bits(v0) | (float_to_bf16_bits(v1) << 16);
            }
        }
        uint4* dst = reinterpret_cast<uint4*>(out + (size_t)blockIdx.x * K + (size_t)c * 16u);
        dst[0] = make_uint4(o[0], o[1], o[2], o[3]);
        dst[1] = make_uint4(o[4], o[5], o[6], o[7]);
    }
}

// Largest element of a vector and its index (ties: the lowest index, as the host loop of
// src/engine.cpp:740-747 finds it).  A thread-block cluster of up to 8 CTAs shares the vector:
// 16-byte loads, a shuffle and shared-memory reduction per CTA, then every CTA hands its
// candidate to CTA 0 through distributed shared memory and CTA 0's first thread holds the result.
//
// A candidate is one 64-bit key, value above inverted index, in an order that integers compare: one compare
// per element and one shuffle pair per reduction step.  (What a call costs is latency: the first form had
// every thread walk the 32 warps' candidates one after the other.)
struct Best {
    float v;
    uint32_t i;
};
constexpr int ARGMAX_THREADS = 1024, ARGMAX_CLUSTER = 8;
__device__ __forceinline__ unsigned long long best_key(float v, uint32_t i) {
    return v == v ? peer_best_key(__float_as_uint(v == 0.0f ? 0.0f : v), i) : 0ull;  // the zeros are equal
}
__device__ __forceinline__ Best best_of_key(unsigned long long k) {
    const PeerBest b = peer_best_from_key(k);
    return Best{b.v, b.i};
}
__device__ __forceinline__ unsigned long long key_max(unsigned long long a, unsigned long long b) { return a > b ? a : b; }
__device__ __forceinline__ unsigned long long warp_key_max(unsigned long long k) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) k = key_max(k, __shfl_xor_sync(0xFFFFFFFFu, k, o));
    return k;
}
__device__ __forceinline__ uint32_t cluster_ctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t cluster_nctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t max_bf16x2(uint32_t a, uint32_t b) {  // of a number and a NaN the number
    uint32_t r;
    asm("max.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
template <bool BF16>
__device__ __forceinline__ float fresh_value(const void* v, uint32_t i) {
    if constexpr (BF16) return bf16_bits_to_float(ld_fresh(static_cast<const uint16_t*>(v) + i));
    else return ld_fresh(static_cast<const float*>(v) + i);
}
// This CTA's best over its slice of v[0, n), in thread 0.  Ties go to the lower index.
template <bool BF16>
__device__ __forceinline__ unsigned long long block_argmax(const void* __restrict__ v, uint32_t n, uint32_t index0,
                                                           unsigned long long* warp_best) {
    constexpr uint32_t PER = BF16 ? 8u : 4u;  // elements per 16-byte load
    const uint32_t nct = cluster_nctarank(), cr = cluster_ctarank();
    // slices of whole 16-byte pieces; the last CTA also takes the ragged tail
    const uint32_t pieces = n / PER, per_cta = (pieces + nct - 1u) / nct;
    const uint32_t p0 = min(cr * per_cta, pieces), p1 = min(p0 + per_cta, pieces);
    // A thread looks for its best piece by the pieces' maxima (three packed maxima for eight bf16) and for the element in
    // it at the end.  It sees its pieces and elements in ascending order, so that the first of equals stays.  (Element by
    // element, with a value and an index to select for each, a vector of 131072 took 2.86 us, now 2.64.)
    float bv = -INFINITY;
    uint32_t bi = 0xFFFFFFFFu, bp = 0xFFFFFFFFu;
    uint4 bw = make_uint4(0u, 0u, 0u, 0u);
    const bool vec_ok = (reinterpret_cast<uintptr_t>(v) & 15u) == 0;
    if (vec_ok) {
        const uint4* v4 = static_cast<const uint4*>(v);
#pragma unroll 2
        for (uint32_t p = p0 + threadIdx.x; p < p1; p += ARGMAX_THREADS) {
            const uint4 w = ld_fresh(v4 + p);
            float m;  // NaN only if all of them are
            if constexpr (BF16) {
                const uint32_t m2 = max_bf16x2(max_bf16x2(w.x, w.y), max_bf16x2(w.z, w.w));
                m = fmaxf(bf16lo(m2), bf16hi(m2));
            } else {
                m = fmaxf(fmaxf(__uint_as_float(w.x), __uint_as_float(w.y)), fmaxf(__uint_as_float(w.z), __uint_as_float(w.w)));
            }
            if (m > bv || (bp == 0xFFFFFFFFu && m == m)) bv = m, bp = p, bw = w;
        }
        if (bp != 0xFFFFFFFFu) {
            const uint32_t ww[4] = {bw.x, bw.y, bw.z, bw.w};
#pragma unroll
            for (int k = (int)PER - 1; k >= 0; --k) {
                const float f = !BF16 ? __uint_as_float(ww[k]) : k & 1 ? bf16hi(ww[k >> 1]) : bf16lo(ww[k >> 1]);
                if (f == bv) bi = index0 + bp * PER + (uint32_t)k;
            }
        }
    }
    auto see = [&](float f, uint32_t i) {
        if (f > bv || (f == bv && i < bi)) bv = f, bi = i;
    };
    // scalar part: everything when v is not 16-byte aligned (dealt to the CTAs), else the tail past the last
    // whole piece (last CTA)
    uint32_t s0 = n, step = ARGMAX_THREADS;
    if (!vec_ok) s0 = cr * ARGMAX_THREADS + threadIdx.x, step = nct * ARGMAX_THREADS;
    else if (cr == nct - 1u) s0 = pieces * PER + threadIdx.x;
    for (uint32_t i = s0; i < n; i += step)
        see(fresh_value<BF16>(v, i), index0 + i);
    const unsigned long long mine = warp_key_max(bi == 0xFFFFFFFFu ? 0ull : best_key(bv, bi));
    if ((threadIdx.x & 31u) == 0) warp_best[threadIdx.x >> 5] = mine;
    __syncthreads();
    return threadIdx.x < 32u ? warp_key_max(warp_best[threadIdx.x]) : 0ull;
}
// A candidate's value with the sign that its zero has in v (keys know one zero).
template <bool BF16>
__device__ __forceinline__ Best signed_zero(Best b, const void* __restrict__ v, uint32_t index0) {
    if (b.v == 0.0f) b.v = fresh_value<BF16>(v, b.i - index0);
    return b;
}
// Cluster-wide result, valid in thread 0 of CTA 0 of the cluster.  Every thread of every CTA of
// the cluster must call it (it contains cluster barriers).  cta_best: ARGMAX_CLUSTER entries of
// shared memory, at the same offset in every CTA.
template <bool BF16>
__device__ __forceinline__ Best cluster_argmax(const void* __restrict__ v, uint32_t n, uint32_t index0,
                                               unsigned long long* warp_best, unsigned long long* cta_best) {
    unsigned long long mine = block_argmax<BF16>(v, n, index0, warp_best);
    const uint32_t nct = cluster_nctarank(), cr = cluster_ctarank();
    if (nct == 1u) return signed_zero<BF16>(best_of_key(mine), v, index0);
    if (threadIdx.x == 0) {
        uint32_t remote;  // cta_best[cr] in CTA 0's shared memory
        asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(remote) : "r"(smem_addr(cta_best + cr)));
        asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(remote), "l"(mine) : "memory");
    }
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (cr == 0u && threadIdx.x == 0)
        for (uint32_t c = 1; c < nct; ++c) mine = key_max(mine, cta_best[c]);
    return cr == 0u ? signed_zero<BF16>(best_of_key(mine), v, index0) : best_of_key(mine);
}
template <bool BF16>
__global__ void __launch_bounds__(ARGMAX_THREADS)
argmax_kernel(const void* __restrict__ v, uint32_t n, uint32_t index0, uint32_t* __restrict__ out_index,
              float* __restrict__ out_value) {
    __shared__ unsigned long long warp_best[ARGMAX_THREADS / 32], cta_best[ARGMAX_CLUSTER];
    pdl_launch_dependents();
    pdl_wait_prior();
    const Best all = cluster_argmax<BF16>(v, n, index0, warp_best, cta_best);
    if (cluster_ctarank() == 0u && threadIdx.x == 0) {
        *out_index = all.i;
        if (out_value) *out_value = all.v;
    }
}
// CTAs for a vector of n elements: one per 8192 elements, at most a cluster of 8.
inline unsigned argmax_ctas(uint32_t n) {
    const unsigned c = (n + 8191u) / 8192u;
    return c >= 8u ? 8u : c >= 4u ? 4u : c >= 2u ? 2u : 1u;
}
// Launch with `ctas` CTAs forming one cluster.
template <class... KArgs, class... Args>
inline cudaError_t launch_cluster(void (*kernel)(KArgs...), unsigned ctas, unsigned threads, cudaStream_t stream,
                                  bool pdl, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ctas);
    cfg.blockDim = dim3(threads);
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    unsigned na = 0;
    attr[na].id = cudaLaunchAttributeClusterDimension;
    attr[na].val.clusterDim.x = ctas;
    attr[na].val.clusterDim.y = 1;
    attr[na].val.clusterDim.z = 1;
    ++na;
    if (pdl) {
        attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[na].val.programmaticStreamSerializationAllowed = 1;
        ++na;
    }
    cfg.attrs = attr;
    cfg.numAttrs = na;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

}  // namespace neighbors
}  // namespace miori_b200

using namespace miori_b200;

MIORI_API int miori_rmsnorm(const void* x, const void* gamma, void* y, uint32_t rows, uint32_t n, float eps,
                            uint32_t flags, void* stream) {
    if (!x || !gamma || !y) return fail(MIORI_E_INVALID, "miori_rmsnorm: null pointer");
    if (rows == 0 || n == 0) return fail(MIORI_E_INVALID, "miori_rmsnorm: empty shape rows=%u n=%u", rows, n);
    const bool vec = n % 4u == 0u && aligned16(x) && (reinterpret_cast<uintptr_t>(gamma) & 7u) == 0 && (reinterpret_cast<uintptr_t>(y) & 7u) == 0;
    auto run = [&](auto split) {
        constexpr Split S = decltype(split)::value;
        auto kern = !vec || n > 8192u ? neighbors::rmsnorm_kernel<0, S> : n <= 2048u ? neighbors::rmsnorm_kernel<2, S> : neighbors::rmsnorm_kernel<8, S>;
        return launch<S>(kern, dim3(rows), dim3(neighbors::NORM_THREADS), 0, (cudaStream_t)stream, (flags & MIORI_LAUNCH_PDL) != 0,
                         static_cast<const float*>(x), static_cast<const uint16_t*>(gamma), static_cast<uint16_t*>(y), n, eps);
    };
    const cudaError_t e = rows <= 4u ? run(std::integral_constant<Split, Split::SHARED>()) : run(std::integral_constant<Split, Split::DRIVERS>());
    if (e != cudaSuccess) return cuda_fail(e, "miori_rmsnorm launch");
    return MIORI_OK;
}

MIORI_API int miori_post_norm_add(const void* x, const void* src, const void* gamma, void* out, uint32_t rows,
                                  uint32_t n, float eps, uint32_t flags, void* stream) {
    if (!x || !src || !gamma || !out) return fail(MIORI_E_INVALID, "miori_post_norm_add: null pointer");
    if (rows == 0 || n == 0) return fail(MIORI_E_INVALID, "miori_post_norm_add: empty shape rows=%u n=%u", rows, n);
    auto run = [&](auto split) {
        constexpr Split S = decltype(split)::value;
        return launch<S>(neighbors::post_norm_add_kernel<S>, dim3(rows), dim3(neighbors::NORM_THREADS), 0, (cudaStream_t)stream,
                         (flags & MIORI_LAUNCH_PDL) != 0, static_cast<const float*>(x), static_cast<const float*>(src),
                         static_cast<const uint16_t*>(gamma), static_cast<float*>(out), n, eps, neighbors::norm_vec(n, x, src, out, gamma));
    };
    const cudaError_t e = rows <= 4u ? run(std::integral_constant<Split, Split::SHARED>()) : run(std::integral_constant<Split, Split::DRIVERS>());
    if (e != cudaSuccess) return cuda_fail(e, "miori_post_norm_add launch");
    return MIORI_OK;
}

MIORI_API int miori_silu_mul(const void* gate, const void* up, void* out, size_t n, uint32_t flags, void* stream) {
    if (!gate || !up || !out) return fail(MIORI_E_INVALID, "miori_silu_mul: null pointer");
    if (n == 0) return fail(MIORI_E_INVALID, "miori_silu_mul: empty vector");
    const bool vec = n % 4u == 0u && aligned16(gate) && aligned16(up) && (reinterpret_cast<uintptr_t>(out) & 7u) == 0;
    const unsigned blocks = (unsigned)std::min<size_t>((n / (vec ? 4u : 1u) + 255) / 256, (size_t)sm_count() * 16);
    const cudaError_t e = launch(vec ? neighbors::silu_mul_kernel<true> : neighbors::silu_mul_kernel<false>, dim3(blocks), dim3(256), 0, (cudaStream_t)stream,
                                 (flags & MIORI_LAUNCH_PDL) != 0, static_cast<const float*>(gate),
                                 static_cast<const float*>(up), static_cast<uint16_t*>(out), n);
    if (e != cudaSuccess) return cuda_fail(e, "miori_silu_mul launch");
    return MIORI_OK;
}

MIORI_API int miori_embed8(const void* q, const void* s, const void* b, const void* tokens, void* out,
                           uint32_t T, uint32_t rows, uint32_t K, uint32_t group, uint32_t flags, void* stream) {
    if (!q || !s || !b || !tokens || !out) return fail(MIORI_E_INVALID, "miori_embed8: null pointer");
    if (group != 32 && group != 64) return fail(MIORI_E_INVALID, "miori_embed8: group must be 32 or 64 (got %u)", group);
    if (T == 0 || rows == 0 || K == 0 || K % group != 0 || K % 16 != 0)
        return fail(MIORI_E_INVALID, "miori_embed8: bad shape T=%u rows=%u K=%u group=%u", T, rows, K, group);
    if (!aligned16(q) || !aligned16(out)) return fail(MIORI_E_INVALID, "miori_embed8: q and out must be 16-byte aligned");
    const cudaError_t e = launch(neighbors::embed8_kernel, dim3(T), dim3(128), 0, (cudaStream_t)stream,
                                 (flags & MIORI_LAUNCH_PDL) != 0, static_cast<const uint4*>(q),
                                 static_cast<const uint16_t*>(s), static_cast<const uint16_t*>(b),
                                 static_cast<const uint32_t*>(tokens), static_cast<uint16_t*>(out), K,
                                 group == 32 ? 5u : 6u, rows);
    if (e != cudaSuccess) return cuda_fail(e, "miori_embed8 launch");
    return MIORI_OK;
}

MIORI_API int miori_argmax(const void* v, uint32_t n, uint32_t flags, void* out_index, void* out_value,
                           void* stream) {
    if (!v || !out_index) return fail(MIORI_E_INVALID, "miori_argmax: null pointer");
    if (n == 0) return fail(MIORI_E_INVALID, "miori_argmax: empty vector");
    cudaError_t e;
    if (flags & MIORI_OUT_BF16)
        e = neighbors::launch_cluster(neighbors::argmax_kernel<true>, neighbors::argmax_ctas(n),
                                      neighbors::ARGMAX_THREADS, (cudaStream_t)stream,
                                      (flags & MIORI_LAUNCH_PDL) != 0, v, n, 0u, static_cast<uint32_t*>(out_index),
                                      static_cast<float*>(out_value));
    else
        e = neighbors::launch_cluster(neighbors::argmax_kernel<false>, neighbors::argmax_ctas(n),
                                      neighbors::ARGMAX_THREADS, (cudaStream_t)stream,
                                      (flags & MIORI_LAUNCH_PDL) != 0, v, n, 0u, static_cast<uint32_t*>(out_index),
                                      static_cast<float*>(out_value));
    if (e != cudaSuccess) return cuda_fail(e, "miori_argmax launch");
    return MIORI_OK;
}
