// int4 / int8 -> bf16 weight cache build.  out = bf16(float(code)*scale + bias) evaluated
// exactly as the reference does (src/cpu_ref.h:16-23,33,44): an fp32 multiply, an fp32 add
// (kept unfused so that overflow behaves identically) and the integer RNE to bf16.
//
// Bound by HBM: 0.5625-1.125 B read and 2 B written per weight.  Rows follow one another without gaps and
// hold whole scale groups, so the tensor is one array: unit i is eight weights, its scale is number
// 8 i / group, and no row or column is ever computed.
//
// Large tensors (dequant_wide_kernel): a grid that is resident at once, a thread per 32 weights, its next ones read before
// it works on these, 32-byte stores.  Chains of launches, the kernel of four units a thread and this, us: 4-bit
// 16384 x 2048 17.2 -> 15.4 (5.6 TB/s), over one buffer 14.3 -> 12.2, 2048 x 2048 3.5 -> 3.15, 1024 x 8192 5.4 -> 4.5; 8-bit
// 8192 x 2048 11.0 -> 8.8.  (16 weights a thread 15.7; two iterations ahead 16.9; blocks of four units without a loop
// are 3.5 waves, and each of their 4096 CTAs ends with a fence.)
#pragma once
#include "common.cuh"

#include <algorithm>

namespace miori_b200 {

// eight weights of one group -> eight bf16
template <int BITS>
__device__ __forceinline__ uint4 dequant_unit(const uint32_t (&w)[BITS / 4], uint32_t sbits, uint32_t bbits) {
    const float sc = bf16_bits_to_float(sbits), bi = bf16_bits_to_float(bbits);
    float f[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        // byte k of a register into the low byte of 2^23: 2^23 + code, exactly
        const uint32_t by = BITS == 8 ? w[BITS == 8 ? j >> 2 : 0] : (j & 1) ? (w[0] >> 4) & 0x0F0F0F0Fu : w[0] & 0x0F0F0F0Fu;
        const int k = BITS == 8 ? j & 3 : j >> 1;
        const float q = __uint_as_float(__byte_perm(by, 0x4B000000u, 0x7440 + k)) - 8388608.0f;
        f[j] = __fadd_rn(__fmul_rn(q, sc), bi);
    }
    uint32_t o[4];
    if ((sbits & 0x7F80u) != 0x7F80u && (bbits & 0x7F80u) != 0x7F80u) {
        // finite scale and bias: no NaN can arise, and the conversion instruction rounds by the same rule
#pragma unroll
        for (int p = 0; p < 4; ++p)
            asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(o[p]) : "f"(f[2 * p + 1]), "f"(f[2 * p]));
    } else {
#pragma unroll
        for (int p = 0; p < 4; ++p) o[p] = float_to_bf16_bits(f[2 * p]) | (float_to_bf16_bits(f[2 * p + 1]) << 16);
    }
    return make_uint4(o[0], o[1], o[2], o[3]);
}

constexpr int DEQUANT_THREADS = 256;

template <int BITS, int UNITS>
__global__ void __launch_bounds__(DEQUANT_THREADS)
dequant_rowmajor_kernel(const uint32_t* __restrict__ q, const uint16_t* __restrict__ s, const uint16_t* __restrict__ b,
                        uint4* __restrict__ out, uint64_t units, uint32_t ushift) {
    pdl_wait_prior();  // a programmatic launch, which costs the host less
    const uint64_t first = (uint64_t)blockIdx.x * (DEQUANT_THREADS * UNITS) + threadIdx.x;
    uint32_t w[UNITS][BITS / 4], sc[UNITS], bi[UNITS];
#pragma unroll
    for (int j = 0; j < UNITS; ++j) {
        const uint64_t i = first + (uint64_t)(j * DEQUANT_THREADS);
        if (i < units) {
            if constexpr (BITS == 4) {
                w[j][0] = ld_fresh<uint32_t, true>(q + i);
            } else {
                const uint2 v = ld_fresh<uint2, true>(reinterpret_cast<const uint2*>(q) + i);
                w[j][0] = v.x, w[j][1] = v.y;
            }
            sc[j] = ld_fresh(s + (i >> ushift));
            bi[j] = ld_fresh(b + (i >> ushift));
        }
    }
#pragma unroll
    for (int j = 0; j < UNITS; ++j) {
        const uint64_t i = first + (uint64_t)(j * DEQUANT_THREADS);
        if (i < units) out[i] = dequant_unit<BITS>(w[j], sc[j], bi[j]);
    }
    // No early trigger: dependents start when every CTA has exited, and a CTA exits with its weights written.
    // A product launched early fetches its first tiles of a cache ahead of its wait for the kernel before it, and
    // that may be the cache's build.  (Built and multiplied in turn in a graph, 2048 x 2048 gave wrong products with
    // the trigger at the top.  The fence costs 0.6 us: 16384 x 2048 16.6 -> 17.3; without it the writes of a CTA
    // that has exited may still be under way, though no product has come out wrong then.)
    __threadfence();
}

// The same by a resident grid, 32 weights -- four units of one scale group -- a thread and step.  out: 32-byte aligned.
constexpr uint32_t WIDE_UNITS = 4, WIDE_CTAS = 6;  // a step; CTAs of an SM
template <int BITS>
__global__ void __launch_bounds__(DEQUANT_THREADS)
dequant_wide_kernel(const uint4* __restrict__ q, const uint16_t* __restrict__ s, const uint16_t* __restrict__ b,
                    uint4* __restrict__ out, uint64_t steps, uint32_t sshift) {
    constexpr int WORDS = BITS, PER = BITS / 4;  // of a step, of a unit
    struct Step { uint32_t w[WORDS], sc, bi; };
    pdl_wait_prior();  // a programmatic launch, which costs the host less
    const uint64_t stride = (uint64_t)gridDim.x * DEQUANT_THREADS;
    auto load = [&](uint64_t i, Step& l) {
        if (i >= steps) return;
#pragma unroll
        for (int k = 0; k < WORDS / 4; ++k) {
            const uint4 v = ld_fresh<uint4, true>(q + i * (WORDS / 4) + k);
            l.w[4 * k] = v.x, l.w[4 * k + 1] = v.y, l.w[4 * k + 2] = v.z, l.w[4 * k + 3] = v.w;
        }
        l.sc = ld_fresh(s + (i >> sshift));
        l.bi = ld_fresh(b + (i >> sshift));
    };
    uint64_t i = (uint64_t)blockIdx.x * DEQUANT_THREADS + threadIdx.x;
    Step cur, next;
    load(i, cur);
    for (; i < steps; i += stride) {
        load(i + stride, next);
#pragma unroll
        for (int u = 0; u < (int)WIDE_UNITS; u += 2) {
            uint32_t w0[PER], w1[PER];
#pragma unroll
            for (int k = 0; k < PER; ++k) w0[k] = cur.w[u * PER + k], w1[k] = cur.w[(u + 1) * PER + k];
            const uint4 lo = dequant_unit<BITS>(w0, cur.sc, cur.bi), hi = dequant_unit<BITS>(w1, cur.sc, cur.bi);
            asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                         ::"l"(out + i * WIDE_UNITS + u), "r"(lo.x), "r"(lo.y), "r"(lo.z), "r"(lo.w), "r"(hi.x), "r"(hi.y), "r"(hi.z), "r"(hi.w)
                         : "memory");
        }
        cur = next;
    }
    __threadfence();  // no early trigger: as above
}

template <int BITS>
int launch_dequant_rowmajor(const void* q, const void* s, const void* b, void* out, uint32_t N,
                            uint32_t K, uint32_t group, cudaStream_t stream) {
    const uint64_t units = (uint64_t)N * (K >> 3);
    const uint32_t ushift = group == 32 ? 2u : 3u;  // log2 of the units per scale group
    // one unit per thread while four leave SMs without a block (256 x 2048: 1.94 us, 2.04 on the resident grid)
    const bool wide = units >= (uint64_t)sm_count() * DEQUANT_THREADS * 8u;
    const uint64_t per_block = (uint64_t)DEQUANT_THREADS * (wide ? 4u : 1u), blocks = (units + per_block - 1u) / per_block;
    if (blocks > 0x7FFFFFFFull) return fail(MIORI_E_INVALID, "dequant: N=%u K=%u is too large", N, K);
    if (wide && (reinterpret_cast<uintptr_t>(out) & 31u) == 0) {  // (a row is a multiple of 32 weights)
        const uint64_t steps = units / WIDE_UNITS, fill = (steps + DEQUANT_THREADS - 1u) / DEQUANT_THREADS;
        const cudaError_t e = launch(dequant_wide_kernel<BITS>, dim3((unsigned)std::min<uint64_t>((uint64_t)sm_count() * WIDE_CTAS, fill)),
                                     dim3(DEQUANT_THREADS), 0, stream, true, reinterpret_cast<const uint4*>(q),
                                     reinterpret_cast<const uint16_t*>(s), reinterpret_cast<const uint16_t*>(b),
                                     reinterpret_cast<uint4*>(out), steps, ushift - 2u);
        if (e != cudaSuccess) return cuda_fail(e, "dequant_wide launch");
        return MIORI_OK;
    }
    auto kern = wide ? dequant_rowmajor_kernel<BITS, 4> : dequant_rowmajor_kernel<BITS, 1>;
    cudaError_t e = launch(kern, dim3((unsigned)blocks), dim3(DEQUANT_THREADS), 0, stream, true,
                           reinterpret_cast<const uint32_t*>(q), reinterpret_cast<const uint16_t*>(s),
                           reinterpret_cast<const uint16_t*>(b), reinterpret_cast<uint4*>(out), units, ushift);
    if (e != cudaSuccess) return cuda_fail(e, "dequant_rowmajor launch");
    return MIORI_OK;
}

}  // namespace miori_b200
