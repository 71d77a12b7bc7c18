// Weight-streaming GEMV for 1 <= M <= 32 activation rows on the packed 4- or 8-bit weights.  (One and two rows of 4-bit
// weights in groups of 64 come here only where gemv_digits.cuh does not take K: gemv.cuh.)
//
//   y[m][n] = sum_g ( s[n][g] * sum_{k in g} code[n][k] * x[m][k]  +  b[n][g] * sum_{k in g} x[m][k] )
//
// The inner sum runs on mma.sync.m16n8k16 with fp16 operands and fp32 accumulators:
//   * a code in the mantissa bits of a 16-bit half IS an fp16 value, the subnormal code * 2^-24 times its
//     place.  So a word of eight 4-bit codes becomes its four A registers with two shifts and four ANDs, the
//     codes in bits 2 .. 5 of a half or in bits 6 .. 9, where they count 16 times as much (their activations
//     are staged divided by 16); a word of four 8-bit codes becomes two registers with one shift and two
//     ANDs.  No offset is added to the codes, so none has to be subtracted from the sums.  (The place matters:
//     the tensor core aligns its products by the operands' exponents, and a subnormal's is that of 2^-14, so
//     what a code leaves empty above itself is cut off the sum.  With codes in bits 0 .. 7, one shift fewer,
//     the error against 64-bit sums was 1.9e-7, 5.6e-7, 5.2e-7 of the result at 1, 4, 8 rows of 2048 x 2048, now
//     0.7e-7, 1.3e-7, 1.2e-7, for 1 % of the time; every code in bits 6 .. 9: 0.7e-7, 1.0e-7, 1.1e-7, for 3-5 %.)
//   * a scale group's activations are multiplied by the power of two that puts the largest into
//     [2^15, 2^16): bf16's eight bits are exact in fp16 for every activation of at least 2^-28 of the
//     group's largest (the error below that is under 2^-36 of the largest).
// Every lane of the accumulator then applies the group's fp32 scale and bias: fp32 dequantization, the
// arithmetic class of the reference's gemv4 / gemv4_b / gemv8, for every M.  (The same product with
// e4m3 operands, whose subnormals hold a 4-bit code in a byte, halves the unpacking but takes as many MMAs, for
// bf16's eight bits need two e4m3 terms: 16384 x 2048 at 8 rows took 14.8 us against 12.4 at the time.)
//
// What bounds it: HBM for long 8-bit streams, the issue slots (some 136 warp instructions per KiB of codes at K = 2048)
// for long 4-bit ones, the hand-over between dependent launches and the trip of x through L2 for short
// ones.  Measured in chains of dependent launches over weights larger than L2, with codes as bf16 128 + code
// and one producer, and now, us: 8-bit head 131072 x 2048 at 1, 4, 16 rows 53.1, 60.3, 93 -> 42.7
// (6.7 TB/s, what a plain copy does), 44.2, 72.5; 4-bit 16384 x 2048 at 1, 4, 8 rows 7.44, 8.80, 10.2 ->
// 6.67, 7.28, 7.94; 2048 x 8192 at 1, 4 rows 6.58, 9.56 -> 4.63, 6.31.  2048 x 2048 at 1 row is no faster: 2.68
// and 2.70.
//
// One CTA per SM owns every gridDim-th 16-row tile.  A slab -- 16 rows x up to 1 KiB of codes -- is one
// 2-D TMA copy into a shared-memory ring; a tile's scales and biases (contiguous in memory) are two
// bulk copies into a ring of their own.  Completion is counted in bytes on mbarriers, buffers are
// handed back through "empty" mbarriers.  The rings are filled BEFORE the kernel waits for its
// predecessor (programmatic dependent launch): weights are immutable, so a CTA that starts as its
// predecessor's CTA exits has its first slabs in flight while the grids hand over.
//
// The 16 compute warps work in four independent groups of four; a group owns whole tiles, each of its
// warps multiplies a run of four neighbouring 64-byte steps of a slab, and the four partial sums per
// output are combined through shared memory behind a group-private named barrier by a fixed shuffle
// tree.  There is no CTA-wide barrier in the main loop.  Every group has a producer warp of its own,
// which only issues copies: with one producer for the CTA its hundred dependent instructions per slab and
// tile bounded long streams (151 MB of 4-bit weights: 46 us, 31 now), not the math.  Out-of-range rows
// and columns are zero-filled by TMA and staged as zeros.
//
// The eight MMA columns.  With more than four activation rows they are rows, and the quad's lanes read
// 4 or 8 bytes each so that a chain of MMAs covers one scale group.  With one, two or four rows the lanes
// read 16 bytes and the columns are (slot, row) with 8, 4 or 2 slots: a slot is one scale group of the
// run, its activations are zero in the lanes and steps that hold other groups, so one accumulator
// collects the sums of up to eight groups, each column its own, and scales are applied once per eight
// groups instead of once per group.  The sums of a row then meet in the same order for one to four rows:
// lane and register hold the groups of one residue modulo eight, added up in a fixed tree.
//
// Optional neighbours of the projection: the template value FUSED has the RMSNorm of fp32 activations inside
// the staging pass and SiLU x up behind the fused gate + up rows, POSTNORM the post-norm and residual add by
// the CTA that finishes last, SHARDED / ARGMAX the exchange with the peer GPUs and the greedy pick of a
// sharded head.  The plain instantiation is compiled as if they did not exist.  FUSED is one instantiation
// with run-time switches because a step's kernels evict one another from the instruction cache (code
// not there costs 70 ns per KiB): with three instantiations instead of two a 24-layer step took 588 us, now
// 574.  (With the switches in the plain kernel too: 561, but every projection by itself 0.17 us more.)
#pragma once
#include "common.cuh"
#include "norm.cuh"
#include "peers.cuh"
#include "tma_host.cuh"

#include <algorithm>
#include <type_traits>

namespace miori_b200 {
namespace gemvtma {

constexpr int GROUPS = 4;                        // independent groups of 4 warps
constexpr int WARPS = 4 * GROUPS;                // compute warps
constexpr int COMPUTE = WARPS * 32;
constexpr int THREADS = COMPUTE + GROUPS * 32;   // plus one producer warp per group
constexpr int MAX_NSG = 8;                       // code stages (and scale buffers) of one group
constexpr uint32_t SLAB_ROW = 1024;              // packed bytes of one row in a full slab
constexpr uint32_t STEP_BYTES = 64;              // packed bytes of one row in a step

constexpr int cmin(int a, int b) { return a < b ? a : b; }
constexpr int cmax(int a, int b) { return a > b ? a : b; }

// How a launch maps codes and activation rows to MMA operands.  ROWS: 1, 2, 4, 8, 16 or 32.
template <int BITS_, int GROUP_, int ROWS_>
struct Shape {
    static constexpr int BITS = BITS_, GROUP = GROUP_, ROWS = ROWS_;
    static constexpr int GPS = (int)STEP_BYTES * 8 / BITS / GROUP;  // scale groups per step: 1, 2 or 4
    static constexpr bool SLOTTED = ROWS < 8;
    static constexpr int NT = cmax(1, ROWS / 8);                    // sets of eight columns
    static constexpr int RC = cmin(ROWS, 8);                        // activation rows per set
    // slotted: columns are (slot, row); a pass covers SPA steps into SETS accumulators
    static constexpr int SLOTS = 8 / RC;
    static constexpr int SPA = cmin(4, cmax(1, SLOTS / GPS));
    static constexpr int SETS = cmax(1, GPS / SLOTS);
    static constexpr int NCLS = cmin(8, 4 * GPS);                   // residue classes of groups kept apart
    static constexpr int ACCN = SLOTTED ? cmax(1, NCLS / SLOTS) : NT;
    // bytes a lane reads of a row per chain, chains per step
    static constexpr int W = SLOTTED ? 16 : 16 / GPS;
    static constexpr int CH = 16 / W;
    static constexpr int NW = W / 4;
    static constexpr int XB = W * 8 / BITS * 2;                     // bytes of staged x per lane and chain
    static constexpr uint32_t KC = SLAB_ROW * 8 / BITS;             // codes per full slab
    static constexpr uint32_t SK = STEP_BYTES * 8 / BITS;           // codes per step
    // Row pitches in shared memory are these many bytes past a multiple of 128, so that the rows that a
    // quarter-warp (16-byte loads), half-warp (8) or warp (4) reads fall into different banks.
    static constexpr uint32_t QPAD = W == 16 ? 64 : W == 8 ? 32 : 16;
    static constexpr uint32_t XPAD = XB == 16 ? 64 : 16;
};

// zeros read by the lanes whose codes belong to another slot
constexpr uint32_t ZERO_BYTES = 64;

// Partial outputs of a group's four warps: [buffers][16 * ROWS outputs][4 warps] floats.  Two buffers, so
// that one barrier per tile is enough; one where two would cost stages of the code ring.
template <int ROWS>
struct Red {
    static constexpr int BUFS = ROWS <= 8 ? 2 : 1;
    static constexpr int FLOATS = 16 * ROWS * 4;
};

// Shared-memory loads by 32-bit shared address (one instruction each, no generic addressing).
// volatile: the data arrives through TMA, so the loads must stay behind the mbarrier wait.
__device__ __forceinline__ uint4 lds128(uint32_t a) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
    return v;
}
__device__ __forceinline__ uint2 lds64(uint32_t a) {
    uint2 v;
    asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a));
    return v;
}
__device__ __forceinline__ float4 ldsf128(uint32_t a) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
    return v;
}
__device__ __forceinline__ uint32_t lds32(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ uint32_t lds16(uint32_t a) {
    uint16_t v;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(a));
    return v;
}
template <int BYTES>
__device__ __forceinline__ void lds_words(uint32_t (&r)[BYTES / 4], uint32_t a) {
    static_assert(BYTES == 4 || BYTES == 8 || BYTES % 16 == 0, "");
    if constexpr (BYTES == 4) {
        r[0] = lds32(a);
    } else if constexpr (BYTES == 8) {
        const uint2 v = lds64(a);
        r[0] = v.x, r[1] = v.y;
    } else {
#pragma unroll
        for (int i = 0; i < BYTES / 16; ++i) {
            const uint4 v = lds128(a + 16u * i);
            r[4 * i] = v.x, r[4 * i + 1] = v.y, r[4 * i + 2] = v.z, r[4 * i + 3] = v.w;
        }
    }
}
__device__ __forceinline__ void named_barrier(uint32_t id, uint32_t threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// D += A B, 16 x 8 x 16, fp16 operands, fp32 accumulators.
__device__ __forceinline__ void mma_f16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                        uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ void mma_f16_z(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                          uint32_t b0, uint32_t b1) {  // D = A B
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%10,%10,%10,%10};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.0f));
}

// The A registers of one lane for one chain: codes of rows g and g + 8.
template <int BITS, int NW>
struct AFrag {
    static constexpr int AR = BITS == 4 ? 4 : 2;  // registers per word and row
    static constexpr int MMAS = NW * AR / 2;
    uint32_t r0[NW][AR], r1[NW][AR];
    __device__ __forceinline__ void unpack(const uint32_t (&q0)[NW], const uint32_t (&q1)[NW]) {
#pragma unroll
        for (int w = 0; w < NW; ++w) {
            if constexpr (BITS == 4) {
                const uint32_t l0 = q0[w] << 2, h0 = q0[w] >> 6, l1 = q1[w] << 2, h1 = q1[w] >> 6;
                r0[w][0] = l0 & 0x003C003Cu, r0[w][1] = l0 & 0x03C003C0u, r0[w][2] = h0 & 0x003C003Cu, r0[w][3] = h0 & 0x03C003C0u;
                r1[w][0] = l1 & 0x003C003Cu, r1[w][1] = l1 & 0x03C003C0u, r1[w][2] = h1 & 0x003C003Cu, r1[w][3] = h1 & 0x03C003C0u;
            } else {
                const uint32_t h0 = q0[w] >> 8, h1 = q1[w] >> 8;
                r0[w][0] = q0[w] & 0x00FF00FFu, r0[w][1] = h0 & 0x00FF00FFu;
                r1[w][0] = q1[w] & 0x00FF00FFu, r1[w][1] = h1 & 0x00FF00FFu;
            }
        }
    }
    // MMA i of the chain against its two B registers
    __device__ __forceinline__ void mma(bool first, int i, float (&d)[4], uint32_t b0, uint32_t b1) const {
        const int w = i / (AR / 2), p = i % (AR / 2) * 2;
        if (first) mma_f16_z(d, r0[w][p], r1[w][p], r0[w][p + 1], r1[w][p + 1], b0, b1);
        else mma_f16(d, r0[w][p], r1[w][p], r0[w][p + 1], r1[w][p + 1], b0, b1);
    }
};

// ---- staging of the activations ------------------------------------------------------------

// two floats -> packed fp16 pair (lo, hi), round to nearest even
__device__ __forceinline__ uint32_t f16x2_bits(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}

// Stage one unit -- eight consecutive activations of a row as bf16 -- for the MMA B operand: scaled fp16
// pairs in the order of the A registers and, by the first lane of each scale group, the group's {power
// of two that undoes the scaling, sum of x} / UNSCALE (so that the power of two stays finite for every
// input; the outputs are multiplied at the end).  The GROUP / 8 lanes of a group hold neighbouring
// units; every lane of the warp calls.  512 for codes that count from bit 0 of a half, 128 from bit 2.
template <int BITS>
constexpr float UNSCALE = BITS == 4 ? 128.0f : 512.0f;
template <int BITS, int GROUP>
__device__ __forceinline__ void stage_unit(const uint4& v, bool live, uint32_t x_addr, bool first, uint32_t ms_addr) {
    const uint32_t a = v.x & 0x7FFF7FFFu, b = v.y & 0x7FFF7FFFu, c = v.z & 0x7FFF7FFFu, d = v.w & 0x7FFF7FFFu;
    const uint32_t mx2 = __vmaxu2(__vmaxu2(a, b), __vmaxu2(c, d));
    uint32_t mx = max(mx2 & 0xFFFFu, mx2 >> 16);
    const float f[8] = {bf16lo(v.x), bf16hi(v.x), bf16lo(v.y), bf16hi(v.y), bf16lo(v.z), bf16hi(v.z), bf16lo(v.w), bf16hi(v.w)};
    float sum = ((f[0] + f[1]) + (f[2] + f[3])) + ((f[4] + f[5]) + (f[6] + f[7]));
#pragma unroll
    for (int o = 1; o < GROUP / 8; o <<= 1) {
        mx = max(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, o));
        sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
    }
    const uint32_t e = max(mx >> 7, 15u);  // exponent field of the largest; tiny groups stay below 2^15
    const float scale = __uint_as_float((269u - e) << 23);
    uint32_t o[4];
    if constexpr (BITS == 4) {
        const float low = 0.0625f * scale;  // for the codes that count 16 times
        o[0] = f16x2_bits(f[0] * scale, f[4] * scale), o[1] = f16x2_bits(f[1] * low, f[5] * low);
        o[2] = f16x2_bits(f[2] * scale, f[6] * scale), o[3] = f16x2_bits(f[3] * low, f[7] * low);
    } else {
        o[0] = f16x2_bits(f[0] * scale, f[2] * scale), o[1] = f16x2_bits(f[1] * scale, f[3] * scale);
        o[2] = f16x2_bits(f[4] * scale, f[6] * scale), o[3] = f16x2_bits(f[5] * scale, f[7] * scale);
    }
    if (live) {
        asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(x_addr), "r"(o[0]), "r"(o[1]), "r"(o[2]), "r"(o[3]) : "memory");
        if (first)
            asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(ms_addr), "f"(__uint_as_float(e << 23)), "f"(sum * (1.0f / UNSCALE<BITS>)) : "memory");
    }
}

// Where the staged activations of a CTA lie.
struct XArea {
    uint32_t x;      // shared address: [M][pitch] bytes
    uint32_t pitch;
    uint32_t ms;     // shared address: [K / GROUP][ROWS] float2
};
template <class S>
__device__ __forceinline__ void stage_unit_at(const XArea& xa, const uint4& v, bool live, uint32_t m, uint32_t u) {
    constexpr uint32_t UPG = S::GROUP / 8;
    stage_unit<S::BITS, S::GROUP>(v, live, xa.x + m * xa.pitch + 16u * u, (u & (UPG - 1u)) == 0u,
                                  xa.ms + ((u / UPG) * S::ROWS + m) * 8u);
}

// Stage M rows of K bf16 activations, several units per thread and trip with all loads issued first: every
// CTA of the grid asks L2 for the same lines at the same moment, and each dependent trip pays that queue
// again.  (Fewer for one row, which has at most two units per thread up to K = 8192: code that runs once
// per launch costs its instruction fetches, 0.1 us here.  Loading the next trip's units before working on
// this trip's, and copying all units first and working in place in a short loop, were both slower by 0.1
// to 1 us from two rows up.)  inv_upr = ceil(2^32 / (K / 8)).
template <class S>
__device__ __forceinline__ void stage_x(const XArea& xa, const uint16_t* __restrict__ x, uint32_t M, uint32_t K, uint32_t inv_upr) {
    const uint32_t upr = K >> 3, total = M * upr, lane = threadIdx.x & 31u;
    constexpr int AHEAD = S::ROWS == 1 ? 2 : 4;
    for (uint32_t i0 = threadIdx.x - lane; i0 < total; i0 += AHEAD * COMPUTE) {
        uint4 v[AHEAD];
        uint32_t m[AHEAD], u[AHEAD];
#pragma unroll
        for (int h = 0; h < AHEAD; ++h) {
            const uint32_t i = i0 + lane + (uint32_t)h * COMPUTE;
            m[h] = S::ROWS == 1 ? 0u : __umulhi(i, inv_upr);
            u[h] = i - m[h] * upr;
            v[h] = make_uint4(0u, 0u, 0u, 0u);
            if (i < total) v[h] = ld_fresh(reinterpret_cast<const uint4*>(x) + i);
        }
#pragma unroll
        for (int h = 0; h < AHEAD; ++h) {
            if (i0 + (uint32_t)h * COMPUTE >= total) break;  // warp-uniform
            stage_unit_at<S>(xa, v[h], i0 + lane + (uint32_t)h * COMPUTE < total, m[h], u[h]);
        }
    }
}

// The stand-alone norm kernel's arithmetic for two activations: x * inv * gamma, rounded to bf16.
__device__ __forceinline__ uint32_t normed2(float lo, float hi, float inv, uint32_t g2) {
    return float_to_bf16_bits(lo * inv * bf16lo(g2)) | (float_to_bf16_bits(hi * inv * bf16hi(g2)) << 16);
}
__device__ __forceinline__ uint4 normed8(const float4& a, const float4& c, float inv, const uint4& g) {
    return make_uint4(normed2(a.x, a.y, inv, g.x), normed2(a.z, a.w, inv, g.y), normed2(c.x, c.y, inv, g.z),
                      normed2(c.z, c.w, inv, g.w));
}

// Meeting point of the compute warps.
__device__ __forceinline__ void compute_sync() { named_barrier(15u, COMPUTE); }

// Staging with the RMSNorm in it (shaders/ops.metal:86-115): x is fp32.  Up to four rows of K <= 4096 take
// one trip to L2: thread u loads unit u of every row together with its norm weights, the warps add up
// the rows' squares (shuffles, 16 warp sums per row through shared memory, every thread adds them in
// order) and each thread normalises what it holds.  Anything larger sums the squares of four rows at a
// time first and normalises in the loader of the plain staging.  Called by the compute warps.
template <class S>
__device__ __forceinline__ void stage_x_normed(const XArea& xa, const float* __restrict__ x,
                                               const uint16_t* __restrict__ gamma, float eps, uint32_t M, uint32_t K,
                                               uint32_t inv_upr, float (&part)[4][WARPS], float (&inv_row)[32]) {
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, upr = K >> 3;
    const float4* x4 = reinterpret_cast<const float4*>(x);
    const uint4* g4 = reinterpret_cast<const uint4*>(gamma);
    constexpr uint32_t R = S::ROWS < 4 ? S::ROWS : 4;
    if (S::ROWS <= 4 && upr <= (uint32_t)COMPUTE) {
        const bool mine = tid < upr;
        float4 a[R], c[R];
        uint4 g = make_uint4(0u, 0u, 0u, 0u);
        if (mine) g = __ldg(g4 + tid);
#pragma unroll
        for (uint32_t m = 0; m < R; ++m) {
            a[m] = c[m] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (mine && m < M) {
                a[m] = ld_fresh(x4 + ((size_t)m * upr + tid) * 2u);
                c[m] = ld_fresh(x4 + ((size_t)m * upr + tid) * 2u + 1u);
            }
        }
#pragma unroll
        for (uint32_t m = 0; m < R; ++m) {
            if (m >= M) break;
            float ss = a[m].x * a[m].x;
            ss = __fmaf_rn(a[m].y, a[m].y, ss), ss = __fmaf_rn(a[m].z, a[m].z, ss), ss = __fmaf_rn(a[m].w, a[m].w, ss);
            ss = __fmaf_rn(c[m].x, c[m].x, ss), ss = __fmaf_rn(c[m].y, c[m].y, ss), ss = __fmaf_rn(c[m].z, c[m].z, ss);
            ss = __fmaf_rn(c[m].w, c[m].w, ss);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xFFFFFFFFu, ss, o);
            if (lane == 0) part[m][warp] = ss;
        }
        compute_sync();
        if (warp * 32u >= upr) return;
#pragma unroll
        for (uint32_t m = 0; m < R; ++m) {
            if (m >= M) break;
            float tot = 0.0f;
#pragma unroll
            for (int w = 0; w < WARPS; ++w) tot += part[m][w];
            const float inv = rsqrtf(tot / (float)K + eps);
            stage_unit_at<S>(xa, normed8(a[m], c[m], inv, g), mine, m, tid);
        }
        return;
    }
    const uint32_t qpr = K >> 2;
    for (uint32_t m0 = 0; m0 < M; m0 += 4u) {
        float ss[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        for (uint32_t i = tid; i < qpr; i += COMPUTE) {
#pragma unroll
            for (uint32_t r = 0; r < 4u; ++r) {
                if (m0 + r < M) {
                    const float4 v = ld_fresh(x4 + (size_t)(m0 + r) * qpr + i);
                    ss[r] = __fmaf_rn(v.w, v.w, __fmaf_rn(v.z, v.z, __fmaf_rn(v.y, v.y, __fmaf_rn(v.x, v.x, ss[r]))));
                }
            }
        }
#pragma unroll
        for (uint32_t r = 0; r < 4u; ++r) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) ss[r] += __shfl_xor_sync(0xFFFFFFFFu, ss[r], o);
            if (lane == 0) part[r][warp] = ss[r];
        }
        compute_sync();
        if (tid < 4u && m0 + tid < M) {
            float tot = 0.0f;
            for (int w = 0; w < WARPS; ++w) tot += part[tid][w];
            inv_row[m0 + tid] = rsqrtf(tot / (float)K + eps);
        }
        compute_sync();
    }
#pragma unroll 2
    for (uint32_t i0 = tid - lane; i0 < M * upr; i0 += COMPUTE) {  // whole warps
        const uint32_t i = i0 + lane, m = S::ROWS == 1 ? 0u : __umulhi(i, inv_upr), u = i - m * upr;
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (i < M * upr) v = normed8(ld_fresh(x4 + 2 * (size_t)i), ld_fresh(x4 + 2 * (size_t)i + 1), inv_row[m], __ldg(g4 + u));
        stage_unit_at<S>(xa, v, i < M * upr, m, u);
    }
}

// What the post-norm epilogue needs besides the GEMV's own arguments (null residual: off).
struct PostNorm {
    const float* residual = nullptr;   // x of post_norm_add, fp32 [M][N]
    const uint16_t* gamma = nullptr;   // bf16 [N]
    unsigned int* arrivals = nullptr;  // one zeroed word; the kernel leaves it zero
    float eps = 0.0f;
    bool vec = false;                  // neighbors::norm_vec
};

// What the norm prologue needs (null gamma: off): x then points at fp32 activations.
struct PreNorm {
    const uint16_t* gamma = nullptr;  // bf16 [K]
    float eps = 0.0f;
};

// What is fused around the product.
//   SHARDED: rows [row0, row0 + N) of an n_total-row output, exchanged with the peer GPUs
//   ARGMAX:  the head of a greedy decode step (one activation row).  The rows go to this rank's y only --
//            no packets -- and every thread tracks the best (value, index) of what it stores; the
//            candidates meet in a 64-bit atomic maximum, and the CTA that finishes last exchanges this
//            rank's best with the peers (peers.cuh: peer_argmax_exchange), so the kernel ends with the
//            winning token on every rank and nothing else has crossed NVLink
//   FUSED, gated: the weight rows are a gate half [0, N/2) and an up half [N/2, N) (the fused w1/w3
//            projection); a tile is eight rows of each, so that after the tile's reduction one thread
//            pair holds gate and up of the same output, and y is bf16 [M][N/2] of silu(gate) * up
//   POSTNORM: y = residual + v * rsqrt(mean(v^2) + eps) * gamma over each whole output row v of the GEMV
//            (shaders/ops.metal:605-631).  Every CTA stores its part of v into y; the CTA that arrives
//            last then runs the stand-alone kernel's row pass over y in place
//   FUSED, normed: x is fp32; bf16(x * rsqrt(mean(x^2) + eps) * gamma) is what is multiplied
//   LONG: one row of a K whose scales do not fit beside it: they are read from global memory as they are needed.
//            Plain or normed
enum Fuse { NONE, FUSED, SHARDED, ARGMAX, POSTNORM, LONG };

struct Args {
    const uint16_t* x;      // activations, bf16 [M][K] (fp32 when normed)
    void* y;
    PreNorm pre;
    uint32_t N, K, M;
    uint32_t ngrp, nsg;     // active groups of four warps; code stages per group
    uint32_t nsb;           // scale buffers of every set of groups that share a tile
    uint32_t kpar;          // groups that share a tile (1, 2 or 4), each taking every kpar-th slab
    uint32_t slab_row;      // bytes of a row in a slab: SLAB_ROW, or a shorter whole row rounded up to 128
    uint32_t inv_upr;       // ceil(2^32 / (K / 8))
    uint32_t out_bf16;
    uint32_t gated;         // SiLU x up of the two halves
    uint32_t early;         // prefetch before the predecessor is complete
    uint32_t n_total, row0; // the whole output's rows and this launch's first one
    const uint16_t *s, *b;  // scales and biases, [N][K / GROUP]
    PostNorm post;
    size_t y_off;
    unsigned long long* best;
    PeerArgs pa;
};

// The dynamic shared memory, identical on host and device (bytes from a 128-byte aligned base).
struct Layout {
    uint32_t qpitch, stage_bytes, sb_half, x_pitch;
    uint32_t sb, x, ms, zeros, red, total;
};
template <class S>
__host__ __device__ inline Layout layout(uint32_t K, uint32_t M, uint32_t stages, uint32_t sb_bufs, uint32_t slab_row,
                                         uint32_t red_bufs = Red<S::ROWS>::BUFS) {
    Layout L;
    L.qpitch = slab_row + S::QPAD;
    L.stage_bytes = 16u * L.qpitch;
    L.sb_half = 32u * (K / S::GROUP);  // 16 rows of scales (or of biases)
    const uint32_t kpad = (K + S::SK - 1u) / S::SK * S::SK;
    L.x_pitch = (2u * kpad + 127u) / 128u * 128u + S::XPAD;
    uint32_t at = stages * L.stage_bytes;
    L.sb = at;
    at += sb_bufs * 2u * L.sb_half;
    at = (at + 127u) / 128u * 128u;
    L.x = at;
    at += M * L.x_pitch;
    L.ms = at;
    at += (kpad / S::GROUP + 8u) * S::ROWS * 8u;  // (a last pass may read, not use, a few groups more)
    at = (at + 15u) / 16u * 16u;
    L.zeros = at;
    at += ZERO_BYTES;
    L.red = at;  // 16-byte aligned
    at += GROUPS * red_bufs * Red<S::ROWS>::FLOATS * 4u;  // last: nothing else lies by their number
    L.total = at;
    return L;
}

// ---- epilogues, shared by the kernels of the decode GEMV

// One output element: y[m][row0 + row].  N-sharded launch (pa.world > 1): this rank's rows [row0, row0 + N) of an
// n_total-row output go into its own y (at user offset y_off of its arena) and, as {value, launch number} packets,
// into every peer's inbox; before the CTA exits it collects its share of the peers' rows (peers.cuh).
// SHARDED is a template value rather than a run-time test because the single-GPU instantiation then compiles
// exactly as if the peer path did not exist (a run-time branch cost 3-16 %).
template <Fuse F, class A_>
__device__ __forceinline__ void store_out(const A_& A, uint32_t m, uint32_t row, float v, unsigned long long& my_best) {
    const size_t idx = (size_t)m * A.n_total + A.row0 + row;
    const uint32_t bits = A.out_bf16 ? float_to_bf16_bits(v) : __float_as_uint(v);
    if (A.out_bf16) reinterpret_cast<uint16_t*>(A.y)[idx] = (uint16_t)bits;
    else reinterpret_cast<uint32_t*>(A.y)[idx] = bits;
    if constexpr (F == ARGMAX) {  // compare what was stored (the rounded value when the output is bf16)
        if (v == v) {
            const unsigned long long key = peer_best_key(A.out_bf16 ? bits << 16 : bits, A.row0 + row);
            my_best = key > my_best ? key : my_best;
        }
    } else if constexpr (F == SHARDED) {
        if (A.pa.world > 1u) {
            const uint32_t e = peer_epoch(A.pa);
            const size_t elem = A.y_off / (A.out_bf16 ? 2u : 4u) + idx;
            for (uint32_t p = 0; p < A.pa.world; ++p)
                if (p != A.pa.rank) peer_send(peer_slot(A.pa, peer_arena(A.pa, p), e, elem), bits, e);
        }
    }
}
// gated: y[m][row] = bf16(silu(gate) * up) of the N/2-column output, with the arithmetic of the stand-alone
// activation kernel (shaders/ops.metal:129-139)
template <class A_>
__device__ __forceinline__ void store_gated(const A_& A, uint32_t m, uint32_t row, float gate, float up) {
    const float sg = gate / (1.0f + expf(-gate));
    reinterpret_cast<uint16_t*>(A.y)[(size_t)m * (A.N >> 1) + row] = (uint16_t)float_to_bf16_bits(sg * up);
}
// What the grid does together once its rows are stored.  Every thread of every CTA gets here, behind a CTA-wide
// barrier for all but the plain launch; WORK of the CTA's ALL warps have stored outputs.
template <Fuse F, int WORK, int ALL, class A_>
__device__ __forceinline__ void close_launch(const A_& A, unsigned long long my_best) {
    if constexpr (F == POSTNORM) {
        __shared__ float pn_part[neighbors::NORM_THREADS / 32];
        __shared__ uint32_t pn_last;
        __threadfence();  // this thread's rows of v are visible before the CTA reports in
        __syncthreads();
        if (threadIdx.x == 0) {
            pn_last = atomicAdd(A.post.arrivals, 1u) == gridDim.x - 1u ? 1u : 0u;
            __threadfence();
        }
        __syncthreads();
        if (pn_last && threadIdx.x < (uint32_t)neighbors::NORM_THREADS) {
            float* out = reinterpret_cast<float*>(A.y);
            for (uint32_t m = 0; m < A.M; ++m) {
                const size_t at = (size_t)m * A.N;
                neighbors::post_norm_add_any<9, true>(A.post.residual + at, out + at, A.post.gamma, out + at, A.N, A.post.eps,
                                                      pn_part, A.post.vec);
                neighbors::norm_sync<9>();  // pn_part is reused by the next row
            }
            if (threadIdx.x == 0) *A.post.arrivals = 0u;  // ready for the next launch
        }
    } else if constexpr (F == ARGMAX) {
        const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
        unsigned long long k = my_best;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long other = __shfl_xor_sync(0xFFFFFFFFu, k, o);
            k = other > k ? other : k;
        }
        __shared__ unsigned long long warp_keys[ALL];
        if (lane == 0) warp_keys[warp] = k;
        __syncthreads();
        if (threadIdx.x == 0) {
            for (uint32_t w = 1; w < (uint32_t)WORK; ++w) k = warp_keys[w] > k ? warp_keys[w] : k;
            if (k != 0ull) atomicMax(A.best, k);  // one candidate per CTA
            unsigned int* arrived = reinterpret_cast<unsigned int*>(A.best + 1);
            __threadfence();
            if (atomicAdd(arrived, 1u) == gridDim.x - 1u) {  // the last CTA: every candidate is in
                __threadfence();
                const unsigned long long win = atomicExch(A.best, 0ull);  // read, and reset for the next launch
                *arrived = 0u;
                uint32_t* pairs = reinterpret_cast<uint32_t*>(A.best) + 4;
                const size_t at = (size_t)(reinterpret_cast<uint8_t*>(pairs) - (A.pa.local + PEER_CTL_BYTES)) / 4u;
                peer_argmax_exchange(A.pa, pairs, at, peer_best_from_key(win));
            }
        }
    } else if constexpr (F == SHARDED) {
        if (A.pa.world > 1u) {
            const uint32_t e = peer_epoch(A.pa);
            __syncthreads();
            if (A.out_bf16) peer_collect<true>(A.pa, e, A.y_off, A.M, A.n_total, A.row0, A.N);
            else peer_collect<false>(A.pa, e, A.y_off, A.M, A.n_total, A.row0, A.N);
            __syncthreads();
            if (threadIdx.x == 0) peer_finish(A.pa, e);
        }
    }
}

template <class S, Fuse F>
__global__ void __launch_bounds__(THREADS, 1)
gemv_tma_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ Args A) {
    constexpr bool LONG_ = F == LONG;
    const bool gated = F == FUSED && S::BITS == 4 && S::ROWS <= 16 && A.gated != 0u, normed = (F == FUSED || LONG_) && A.pre.gamma != nullptr;
    constexpr bool SHARDED_ = F == SHARDED, ARGMAX_ = F == ARGMAX, POSTNORM_ = F == POSTNORM;
    constexpr int BITS = S::BITS, NT = S::NT, ROWS = S::ROWS, GPS = S::GPS, RC = S::RC;
    const uint32_t N = A.N, K = A.K, M = A.M, kpar = A.kpar, nsg = A.nsg, ngrp = A.ngrp;

    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t grp = warp < WARPS ? warp >> 2 : warp - WARPS;  // group of four warps, or its producer
    const uint32_t tiles = (N + 15u) >> 4;
    const uint32_t row_bytes = K * BITS / 8u, ng = K / S::GROUP;
    const uint32_t kslabs = (row_bytes + SLAB_ROW - 1u) / SLAB_ROW;

    extern __shared__ __align__(128) uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t full_bars[GROUPS * MAX_NSG], empty_bars[GROUPS * MAX_NSG];
    __shared__ __align__(8) uint64_t sb_full[GROUPS * MAX_NSG], sb_empty[GROUPS * MAX_NSG];
    __shared__ volatile uint32_t abort_flag;

    // A launch that may not start early waits here, and lets its dependents start only when its predecessor is
    // complete: they prefetch what that may have written.
    if (A.early == 0u) pdl_wait_prior();
    pdl_launch_dependents();

    // This CTA's tiles are dealt round-robin (tile = blockIdx.x + j * gridDim.x): at any moment the
    // CTAs stream one contiguous window of the weight matrix, which HBM serves best.  Group gi takes the
    // virtual tiles gi, gi + ngrp, ...  When a CTA has fewer tiles than groups and K spans several slabs,
    // kpar neighbouring groups share a tile: virtual tile v is tile v / kpar and slabs v % kpar,
    // v % kpar + kpar, ... of it, and the partial outputs are summed in a fixed order at the end (kslabs
    // and ngrp are multiples of kpar).  The group's k-th slab lives in its stage k % nsg; the scales of
    // its i-th tile in buffer i % nsb of the first of the groups that share it.
    const uint32_t kshift = kpar >> 1;  // log2
    const uint32_t my_tiles = (tiles - blockIdx.x + gridDim.x - 1u) / gridDim.x;
    const uint32_t vtiles = my_tiles << kshift, kp = grp & (kpar - 1u);
    const Layout L = layout<S>(K, M, ngrp * nsg, (ngrp >> kshift) * A.nsb, A.slab_row);
    const uint32_t base = smem_addr(smem_raw), qpitch = L.qpitch;
    const uint32_t bar0 = grp * nsg, sb0 = (grp >> kshift) * A.nsb;  // this group's first barriers

    if (warp >= WARPS) {
        // ---- producer of group `grp`: one lane.  Nothing here depends on the predecessor kernel.
        if (lane == 0) {
            abort_flag = 0u;  // by every producer: each reads it without having met the others
            if (grp < ngrp) {
                for (uint32_t i = 0; i < nsg; ++i) {
                    mbar_init(smem_addr(&full_bars[bar0 + i]), 1);
                    mbar_init(smem_addr(&empty_bars[bar0 + i]), 4);
                }
                if (kp == 0u)
                    for (uint32_t i = 0; i < A.nsb; ++i) {
                        mbar_init(smem_addr(&sb_full[sb0 + i]), 1);
                        mbar_init(smem_addr(&sb_empty[sb0 + i]), 4u * kpar);
                    }
            }
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        __syncwarp();
        asm volatile("bar.arrive 14, %0;" ::"n"(THREADS) : "memory");
        if (lane == 0 && grp < ngrp) {
            // next buffers, and the parities of their previous releases
            uint32_t st = 0, st_par = 1u, sb = 0, sb_par = 1u;
            bool st_wait = false, sb_wait = false, ok = true;
            // a buffer has to come back: the consumers start after the predecessor, and so does the time limit
            auto reuse = [&](uint64_t* empty, uint32_t parity, uint32_t where) {
                pdl_wait_prior();
                ok = mbar_wait(smem_addr(empty), parity, &abort_flag, where);
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                return ok;
            };
            uint32_t row = (blockIdx.x + (grp >> kshift) * gridDim.x) * 16u;
            const uint32_t row_step = (ngrp >> kshift) * gridDim.x * 16u;
            for (uint32_t vt = grp; vt < vtiles && ok; vt += ngrp, row += row_step) {
                // The tile's scales and biases come with its first slab, on the slab's barrier (their buffer is
                // free when that slab's stage is: plan_launch).  Groups that share a tile share one copy, made
                // by the first of them, with barriers of its own.
                const bool shared = kpar > 1u;
                uint32_t sb_bar = smem_addr(&full_bars[bar0 + st]), extra = 2u * L.sb_half;
                const uint32_t sdst = base + L.sb + (sb0 + sb) * 2u * L.sb_half;
                const uint32_t r0 = gated ? row >> 1 : row;  // gated: N is a multiple of 16, eight whole rows of each half
                const uint8_t* src_s = reinterpret_cast<const uint8_t*>(A.s) + (size_t)r0 * (2u * ng);
                const uint8_t* src_b = reinterpret_cast<const uint8_t*>(A.b) + (size_t)r0 * (2u * ng);
                if (!LONG_ && row + 16u > N && kp == 0u) {  // a ragged last tile: whole 16-byte pieces by bulk copy ...
                    if (!shared && st_wait && !reuse(&empty_bars[bar0 + st], st_par, 0x16)) break;
                    if (shared && sb_wait && !reuse(&sb_empty[sb0 + sb], sb_par, 0x15)) break;
                    const uint32_t n = (N - row) * ng;
                    extra = (2u * n & ~15u) * 2u;
                    for (uint32_t i = n & ~7u; i < n; ++i) {  // ... the rest by this thread, before it arrives
                        asm volatile("st.shared.u16 [%0], %1;" ::"r"(sdst + 2u * i), "h"(reinterpret_cast<const uint16_t*>(src_s)[i]) : "memory");
                        asm volatile("st.shared.u16 [%0], %1;" ::"r"(sdst + L.sb_half + 2u * i), "h"(reinterpret_cast<const uint16_t*>(src_b)[i]) : "memory");
                    }
                }
                auto copy_sb = [&] {
                    if (gated) {
                        const uint32_t half = L.sb_half >> 1;
                        const size_t up = (size_t)(N >> 1) * (2u * ng);
                        bulk_g2s(sdst, src_s, half, sb_bar);
                        bulk_g2s(sdst + half, src_s + up, half, sb_bar);
                        bulk_g2s(sdst + L.sb_half, src_b, half, sb_bar);
                        bulk_g2s(sdst + L.sb_half + half, src_b + up, half, sb_bar);
                    } else if (extra) {
                        bulk_g2s(sdst, src_s, extra >> 1, sb_bar);
                        bulk_g2s(sdst + L.sb_half, src_b, extra >> 1, sb_bar);
                    }
                };
                if (!LONG_ && shared && kp == 0u) {
                    sb_bar = smem_addr(&sb_full[sb0 + sb]);
                    if (sb_wait && !reuse(&sb_empty[sb0 + sb], sb_par, 0x15)) break;
                    mbar_expect_tx(sb_bar, extra);
                    copy_sb();
                }
                for (uint32_t ks = kp; ks < kslabs; ks += kpar) {
                    const uint32_t bar = smem_addr(&full_bars[bar0 + st]), dst = base + (bar0 + st) * L.stage_bytes;
                    if (st_wait && !reuse(&empty_bars[bar0 + st], st_par, 0x14)) break;
                    const int c0 = (int)(ks * (SLAB_ROW / 8u));
                    const bool with_sb = !LONG_ && !shared && ks == 0u;
                    mbar_expect_tx(bar, L.stage_bytes + (with_sb ? extra : 0u));
                    if (gated) {  // the tensor map's boxes are eight rows high
                        tma_load_2d(dst, &tmap_q, c0, (int)r0, bar);
                        tma_load_2d(dst + 8u * qpitch, &tmap_q, c0, (int)((N >> 1) + r0), bar);
                    } else {
                        tma_load_2d(dst, &tmap_q, c0, (int)row, bar);
                    }
                    if (with_sb) copy_sb();
                    if (++st == nsg) st = 0u, st_wait = true, st_par ^= 1u;
                }
                if (++sb == A.nsb) sb = 0u, sb_wait = true, sb_par ^= 1u;
            }
        }
        __syncwarp();
    }

    // y is one launch's output; ARGMAX: key of the best element this thread has stored
    unsigned long long my_best = 0ull;
    if (warp < WARPS) {
        // zeros: what lanes of other slots read, and the activations past the end of K
        const XArea xa = {base + L.x, L.x_pitch, base + L.ms};
        const uint32_t tid = threadIdx.x;
        if (tid < ZERO_BYTES / 16u) *reinterpret_cast<uint4*>(smem_raw + L.zeros + 16u * tid) = make_uint4(0u, 0u, 0u, 0u);
        if (const uint32_t tail = (K + S::SK - 1u) / S::SK * S::SK - K) {
            for (uint32_t i = tid; i < M * (tail >> 3); i += COMPUTE) {
                const uint32_t m = i / (tail >> 3), u = i - m * (tail >> 3);
                *reinterpret_cast<uint4*>(smem_raw + L.x + m * L.x_pitch + 2u * K + 16u * u) = make_uint4(0u, 0u, 0u, 0u);
            }
        }

        pdl_wait_prior();  // x (and y) belong to the predecessor until here

        if (normed) {
            __shared__ float nm_part[4][WARPS];
            __shared__ float nm_inv[32];
            stage_x_normed<S>(xa, reinterpret_cast<const float*>(A.x), A.pre.gamma, A.pre.eps, M, K, A.inv_upr, nm_part, nm_inv);
        } else {
            stage_x<S>(xa, A.x, M, K, A.inv_upr);
        }
        asm volatile("bar.sync 14, %0;" ::"n"(THREADS) : "memory");  // x is staged, the barriers exist

        auto store_out = [&](uint32_t m, uint32_t row, float v) { gemvtma::store_out<F>(A, m, row, v, my_best); };

        // ---- this lane's place in the MMAs.  As a B operand it supplies column n = lane / 4 = (slot n / RC,
        // row n % RC); as an accumulator it holds columns 2 t and 2 t + 1.
        const uint32_t g = lane >> 2, t = lane & 3u, wg = warp & 3u;
        const uint32_t sl = S::SLOTTED ? 2u * t / RC : 0u, m_acc = S::SLOTTED ? 2u * t % RC : 2u * t;
        uint32_t xb[NT];
#pragma unroll
        for (int j = 0; j < NT; ++j)  // columns past M repeat the last row: results nobody reads
            xb[j] = xa.x + min((uint32_t)(8 * j) + g % (uint32_t)RC, M - 1u) * xa.pitch + t * (uint32_t)S::XB;
        const uint32_t zeros = base + L.zeros;
        const uint32_t q_lane = g * qpitch + t * (uint32_t)S::W;
        // where scales and biases lie from row g's scales; LONG: bits of the number that stands for their address
        const uint32_t sb_row = LONG_ ? 0u : g * ng * 2u, sb_row8 = LONG_ ? 1u : 8u * ng * 2u, sb_half = LONG_ ? 2u : L.sb_half;
        uint32_t long_row = 0;  // LONG: this lane's first row of the tile
        using R = Red<ROWS>;
        const bool vec_sb = ng % 8u == 0u;  // rows of scales start on 16-byte boundaries

        float acc[S::ACCN][4];
#pragma unroll
        for (int j = 0; j < S::ACCN; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.0f;

        // d: sums of columns 2t, 2t + 1 for tile rows g (first two) and g + 8.  ms: {power of two, sum} of both
        // columns; s, b: scales and biases of [row][column]
        auto apply = [&](float (&a)[4], const float (&d)[4], const float4& ms, float s00, float s01, float s10, float s11,
                         float b00, float b01, float b10, float b11) {
            a[0] = __fmaf_rn(s00 * ms.x, d[0], __fmaf_rn(b00, ms.y, a[0]));
            a[1] = __fmaf_rn(s01 * ms.z, d[1], __fmaf_rn(b01, ms.w, a[1]));
            a[2] = __fmaf_rn(s10 * ms.x, d[2], __fmaf_rn(b10, ms.y, a[2]));
            a[3] = __fmaf_rn(s11 * ms.z, d[3], __fmaf_rn(b11, ms.w, a[3]));
        };

        // A run: `steps` steps (four when FULL) of 64 bytes of every row from shared address qa on (row g, this
        // lane's piece), activations xo bytes into the staged rows, first scale group grp0, scales of row g at sa.
        auto run_math = [&](auto full, uint32_t qa, uint32_t xo, uint32_t grp0, uint32_t sa, uint32_t steps) {
            constexpr bool FULL = decltype(full)::value;
            // FULL: the run's scales and biases by one or two wide loads per row (RC == 1 reads pairs in place)
            constexpr int SW = 2 * GPS;  // words: 4 GPS bf16 values
            uint32_t vs0[SW], vb0[SW], vs1[SW], vb1[SW];
            if constexpr (FULL && RC > 1) {
                lds_words<4 * SW>(vs0, sa + 2u * grp0);
                lds_words<4 * SW>(vb0, sa + 2u * grp0 + sb_half);
                lds_words<4 * SW>(vs1, sa + 2u * grp0 + sb_row8);
                lds_words<4 * SW>(vb1, sa + 2u * grp0 + sb_row8 + sb_half);
            }
            const uint32_t half = (sl & 1u) ? 0x3244u : 0x1044u;
            // fp32 value of the run's group c + (SLOTTED: this lane's slot)
            auto pick = [&](const uint32_t (&v)[SW], int c) -> float {
                if constexpr (!S::SLOTTED) return c & 1 ? bf16hi(v[c >> 1]) : bf16lo(v[c >> 1]);
                else if constexpr (S::SLOTS == 4) {
                    if constexpr (SW > 2) return __uint_as_float(__byte_perm((sl & 2u) ? v[(c >> 1) + 1] : v[c >> 1], 0u, half));
                    else return __uint_as_float(__byte_perm((sl & 2u) ? v[1] : v[0], 0u, half));
                } else return __uint_as_float(__byte_perm(v[c >> 1], 0u, half));
            };
            // not FULL: groups of steps that are not this run's, or past the end of K, count as zero
            const uint32_t glim = min(ng, grp0 + steps * GPS);
            auto one = [&](uint32_t at, uint32_t gi) {
                if constexpr (LONG_) {
                    const uint16_t* p = (at & 2u ? A.b : A.s) + (size_t)min(long_row + 8u * (at & 1u), N - 1u) * ng;
                    return __uint_as_float(gi < glim ? (uint32_t)__ldg(p + gi) << 16 : 0u);
                } else {
                    return __uint_as_float(gi < glim ? lds16(at + 2u * gi) << 16 : 0u);
                }
            };
            // apply the sums d to acc: c = first group of the accumulator relative to the run
            auto scale = [&](float (&a)[4], const float (&d)[4], int c, int j) {
                if constexpr (RC == 1) {
                    // two neighbouring groups, one row; with fewer than eight groups a run the upper lanes have
                    // no group: their sums are zero, and their biases count as zero
                    constexpr bool SHORT = 4 * GPS < 8;
                    const uint32_t p = grp0 + (uint32_t)c + (SHORT ? 2u * (t & 1u) : 2u * t);
                    if constexpr (FULL) {
                        const uint32_t s0 = lds32(sa + 2u * p), s1 = lds32(sa + 2u * p + sb_row8);
                        uint32_t b0 = lds32(sa + 2u * p + sb_half), b1 = lds32(sa + 2u * p + sb_row8 + sb_half);
                        if (SHORT && t >= 2u) b0 = b1 = 0u;
                        apply(a, d, ldsf128(xa.ms + p * 8u), bf16lo(s0), bf16hi(s0), bf16lo(s1), bf16hi(s1), bf16lo(b0),
                              bf16hi(b0), bf16lo(b1), bf16hi(b1));
                    } else {
                        const uint32_t lim = SHORT && t >= 2u ? 0u : 2u;
                        const uint32_t p0 = lim ? p : glim, p1 = lim ? p + 1u : glim;
                        float4 ms = ldsf128(xa.ms + (p & ~1u) * 8u);  // (p is even unless the run starts on an odd group)
                        if (p & 1u) {
                            const float4 nx = ldsf128(xa.ms + (p + 1u) * 8u);
                            ms = make_float4(ms.z, ms.w, nx.x, nx.y);
                        }
                        if (p0 >= glim) ms.x = ms.y = 0.0f;
                        if (p1 >= glim) ms.z = ms.w = 0.0f;
                        apply(a, d, ms, one(sa, p0), one(sa, p1), one(sa + sb_row8, p0), one(sa + sb_row8, p1),
                              one(sa + sb_half, p0), one(sa + sb_half, p1), one(sa + sb_row8 + sb_half, p0),
                              one(sa + sb_row8 + sb_half, p1));
                    }
                } else {
                    const uint32_t gi = grp0 + (uint32_t)c + sl;
                    float4 ms = ldsf128(xa.ms + (gi * ROWS + (uint32_t)(8 * j) + m_acc) * 8u);
                    float s0, s1, b0, b1;
                    if constexpr (FULL) {
                        s0 = pick(vs0, c), s1 = pick(vs1, c), b0 = pick(vb0, c), b1 = pick(vb1, c);
                    } else {
                        s0 = one(sa, gi), s1 = one(sa + sb_row8, gi), b0 = one(sa + sb_half, gi), b1 = one(sa + sb_row8 + sb_half, gi);
                        if (gi >= glim) ms = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    }
                    apply(a, d, ms, s0, s0, s1, s1, b0, b0, b1, b1);
                }
            };
            using AF = AFrag<BITS, S::NW>;
            if constexpr (S::SLOTTED) {
#pragma unroll
                for (int p = 0; p < 4 / S::SPA; ++p) {
                    if (!FULL && (uint32_t)(p * S::SPA) >= steps) break;
                    float d[S::SETS][2][4];  // two chains each
#pragma unroll
                    for (int i = 0; i < S::SPA; ++i) {
                        const int step = p * S::SPA + i;
                        if (!FULL && (uint32_t)step >= steps) break;
                        uint32_t q0[4], q1[4];
                        lds_words<16>(q0, qa + (uint32_t)step * STEP_BYTES);
                        lds_words<16>(q1, qa + (uint32_t)step * STEP_BYTES + 8u * qpitch);
                        AF a;
                        a.unpack(q0, q1);
#pragma unroll
                        for (int j = 0; j < S::SETS; ++j) {
                            // this lane's codes belong to slot i GPS + t GPS / 4 of the pass
                            const bool active = g / (uint32_t)RC + (uint32_t)(j * S::SLOTS) == (uint32_t)(i * GPS) + t * (uint32_t)GPS / 4u;
                            const uint32_t x_at = active ? xb[0] + xo + (uint32_t)step * 2u * S::SK : zeros;
#pragma unroll
                            for (int k = 0; k < AF::MMAS; k += 2) {
                                const uint4 b = lds128(x_at + 8u * k);
                                a.mma(i == 0 && k == 0, k, d[j][0], b.x, b.y);
                                a.mma(i == 0 && k == 0, k + 1, d[j][1], b.z, b.w);
                            }
                        }
                    }
#pragma unroll
                    for (int j = 0; j < S::SETS; ++j) {
                        const float sum[4] = {d[j][0][0] + d[j][1][0], d[j][0][1] + d[j][1][1], d[j][0][2] + d[j][1][2], d[j][0][3] + d[j][1][3]};
                        scale(acc[(p * S::SETS + j) % S::ACCN], sum, p * S::SPA * GPS + j * S::SLOTS, 0);
                    }
                }
            } else {
#pragma unroll
                for (int step = 0; step < 4; ++step) {
                    if (!FULL && (uint32_t)step >= steps) break;
#pragma unroll
                    for (int c = 0; c < S::CH; ++c) {
                        uint32_t q0[S::NW], q1[S::NW];
                        lds_words<S::W>(q0, qa + (uint32_t)step * STEP_BYTES + (uint32_t)(c * 4 * S::W));
                        lds_words<S::W>(q1, qa + (uint32_t)step * STEP_BYTES + (uint32_t)(c * 4 * S::W) + 8u * qpitch);
                        AF a;
                        a.unpack(q0, q1);
#pragma unroll
                        for (int j = 0; j < NT; ++j) {
                            float d[4];
#pragma unroll
                            for (int k = 0; k < AF::MMAS; k += 2) {
                                const uint4 b = lds128(xb[j] + xo + (uint32_t)step * 2u * S::SK + (uint32_t)(c * 4 * S::XB) + 8u * k);
                                a.mma(k == 0, k, d, b.x, b.y);
                                a.mma(false, k + 1, d, b.z, b.w);
                            }
                            scale(acc[j], d, step * GPS + c, j);
                        }
                    }
                }
            }
        };

        // `ok` turns false for good once a wait expires; the warp then skips waits and math but still takes
        // part in every group barrier so that no other warp is left waiting.
        bool ok = true;
        uint32_t tile_it = 0, st = 0, st_par = 0, sb = 0, sb_par = 0;
        auto wait = [&](uint64_t* bar, uint32_t parity, uint32_t where) {
            if (!ok) return;
            if (__all_sync(0xFFFFFFFFu, mbar_try_long(smem_addr(bar), parity))) return;
            ok = mbar_wait(smem_addr(bar), parity, &abort_flag, where);
            ok = __all_sync(0xFFFFFFFFu, ok);
        };
        const uint32_t gt = wg * 32u + lane;  // thread index inside the group
        for (uint32_t vt = grp; grp < ngrp && vt < vtiles; vt += ngrp) {
            const uint32_t sa = LONG_ ? 0u : base + L.sb + (sb0 + sb) * 2u * L.sb_half + sb_row;
            if (LONG_) long_row = (blockIdx.x + (vt >> kshift) * gridDim.x) * 16u + g;
            else if (kpar > 1u) wait(&sb_full[sb0 + sb], sb_par, 0x12);
            for (uint32_t ks = kp; ks < kslabs; ks += kpar) {
                wait(&full_bars[bar0 + st], st_par, 0x10);
                if (ok) {
                    // steps of this slab, dealt to the warps in runs: four each in a full slab
                    const uint32_t left = row_bytes - ks * SLAB_ROW;
                    const uint32_t qa = base + (bar0 + st) * L.stage_bytes + q_lane;
                    if (!LONG_ && vec_sb && left >= SLAB_ROW) {
                        run_math(std::true_type(), qa + wg * 4u * STEP_BYTES, 2u * (ks * S::KC + wg * 4u * S::SK),
                                 ks * (S::KC / S::GROUP) + wg * 4u * GPS, sa, 4u);
                    } else {
                        const uint32_t nsteps = (min(left, SLAB_ROW) + STEP_BYTES - 1u) / STEP_BYTES;
                        const uint32_t run = (nsteps + 3u) >> 2, step0 = wg * run;
                        if (step0 < nsteps)
                            run_math(std::false_type(), qa + step0 * STEP_BYTES, 2u * (ks * S::KC + step0 * S::SK),
                                     ks * (S::KC / S::GROUP) + step0 * GPS, sa, min(run, nsteps - step0));
                    }
                    __syncwarp();
                    if (lane == 0) mbar_arrive(smem_addr(&empty_bars[bar0 + st]));  // stage consumed
                }
                if (++st == nsg) st = 0u, st_par ^= 1u;
            }
            if (!LONG_ && kpar > 1u && ok && lane == 0) mbar_arrive(smem_addr(&sb_empty[sb0 + sb]));
            if (++sb == A.nsb) sb = 0u, sb_par ^= 1u;

            // ---- tile complete: the classes of groups in a fixed tree, then the warps' partials (and those of
            // the groups that share the tile) through shared memory
            const uint32_t red0 = base + L.red + (R::BUFS == 2 ? (tile_it & 1u) * (uint32_t)(GROUPS * R::FLOATS * 4) : 0u);
            const uint32_t mine = red0 + grp * (uint32_t)(R::FLOATS * 4) + wg * 4u;  // + 16 * (m * 16 + tile row)
            auto put = [&](uint32_t m, uint32_t r, float v) {
                asm volatile("st.shared.f32 [%0], %1;" ::"r"(mine + (m * 16u + r) * 16u), "f"(v) : "memory");
            };
            auto xor_add = [](float v, int o) { return v + __shfl_xor_sync(0xFFFFFFFFu, v, o); };
            if constexpr (RC == 1) {
                const float v0 = xor_add(xor_add(acc[0][0] + acc[0][1], 1), 2), v1 = xor_add(xor_add(acc[0][2] + acc[0][3], 1), 2);
                if (t < 2u) put(0u, g + 8u * t, t ? v1 : v0);
            } else if constexpr (S::SLOTTED) {
                float r[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    float v[S::ACCN];
#pragma unroll
                    for (int a = 0; a < S::ACCN; ++a) {
                        v[a] = acc[a][e];
                        if constexpr (RC == 2) v[a] = xor_add(v[a], 1);
                        v[a] = xor_add(v[a], 2);
                    }
                    r[e] = v[0];
                    if constexpr (S::ACCN == 2) r[e] = v[0] + v[1];
                    if constexpr (S::ACCN == 4) r[e] = (v[0] + v[1]) + (v[2] + v[3]);
                }
                if constexpr (RC == 2) {  // every lane of the quad has all four: each stores one
                    put(t & 1u, g + 8u * (t >> 1), t == 0u ? r[0] : t == 1u ? r[1] : t == 2u ? r[2] : r[3]);
                } else {                  // lanes t and t ^ 2 have the same four: two each
                    const bool up = t >= 2u;
                    put(m_acc, g + (up ? 8u : 0u), up ? r[2] : r[0]);
                    put(m_acc + 1u, g + (up ? 8u : 0u), up ? r[3] : r[1]);
                }
            } else {
#pragma unroll
                for (int j = 0; j < NT; ++j)
#pragma unroll
                    for (int e = 0; e < 4; ++e) put(8u * j + m_acc + (e & 1), g + 8u * (e >> 1), acc[j][e]);
            }
#pragma unroll
            for (int j = 0; j < S::ACCN; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.0f;
            named_barrier(1u + (grp >> kshift), kpar * 128u);
            // output o = m * 16 + r of the tile: warps first, then groups, in order
            auto total = [&](uint32_t o) {
                float v = 0.0f;
                for (uint32_t j = 0; j < kpar; ++j) {
                    const float4 p = ldsf128(red0 + (grp + j) * (uint32_t)(R::FLOATS * 4) + o * 16u);
                    const float w = (p.x + p.y) + (p.z + p.w);
                    v = j == 0u ? w : v + w;
                }
                return v * UNSCALE<BITS>;
            };
            const uint32_t tile = blockIdx.x + (vt >> kshift) * gridDim.x;
            if (kp == 0u && ok) {
                if (gated) {  // tile rows 0 .. 7 are gates, 8 .. 15 the same outputs' up rows
                    for (uint32_t i = gt; i < 8u * M; i += 128u) {
                        const uint32_t m = i >> 3, r = i & 7u;
                        store_gated(A, m, tile * 8u + r, total(m * 16u + r), total(m * 16u + r + 8u));
                    }
                } else {
                    for (uint32_t o = gt; o < 16u * M; o += 128u) {
                        const uint32_t row = tile * 16u + (o & 15u);
                        const float v = total(o);
                        if (row < N) store_out(o >> 4, row, v);
                    }
                }
            }
            if constexpr (R::BUFS == 1) named_barrier(1u + (grp >> kshift), kpar * 128u);
            ++tile_it;
        }
    }

    if constexpr (POSTNORM_ || ARGMAX_ || SHARDED_) __syncthreads();  // the producers are done too
    if (abort_flag) {  // let copies still in flight land before the CTA's memory is released
        const long long t0 = clock64();
        while (clock64() - t0 < 2000000LL) __nanosleep(1000);
    }
    close_launch<F, WARPS, THREADS / 32>(A, my_best);
}

// Placement of an N-sharded launch's output and the fused neighbours of a launch: peers (world <= 1:
// none, y is a plain pointer), rows of the whole output, this rank's first row, and the offset of y
// inside every arena.
struct Shard {
    PeerArgs pa = {};
    uint32_t n_total = 0, row0 = 0;
    size_t y_off = 0;
    // arg-max epilogue (one activation row): 16 bytes of zeroed scratch {key, arrivals} followed by
    // the (2 world + 2) words of the candidates and the winner, inside the local arena; null: off
    unsigned long long* best = nullptr;
    // gated epilogue (4-bit weights, one GPU): rows [0, N/2) are the gate and [N/2, N) the up
    // projection, y is bf16 [M][N/2] of silu(gate) * up
    bool gated = false;
    // post-norm epilogue (4-bit weights, fp32 out, up to four rows, one GPU); residual null: off
    PostNorm post;
    // norm prologue (one GPU): x is fp32; gamma null: off
    PreNorm pre;
};

// Whether a form of M rows exists.
inline int check_fuse(const Shard& sh, int bits, uint32_t N, uint32_t M, bool out_bf16) {
    const bool sharded = sh.pa.world > 1, argmax = sh.best != nullptr, postnorm = sh.post.residual != nullptr, normed = sh.pre.gamma != nullptr;
    if ((int)argmax + (int)postnorm + (int)(sharded && !argmax) + (int)(sh.gated || normed) > 1)
        return fail(MIORI_E_INVALID, "gemv: this combination of fused neighbours does not exist");
    if (argmax && M != 1u) return fail(MIORI_E_INVALID, "the arg-max epilogue takes one activation row");
    if (postnorm && (bits != 4 || out_bf16 || M > 4u))
        return fail(MIORI_E_INVALID, "the post-norm epilogue takes 4-bit weights, up to four rows, fp32 out");
    if (sh.gated && (bits != 4 || N % 16 != 0 || M > (normed ? 4u : 16u)))
        return fail(MIORI_E_INVALID, "the gated epilogue takes 4-bit weights with N a multiple of 16, up to 16 rows "
                                     "(four with the norm in front)");
    return MIORI_OK;
}

// Launch plan: CTAs, active groups, stages per group, scale buffers.
struct Plan {
    uint32_t grid = 0, ngrp = 0, nsg = 0, nsb = 0, kpar = 1, slab_row = 0;
    size_t smem = 0;
};
// One CTA per SM, which also claims more than half of the SM's shared memory, so that no second CTA of
// any kernel of this family can join it.  Sharing an SM with the successor of a dependent-launch chain
// looks attractive (it prefetches while this one computes) but the placement is not stable: after a
// launch with another footprint the successor's CTAs double up on the SMs that were free and leave
// others without one, every later launch inherits the skew, and a 24-layer chain of four shapes ran
// 17 % slower than the sum of its parts.  With the SM to itself a CTA starts as its predecessor's CTA
// exits, fills its ring during the hand-over between the grids, and the placement is one CTA per SM
// whatever ran before.
constexpr size_t SMEM_LIMIT = 222 * 1024;

// What a launch's size is made of: 16-row tiles of the busiest CTA, slabs of a row.
struct Extent {
    uint32_t tiles, grid, tiles_cta, kslabs, slab_row;
};
template <class S>
Extent extent(uint32_t N, uint32_t K) {
    Extent e;
    const uint32_t row_bytes = K * S::BITS / 8u;
    e.tiles = (N + 15u) / 16u;
    e.grid = std::min<uint32_t>(e.tiles, (uint32_t)sm_count());
    e.tiles_cta = (e.tiles + e.grid - 1u) / e.grid;
    e.kslabs = (row_bytes + SLAB_ROW - 1u) / SLAB_ROW;
    e.slab_row = row_bytes >= SLAB_ROW ? SLAB_ROW : (row_bytes + 127u) / 128u * 128u;
    return e;
}
// Shared memory of a launch whose busiest group has `each` tiles (one reduction buffer is enough for one).
template <class S>
size_t smem_bytes(const Extent& e, uint32_t K, uint32_t M, uint32_t ngrp, uint32_t nsg, uint32_t nsb, uint32_t kpar, uint32_t each) {
    return layout<S>(K, M, ngrp * nsg, ngrp / kpar * nsb, e.slab_row, each == 1u ? 1u : (uint32_t)Red<S::ROWS>::BUFS).total;
}

// How many groups share a tile: with few tiles per CTA and a long K two or four, each taking every kpar-th slab,
// as far as M rows of activations, and a tile's scales, leave room for a stage each.  0: M rows do not fit.
template <class S>
uint32_t choose_kpar(uint32_t N, uint32_t K, uint32_t M, bool scales = true) {
    if (K > (1u << 20)) return 0u;  // (the sums below stay inside 32 bits)
    const Extent e = extent<S>(N, K);
    uint32_t kpar = 1u;
    while (kpar * 2u <= (uint32_t)GROUPS && e.tiles_cta * kpar * 2u <= (uint32_t)GROUPS && e.kslabs % (kpar * 2u) == 0u) kpar *= 2u;
    for (; kpar >= 1u; kpar >>= 1)
        // (whether M rows fit at all must not depend on N: ranks with shards of different heights launch alike)
        if (smem_bytes<S>(e, K, M, kpar, 1u, scales ? 1u : 0u, kpar, kpar == 1u ? 2u : e.tiles_cta) <= SMEM_LIMIT) return kpar;
    return 0u;
}

// The plan for M rows with kpar groups to a tile, which fit.
template <class S>
Plan plan_launch(uint32_t N, uint32_t K, uint32_t M, uint32_t kpar, bool scales = true) {
    Plan p;
    const Extent e = extent<S>(N, K);
    p.grid = e.grid, p.kpar = kpar, p.slab_row = e.slab_row;
    const uint32_t vtiles = e.tiles_cta * kpar, own = e.kslabs / kpar;  // slabs of a tile per group
    uint32_t most = std::min<uint32_t>(GROUPS, vtiles);
    most -= most % kpar;
    for (uint32_t ngrp = most; ngrp >= kpar; ngrp -= kpar) {
        const uint32_t each = (vtiles + ngrp - 1u) / ngrp;  // tiles of the busiest group
        for (uint32_t nsg = std::min<uint32_t>(MAX_NSG, each * own); nsg >= 1u; --nsg) {
            // scales of every tile the code stages reach into: when the stage of a tile's first slab is
            // free, so is the buffer of the tile nsb before it
            const uint32_t nsb = scales ? std::min(each, (nsg - 1u + own - 1u) / own + 1u) : 0u;
            const size_t bytes = smem_bytes<S>(e, K, M, ngrp, nsg, nsb, kpar, each);
            if (bytes > SMEM_LIMIT) continue;
            p.ngrp = ngrp, p.nsg = nsg, p.nsb = nsb;
            p.smem = std::max<size_t>(bytes, 120 * 1024);
            return p;
        }
    }
    return p;
}

template <class S, Fuse F>
int launch_one(const Plan& plan, const void* q, const Args& a, cudaStream_t stream) {
    const bool gated = a.gated != 0u;
    CUtensorMap tq;
    // rows as 64-bit words, so that the box can be wider than 256 words of 32 bits; gated: a tile is two
    // boxes, one from each half
    const int rc = make_tmap_2d(&tq, q, CU_TENSOR_MAP_DATA_TYPE_UINT64, 8, (uint64_t)a.K * S::BITS / 64, a.N,
                                (plan.slab_row + S::QPAD) / 8, gated ? 8 : 16, CU_TENSOR_MAP_SWIZZLE_NONE);
    if (rc) return rc;
    // always with the programmatic attribute (the kernel knows when to wait): 2.0 us of host time against 2.5
    const cudaError_t e = launch(gemv_tma_kernel<S, F>, dim3(plan.grid), dim3(THREADS), plan.smem, stream, true, tq, a);
    if (e != cudaSuccess) return cuda_fail(e, "gemv_tma launch");
    return MIORI_OK;
}

template <class S>
int launch_shape(const void* q, const void* s, const void* b, const void* x, void* y, uint32_t N, uint32_t K, uint32_t M,
                 uint32_t flags, cudaStream_t stream, const Shard& sh, uint32_t kpar, bool wide_k = false) {
    const Plan plan = plan_launch<S>(N, K, M, kpar, !wide_k);
    if (plan.ngrp == 0) return fail(MIORI_E_INVALID, "gemv: no plan for N=%u K=%u M=%u", N, K, M);
    constexpr bool FEW = S::ROWS <= 4 || (S::ROWS == 8 && S::GROUP == 64);  // shapes that up to four 4-bit rows run on
    const bool sharded = sh.pa.world > 1, argmax = sh.best != nullptr;
    const bool postnorm = sh.post.residual != nullptr, normed = sh.pre.gamma != nullptr;
    const bool placed = sharded || argmax;  // y is a slice of an n_total-row output
    Args a;
    a.s = static_cast<const uint16_t*>(s);
    a.b = static_cast<const uint16_t*>(b);
    a.x = static_cast<const uint16_t*>(x);
    a.y = y;
    a.N = N, a.K = K, a.M = M;
    a.ngrp = plan.ngrp, a.nsg = plan.nsg, a.nsb = plan.nsb, a.kpar = plan.kpar, a.slab_row = plan.slab_row;
    a.inv_upr = (uint32_t)((0x100000000ull + K / 8u - 1u) / (K / 8u));
    a.out_bf16 = flags & MIORI_OUT_BF16 ? 1u : 0u;
    a.gated = sh.gated ? 1u : 0u;
    a.n_total = placed ? sh.n_total : N, a.row0 = placed ? sh.row0 : 0u, a.y_off = sh.y_off;
    a.best = sh.best, a.pa = sh.pa, a.post = sh.post, a.pre = sh.pre;
    a.early = (flags & MIORI_LAUNCH_PDL) != 0 ? 1u : 0u;
    const int rc = check_fuse(sh, S::BITS, N, M, a.out_bf16 != 0u);
    if (rc) return rc;
    if (argmax) {
        if constexpr (S::ROWS == 1) return launch_one<S, ARGMAX>(plan, q, a, stream);
    }
    if (postnorm) {
        if constexpr (S::BITS == 4 && FEW) return launch_one<S, POSTNORM>(plan, q, a, stream);
    }
    if constexpr (S::ROWS == 1)
        if (wide_k) return launch_one<S, LONG>(plan, q, a, stream);
    if (normed || sh.gated) return launch_one<S, FUSED>(plan, q, a, stream);
    if (sharded) return launch_one<S, SHARDED>(plan, q, a, stream);
    return launch_one<S, NONE>(plan, q, a, stream);
}

}  // namespace gemvtma
}  // namespace miori_b200
