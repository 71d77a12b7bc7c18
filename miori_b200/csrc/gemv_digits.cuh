// The decode GEMV for one and two activation rows on 4-bit weights in groups of 64, K a multiple of 256 up to 8192.
//
//   y[m][n] = sum_g ( s[n][g] * sum_{k in g} code[n][k] * x[m][k]  +  b[n][g] * sum_{k in g} x[m][k] )
//
// The inner sum runs on mma.sync.m16n8k32 with 8-bit integers, and exactly:
//   * a word of eight 4-bit codes becomes two A registers with two ANDs and no shift: the low nibbles as they
//     are, the high ones where they stand, counting sixteen times as much;
//   * an activation is an integer below 2^26 -- its group's largest decides the power of two; bf16's eight bits
//     are exact for everything of at least 2^-17 of the largest, the rest is rounded by less than 2^-25 of it
//     -- times sixteen for the codes in low nibbles, cut into four digits of -128 .. 127, a column of the MMA
//     each.  With one row the eight columns are the digits of two groups, with two rows those of one.
// What the rounding costs shows only where the large activation's weight is exactly zero.  One of 2^12 a group, the others
// normal, error of the result here and with the fp16 operands of gemv_tma.cuh: its code 8 and b = -8 s 4.7e-5 and 7.0e-4, code
// 1 and b = -s 2.3e-6 and 4.4e-4 (fp16 products are cut off where they meet the large one in the tensor core), code 0 and b = 0
// 1.6e-5 and 4e-8.  b is that small only in a group whose weights hardly reach beyond zero, or to it from one side.
// A row's sums are int32, then fp32 per group: its bits depend neither on the other row, nor on the launch, nor on the grid.
// (The fp16 operands of gemv_tma.cuh take twice the MMAs and three times the ALU work for the unpacking, which
// are worth it only where the columns are full of rows.)
//
// What bounds it: the steps of a launch that follow one another -- the hand-over from grid to grid (0.7 us), the trip of x
// through L2 (0.35), its conversion (0.3; 0.25 a slab beyond with eight warps), each piece of weights (0.33) -- and not HBM.
//   * A 1-KiB slab of a row is cut into eight positions of 128 bytes, and a warp owns a position of the CTA's tiles: it
//     fetches its own pieces (16 rows x 128 bytes by TMA, 128-byte swizzle, and their scales by cp.async) into its own
//     ring, and converts the activations of its own position.  Warps meet once per batch of tiles, when the partial sums
//     of an output are added in a fixed tree.  (With the activations staged by the whole CTA behind a barrier a layer
//     took 4 % more.)
//   * K <= 2048: the activations stay in registers from tile to tile.
//   * The first piece is read while x is on its way.
// Two frames, the same bits:
//   * one row started early, up to 192 KiB of codes an SM: EIGHT warps a CTA and two CTAs to an SM, one of this launch and one of the next, which
//     fetches its weights while this one works.  Behind a norm that is fused into it a launch has one CTA fewer than there
//     are SMs, else one per SM, those without rows included: a launch of fewer lets the next one's double up, and every
//     later launch inherits the skew.  After its first pieces a CTA holds the others back for 800 cycles: it starts when
//     its predecessor fetches x, whose loads would queue up behind them (four projections of a layer 5 % slower when all are
//     fetched at once);
//   * two rows, longer launches, launches that wait for the one before or go over several GPUs: SIXTEEN warps and one CTA to
//     an SM.  Two warps share a position: each converts one row of two, or half the slabs, and beyond one slab only the first
//     multiplies, slabs in order, as with eight warps (with half of them for each warp 2048 x 8192 that waits took 5.3 and
//     6.9 us at one and at two rows, 5.1 and 6.3 so).  All pieces but the first are fetched behind x (16384 x 2048 at one row
//     7.0 us when all are fetched ahead, 6.3 with two first ones, 5.7 with one; none 5.9).  Beside launches that keep to
//     neither rule -- norms, activations, other products -- it is the steadier one: with eight warps a layer's four projections
//     that wait took 24.8 us, 16.9 so, and nine launches of a layer at two rows 28.8 and 22.8.
//
// Measured in chains over weights larger than L2, the kernel of gemv_tma.cuh and this one in turns, us:
//                          one row early     one that waits    two rows early    two that wait
//   2048 x 2048            2.70   2.04       3.41   2.89       2.71   2.79       3.43   3.06
//   3072 x 2048            2.96   2.38       3.75   3.30       2.93   3.07       3.80   3.64
//   16384 x 2048           6.67   5.05       7.70   5.77       7.05   5.75       7.83   6.27
//   131072 x 2048         32.1   27.6       32.2   27.8       34.5   30.2       34.9   30.5
//   32768 x 512            6.55   3.42       7.15   4.26       6.80   4.26       7.43   4.65
//   2048 x 4096            3.29   3.07       4.10   3.72       3.41   3.91       4.10   4.22
//   2048 x 8192            4.63   4.30       5.60   5.07       4.89   5.75       5.60   6.28
//   norm and 3072 x 2048   3.21   3.43       3.95   3.92       3.82   4.08       4.11   4.61
//   a layer's four        16.8   13.4       20.4   16.9       17.4   17.3       20.6   19.1
//   with neighbours, six  21.5   19.0       25.0   21.4       23.7   22.3       25.8   24.4
//   nine launches         22.0   19.5       27.3   24.4       23.2   22.8       27.6   26.8
// Two rows that start early are behind up to some 4000 outputs, and all beyond one slab: converting a row takes 2.2 times the
// instructions of fp16's and is most of the time there.  They run here all the same: a row has the same bits alone and beside
// another, and one row gains.  (Digits from two additions of a power of two, which leave out the conversion instructions, are
// the same and 0.05 to 0.2 us slower: what counts is the number of instructions.)
#pragma once
#include "gemv_tma.cuh"

namespace miori_b200 {
namespace gemvdigits {

using gemvtma::Fuse;
using gemvtma::lds128;
using gemvtma::lds_words;

constexpr int MAX_STAGES = 8;
constexpr uint32_t GROUP = 64;
constexpr uint32_t SLAB = 1024, PIECE = 128, PIECE_BYTES = 16 * PIECE;  // bytes of a row; 16 rows
constexpr uint32_t PK = 2 * PIECE;          // codes of a row in a piece
constexpr uint32_t NG = PK / GROUP;         // its scale groups
constexpr uint32_t XPAD = 64;               // between digit planes: their 64-byte reads fall into different banks
constexpr uint32_t MAX_K = 8192;
constexpr int HEAD_SHARING = 2, HEAD_ALONE = 1;  // pieces of a warp fetched at once; the others after HOLD_CYCLES, or behind x
constexpr long long HOLD_CYCLES = 800, LINGER_CYCLES = 3500;

// W warps a CTA: eight, two CTAs to an SM, or sixteen, one CTA to an SM.
template <int ROWS_, int W_>
struct Shape {
    static constexpr int ROWS = ROWS_, W = W_, THREADS = 32 * W;
    static constexpr bool SHARING = W == 8;           // an SM with the launch before and after
    // Two that share fit the 228 KB of an SM, three do not (and more than 77 KB keep other kernels' CTAs from taking the
    // successor's place); the sixteen warps of the others take all registers.
    static constexpr size_t SMEM_LIMIT = (SHARING ? 112 : 200) * 1024, SMEM_FLOOR = SHARING ? 78 * 1024 : 0;
    static constexpr int GS = 2 / ROWS;               // scale groups side by side in the eight columns
    static constexpr int NU = 2 * GS;                 // MMAs of a chain = units of eight activations per lane
    static constexpr int CH = (int)NG / GS;           // chains of a piece
    static constexpr int QW = NU;                     // words of a row per chain and lane
    static constexpr uint32_t BATCH = 8 / ROWS;       // tiles of a warp between two meetings of the CTA
};

struct Args {
    const uint16_t* x;      // activations, bf16 [ROWS][K] (fp32 when normed)
    void* y;
    const uint16_t *s, *b;  // scales and biases, [N][K / 64]
    const uint8_t* q;
    gemvtma::PreNorm pre;
    gemvtma::PostNorm post;
    uint32_t N, K, M, stages, out_bf16, gated, early;  // M is ROWS
    uint32_t n_total, row0;
    size_t y_off;
    unsigned long long* best;
    PeerArgs pa;
};

__host__ __device__ inline uint32_t slabs_of(uint32_t K) { return (K / 2u + SLAB - 1u) / SLAB; }
// Warps with a ring: beyond one slab a CTA has one tile, and the second warps of the positions only convert.
template <class S>
__host__ __device__ inline uint32_t rings_of(uint32_t nslab) { return nslab > 1u ? 8u : (uint32_t)S::W; }

// Dynamic shared memory, from a 1024-byte aligned base.
struct Layout {
    uint32_t pitch, sc, x, ms, zeros, part, total;
};
constexpr uint32_t SC_ROW = 4u * NG, SC_BYTES = 16u * SC_ROW;  // scales and biases of a row of a piece, and of a piece
template <class S>
__host__ __device__ inline Layout layout(uint32_t K, uint32_t stages, uint32_t parts) {
    Layout L;
    const uint32_t nslab = slabs_of(K);
    const uint32_t rings = rings_of<S>(nslab);
    L.pitch = nslab * PK + XPAD;  // of a digit plane
    uint32_t at = rings * stages * PIECE_BYTES;
    L.sc = at;
    at += rings * stages * SC_BYTES;
    L.x = at;
    at += 8u * S::ROWS * 4u * L.pitch;  // of eight warps, or of eight pairs of them
    L.ms = at;
    at += 8u * nslab * NG * S::ROWS * 16u;
    L.zeros = at;
    at += S::W * 16u;
    L.part = at;
    at += parts * S::ROWS * 128u;  // partial sums of a tile's positions
    L.total = at + 1024u;
    return L;
}

// D += A B, 16 x 8 x 32, codes x digits.
__device__ __forceinline__ void mma_s32(int (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_s32_z(int (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {  // D = A B
    asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "r"(0));
}
__device__ __forceinline__ void cp_async8(uint32_t dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src) : "memory");
}

// Largest magnitudes of two pairs of bf16 (signs to be masked; NaN is the largest).
__device__ __forceinline__ uint32_t max_abs2(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("max.NaN.xorsign.abs.bf16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
// Rows that digits do not hold, by their largest magnitude (bf16 bits): not all finite, or all below 2^-98, where
// digits that end at 2^-122 would be too few.
__device__ __forceinline__ bool no_digits(uint32_t largest) { return largest >= 0x7F80u || (largest != 0u && largest < (29u << 7)); }

// Eight consecutive activations (bf16) -> four digit planes, the even ones times sixteen; the first lane of a
// scale group (eight neighbouring lanes) stores {r, sum of x, 256 r, sum of x}: r r undoes the scaling for the digits
// 0 and 1, (256 r)^2 for 2 and 3.  (As a square, so that neither a scale nor a sum leaves fp32's range when it
// meets half of it.)  Every lane of the warp calls.  Returns the group's largest magnitude.
__device__ __forceinline__ uint32_t stage_unit(const uint4& v, bool live, uint32_t at, uint32_t pitch, bool first, uint32_t ms_at) {
    const uint32_t mx2 = max_abs2(max_abs2(v.x, v.y), max_abs2(v.z, v.w)) & 0x7FFF7FFFu;
    uint32_t mx = max(mx2 & 0xFFFFu, mx2 >> 16);
    const float f[8] = {bf16lo(v.x), bf16hi(v.x), bf16lo(v.y), bf16hi(v.y), bf16lo(v.z), bf16hi(v.z), bf16lo(v.w), bf16hi(v.w)};
    float sum = ((f[0] + f[1]) + (f[2] + f[3])) + ((f[4] + f[5]) + (f[6] + f[7]));
#pragma unroll
    for (int o = 1; o < (int)GROUP / 8; o <<= 1) {
        mx = max(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, o));
        sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
    }
    // half of the largest's exponent field, rounded up: |x| < 2^(2 e - 126); 2^(156 - 2 e) is to stay finite
    const uint32_t e = max((mx >> 7) + 1u, 30u) >> 1;
    const float up = __uint_as_float((279u - 2u * e) << 23), up16 = 16.0f * up;  // 2^(152 - 2 e): |x up| < 2^26
    uint32_t q[8];
#pragma unroll
    for (int i = 0; i < 8; ++i)  // the bytes of (q + 0x80808080) are the digits + 128
        q[i] = ((uint32_t)__float2int_rn(f[i] * (i & 1 ? up : up16)) + 0x80808080u) ^ 0x80808080u;
    uint32_t p[2][4];  // byte l of the even (odd) ones
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const uint32_t l01 = __byte_perm(q[h], q[2 + h], 0x5140), h01 = __byte_perm(q[h], q[2 + h], 0x7362);
        const uint32_t l23 = __byte_perm(q[4 + h], q[6 + h], 0x5140), h23 = __byte_perm(q[4 + h], q[6 + h], 0x7362);
        p[h][0] = __byte_perm(l01, l23, 0x5410), p[h][1] = __byte_perm(l01, l23, 0x7632);
        p[h][2] = __byte_perm(h01, h23, 0x5410), p[h][3] = __byte_perm(h01, h23, 0x7632);
    }
    if (live) {
#pragma unroll
        for (int l = 0; l < 4; ++l)
            asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(at + (uint32_t)l * pitch), "r"(p[0][l]), "r"(p[1][l]) : "memory");
        if (first) {
            const float r = __uint_as_float((49u + e) << 23);  // 2^(e - 78)
            asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(ms_at), "f"(r), "f"(sum), "f"(r * 256.0f), "f"(sum) : "memory");
        }
    }
    return mx;
}

// The slow side of a wait on a barrier, out of the way of the code that runs.
__device__ __noinline__ bool wait_on(uint32_t bar, uint32_t parity, volatile uint32_t* abort, uint32_t where) {
    return __all_sync(0xFFFFFFFFu, mbar_wait(bar, parity, abort, where));
}

// Eight outputs of a row of activations that are not all finite, or all next to nothing, in fp32 by a whole warp: they have no
// digits.  Tensor rows row0 .. row0 + 7, or, gated, row0 .. row0 + 3 and the up rows of the same outputs.  Lane i < 8 gets
// the i-th.
template <bool NORMED>
__device__ __forceinline__ float plain_dots(const Args& A, uint32_t row0, bool gated, uint32_t m, float inv) {
    constexpr uint32_t DOTS = 8;
    const uint32_t ng = A.K / GROUP, words = A.K / 8u, lane = threadIdx.x & 31u;
    uint32_t row[DOTS];
    float sum[DOTS];
#pragma unroll
    for (uint32_t d = 0; d < DOTS; ++d) {
        row[d] = gated ? row0 + (d & 3u) + (d >= 4u ? A.N >> 1 : 0u) : min(row0 + d, A.N - 1u);
        sum[d] = 0.0f;
    }
    for (uint32_t w = lane; w < words; w += 32u) {
        const size_t at = (size_t)m * words + w;
        uint4 v;
        if constexpr (NORMED) {
            const float4* x4 = reinterpret_cast<const float4*>(A.x) + 2u * at;
            v = gemvtma::normed8(ld_fresh(x4), ld_fresh(x4 + 1), inv, __ldg(reinterpret_cast<const uint4*>(A.pre.gamma) + w));
        } else {
            v = ld_fresh(reinterpret_cast<const uint4*>(A.x) + at);
        }
        const float x[8] = {bf16lo(v.x), bf16hi(v.x), bf16lo(v.y), bf16hi(v.y), bf16lo(v.z), bf16hi(v.z), bf16lo(v.w), bf16hi(v.w)};
        const float sx = ((x[0] + x[1]) + (x[2] + x[3])) + ((x[4] + x[5]) + (x[6] + x[7]));
        uint32_t codes[DOTS], s[DOTS], b[DOTS];
#pragma unroll
        for (uint32_t d = 0; d < DOTS; ++d) {
            const size_t g = (size_t)row[d] * ng + w / (GROUP / 8u);
            codes[d] = reinterpret_cast<const uint32_t*>(A.q)[(size_t)row[d] * words + w], s[d] = A.s[g], b[d] = A.b[g];
        }
#pragma unroll
        for (uint32_t d = 0; d < DOTS; ++d) {
            float cx = 0.0f;
#pragma unroll
            for (int i = 0; i < 8; ++i) cx = __fmaf_rn((float)((codes[d] >> (4 * i)) & 15u), x[i], cx);
            sum[d] = __fmaf_rn(bf16_bits_to_float(s[d]), cx, __fmaf_rn(bf16_bits_to_float(b[d]), sx, sum[d]));
        }
    }
    float y = 0.0f;
#pragma unroll
    for (uint32_t d = 0; d < DOTS; ++d) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum[d] += __shfl_xor_sync(0xFFFFFFFFu, sum[d], o);
        if (lane == d) y = sum[d];
    }
    return y;
}

// All outputs of the CTA's tiles in the rows of `wanting`, half a tile a warp.  Returns the arg-max form's best key.  (One
// launch after the other with such a row, a thread an output and so, us: 2048 x 2048 35 -> 9, 16384 x 2048 47 -> 18, 2048 x
// 8192 119 -> 28.)
template <int ROWS, Fuse F>
__device__ __noinline__ unsigned long long plain_rows(const Args& A, uint32_t wanting, uint32_t inv_at, unsigned long long my_best) {
    const bool gated = F == gemvtma::FUSED && A.gated != 0u, normed = F == gemvtma::FUSED && A.pre.gamma != nullptr;
    const uint32_t my_tiles = (((A.N + 15u) >> 4) - blockIdx.x + gridDim.x - 1u) / gridDim.x;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
#pragma unroll 1
    for (uint32_t m = 0; m < (uint32_t)ROWS; ++m) {
        if (!(wanting >> m & 1u)) continue;
        float inv = 0.0f;
        if (normed) asm volatile("ld.shared.f32 %0, [%1];" : "=f"(inv) : "r"(inv_at + 4u * m));
#pragma unroll 1
        for (uint32_t i = warp; i < 2u * my_tiles; i += warps) {
            const uint32_t tile = blockIdx.x + (i >> 1) * gridDim.x, row0 = gated ? tile * 8u + (i & 1u) * 4u : tile * 16u + (i & 1u) * 8u;
            const float y = normed ? plain_dots<true>(A, row0, gated, m, inv) : plain_dots<false>(A, row0, gated, m, 0.0f);
            if (gated) {
                const float up = __shfl_down_sync(0xFFFFFFFFu, y, 4);
                if (lane < 4u) gemvtma::store_gated(A, m, row0 + lane, y, up);
            } else if (lane < 8u && row0 + lane < A.N) {
                gemvtma::store_out<F>(A, m, row0 + lane, y, my_best);
            }
        }
    }
    return my_best;
}

// RES: K <= 2048, one slab: the activations of a warp's position stay in registers.
template <class S, Fuse F, bool RES>
__global__ void __launch_bounds__(S::THREADS, S::SHARING ? 2 : 1)
gemv_digits_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ Args A) {
    constexpr int ROWS = S::ROWS, CH = S::CH, NU = S::NU, GS = S::GS;
    constexpr uint32_t WARPS = S::W;
    constexpr bool PAIRED = WARPS == 16u;  // two warps share a position's activations: each converts one row of two, or half the slabs
    static_assert(PAIRED || ROWS == 1, "a warp converts one row");
    constexpr bool SHARDED_ = F == gemvtma::SHARDED, ARGMAX_ = F == gemvtma::ARGMAX, POSTNORM_ = F == gemvtma::POSTNORM;
    const bool gated = F == gemvtma::FUSED && A.gated != 0u, normed = F == gemvtma::FUSED && RES && A.pre.gamma != nullptr;
    const uint32_t N = A.N, K = A.K, stages = A.stages;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t tiles = (N + 15u) >> 4, row_bytes = K / 2u, ng = K / GROUP;
    const uint32_t full_slabs = row_bytes / SLAB, rest = row_bytes % SLAB, nslab = slabs_of(K);
    // short rows have fewer positions, and the warps of a position share the tiles
    const uint32_t P = full_slabs ? 8u : (rest + PIECE - 1u) / PIECE;
    const uint32_t pshift = P > 4u ? 3u : P > 2u ? 2u : P - 1u, TG = WARPS >> pshift;
    const uint32_t pos = warp & ((1u << pshift) - 1u), tg = warp >> pshift;
    const uint32_t slabs = full_slabs + (pos * PIECE < rest ? 1u : 0u);

    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t bars[WARPS * MAX_STAGES];
    __shared__ volatile uint32_t abort_flag;
    __shared__ uint32_t largest[WARPS][ROWS];  // magnitudes, in what each warp has seen of a row

    const bool early = S::SHARING || A.early != 0u;
    const long long born = clock64();
    if (early) pdl_launch_dependents();

    const uint32_t my_tiles = (tiles - blockIdx.x + gridDim.x - 1u) / gridDim.x;
    const uint32_t batch = TG * S::BATCH;
    const uint32_t wt = my_tiles > tg ? (my_tiles - tg + TG - 1u) / TG : 0u;  // tiles of this warp
    const uint32_t pieces = wt * slabs;
    const Layout L = layout<S>(K, stages, (my_tiles > batch ? 2u * batch : my_tiles) << pshift);
    const uint32_t base = (smem_addr(smem_raw) + 1023u) & ~1023u;
    const uint32_t ring = base + warp * stages * PIECE_BYTES, bar0 = smem_addr(&bars[warp * MAX_STAGES]);
    const uint32_t sc_ring = base + L.sc + warp * stages * SC_BYTES;
    auto tile_of = [&](uint32_t j) { return blockIdx.x + j * gridDim.x; };

    // ---- fetching: tile after tile, slab after slab.  gated: a tile is eight gate rows and the up rows of the same outputs
    auto row_of = [&](uint32_t tile, uint32_t r) {
        return gated ? tile * 8u + (r & 7u) + (r >= 8u ? N >> 1 : 0u) : min(tile * 16u + r, N - 1u);
    };
    const uint32_t ic_first = pos * (PIECE / 8u), ic_end = ic_first + slabs * (SLAB / 8u), ie_first = pos * NG;
    uint32_t issued = 0, itile = tile_of(tg), ic0 = ic_first;
    const uint16_t* const sc_src = lane < 16u ? A.s : A.b;
    size_t ie = (size_t)row_of(itile, lane & 15u) * ng + ie_first;
    const uint32_t sc_dst = sc_ring + (lane & 15u) * SC_ROW + (lane >> 4) * (SC_ROW / 2u);
    auto issue = [&](uint32_t st) {
        const uint32_t bar = bar0 + st * 8u;
        if (lane == 0) {
            const uint32_t dst = ring + st * PIECE_BYTES;
            if (issued >= stages) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // behind the reads of what lay there
            mbar_expect_tx(bar, PIECE_BYTES);
            if (gated) {  // the tensor map's boxes are eight rows high
                tma_load_2d(dst, &tmap_q, (int)ic0, (int)(itile * 8u), bar);
                tma_load_2d(dst + 8u * PIECE, &tmap_q, (int)ic0, (int)((N >> 1) + itile * 8u), bar);
            } else {
                tma_load_2d(dst, &tmap_q, (int)ic0, (int)(itile * 16u), bar);
            }
        }
        cp_async8(sc_dst + st * SC_BYTES, sc_src + ie);
        asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
        ++issued;
        ic0 += SLAB / 8u, ie += 8u * NG;
        if (RES || ic0 == ic_end) {
            ic0 = ic_first;
            itile += TG * gridDim.x;
            ie = (size_t)row_of(itile, lane & 15u) * ng + ie_first;
        }
    };
    if (lane == 0) {
        abort_flag = 0u;
        for (uint32_t i = 0; i < stages; ++i) mbar_init(bar0 + 8u * i, 33);  // the copy's issuer and every lane's scales
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("st.shared.v4.u32 [%0], {%1,%1,%1,%1};" ::"r"(base + L.zeros + 16u * warp), "r"(0u) : "memory");
    }
    __syncwarp();
    // A launch that may not start early waits here, and lets its dependents start only when its predecessor is
    // complete: they prefetch what that may have written.
    if (!early) {
        pdl_wait_prior();
        pdl_launch_dependents();
    }
    const uint32_t ahead = min(stages, pieces);
    auto fill = [&](uint32_t n) {
#pragma unroll 1  // one copy of the code: three copies of it cost a layer with its norms 0.5 to 1.6 us
        while (issued < n) {
            if (S::SHARING && issued == (uint32_t)HEAD_SHARING) {
                const long long t0 = clock64();
                while (clock64() - t0 < HOLD_CYCLES) __nanosleep(40);
            }
            issue(issued);
        }
    };
    fill(S::SHARING ? ahead : min(ahead, (uint32_t)HEAD_ALONE));

    // ---- this lane's place in the MMAs: tile rows prow and prow + 8 (in an order that spreads the swizzled rows which
    // a quarter- or half-warp reads over all banks); as a B operand column lane / 4 = (slot or row, digit)
    const uint32_t g = lane >> 2, t = lane & 3u;
    const uint32_t prow = ROWS == 1 ? ((g & 1u) << 2) | (g >> 1) : ((g & 3u) << 1) | (g >> 2);
    const uint32_t region = PAIRED ? ((tg >> 1) << pshift) + pos : warp;
    const uint32_t xw = base + L.x + region * ROWS * 4u * L.pitch, msw = base + L.ms + region * nslab * (NG * ROWS * 16u);
    const bool mine = ROWS > 1 || (g >> 2) == (t >> 1);  // one row: the codes of this lane belong to its column's group
    const uint32_t xb = mine ? xw + ((ROWS == 1 ? 0u : g >> 2) * 4u + (g & 3u)) * L.pitch + t * (uint32_t)(NU * 8)
                             : base + L.zeros + 16u * warp;
    const uint32_t xstep = mine ? 1u : 0u;
    const uint32_t ms0 = msw + (t >> 1) * 16u + (t & 1u) * 8u;  // one row: of group t / 2; two: of row t / 2
    const uint32_t sel = ROWS == 1 && t >= 2u ? 0x3244u : 0x1044u;
    const uint32_t q_lane = ring + prow * PIECE, s_lane = sc_ring + prow * SC_ROW;
    const uint32_t q_at0 = (t * (uint32_t)(4 * S::QW)) ^ (prow << 4);

    bool ok = true;  // turns false for good once a wait expires; the warp then goes on without waiting, to meet the others
    // a look at a barrier costs 100 cycles: it is made ahead of the work that hides them, and used behind it
    auto test_stage = [&](uint32_t st, uint32_t parity) { return mbar_test(bar0 + st * 8u, parity); };
    auto settle = [&](bool there, uint32_t st, uint32_t parity) {
        if (!__all_sync(0xFFFFFFFFu, there) && ok) ok = wait_on(bar0 + st * 8u, parity, &abort_flag, 0x10);
    };
    struct Codes { uint32_t a[CH * NU][4]; };
    struct Packed { uint32_t q0[CH * NU], q1[CH * NU]; };
    auto load_q = [&](uint32_t stage, Packed& p) {
        const uint32_t qa = q_lane + stage * PIECE_BYTES;
#pragma unroll
        for (int c = 0; c < CH; ++c) {
            uint32_t v0[NU], v1[NU];
            const uint32_t at = qa + (q_at0 ^ (uint32_t)(c * 16 * S::QW));
            lds_words<4 * NU>(v0, at);
            lds_words<4 * NU>(v1, at + 8u * PIECE);
#pragma unroll
            for (int i = 0; i < NU; ++i) p.q0[c * NU + i] = v0[i], p.q1[c * NU + i] = v1[i];
        }
    };
    auto unpack = [&](const Packed& p, Codes& o) {
#pragma unroll
        for (int i = 0; i < CH * NU; ++i) {
            o.a[i][0] = p.q0[i] & 0x0F0F0F0Fu, o.a[i][1] = p.q1[i] & 0x0F0F0F0Fu;
            o.a[i][2] = p.q0[i] & 0xF0F0F0F0u, o.a[i][3] = p.q1[i] & 0xF0F0F0F0u;
        }
    };
    constexpr int SW = (int)NG / 2;
    struct Scales { uint32_t s0[SW], b0[SW], s1[SW], b1[SW]; };
    auto load_s = [&](uint32_t stage, Scales& v) {
        uint32_t r0[2 * SW], r1[2 * SW];
        lds_words<8 * SW>(r0, s_lane + stage * SC_BYTES);
        lds_words<8 * SW>(r1, s_lane + stage * SC_BYTES + 8u * SC_ROW);
#pragma unroll
        for (int i = 0; i < SW; ++i) v.s0[i] = r0[i], v.b0[i] = r0[SW + i], v.s1[i] = r1[i], v.b1[i] = r1[SW + i];
    };
    struct Acts { uint32_t b[CH * NU][2]; float r[CH], sum[CH]; };
    auto load_x = [&](uint32_t slab, Acts& a) {
#pragma unroll
        for (int c = 0; c < CH; ++c) {
            const uint32_t at = xb + xstep * (slab * PK + (uint32_t)c * (GS * GROUP));
#pragma unroll
            for (int i = 0; i < NU; i += 2) {
                const uint4 v = lds128(at + xstep * 8u * i);
                a.b[c * NU + i][0] = v.x, a.b[c * NU + i][1] = v.y, a.b[c * NU + i + 1][0] = v.z, a.b[c * NU + i + 1][1] = v.w;
            }
            asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(a.r[c]), "=f"(a.sum[c])
                         : "r"(ms0 + (slab * NG + (uint32_t)(c * GS)) * (ROWS * 16u)));
        }
    };
    struct Sums { int d[CH][4]; };
    auto multiply = [&](const Codes& q, const Acts& x, Sums& o) {
#pragma unroll
        for (int i = 0; i < NU; ++i)
#pragma unroll
            for (int c = 0; c < CH; ++c) {
                if (i == 0) mma_s32_z(o.d[c], q.a[c * NU], x.b[c * NU][0], x.b[c * NU][1]);
                else mma_s32(o.d[c], q.a[c * NU + i], x.b[c * NU + i][0], x.b[c * NU + i][1]);
            }
    };
    // sums of tile rows prow and prow + 8: of two digits, and with one row of every other group; with two rows even and
    // odd groups apart, so that a row's sums meet in the same order
    constexpr int PAR = ROWS;
    float acc[PAR][2];
    auto apply = [&](const Sums& o, const Scales& sc, const Acts& x) {
#pragma unroll
        for (int c = 0; c < CH; ++c) {
            auto pick = [&](const uint32_t (&w)[SW]) {
                if constexpr (GS == 2) return __uint_as_float(__byte_perm(w[c], 0u, sel));
                else return c & 1 ? bf16hi(w[c >> 1]) : bf16lo(w[c >> 1]);
            };
            const float r = x.r[c];
            const float v0 = (float)(o.d[c][1] * 256 + o.d[c][0]) * r, v1 = (float)(o.d[c][3] * 256 + o.d[c][2]) * r;
            float (&a)[2] = acc[c & (PAR - 1)];
            // the bias term goes with the high digits, where it cancels most of them, and what its rounding leaves with the
            // low ones (error against 64-bit sums at 2048 x 2048 0.68e-7 of the result, 0.89e-7 without the latter, 1.4e-7 with the
            // term among the low ones; fp16 operands: 0.74e-7, 11e-7 with outliers among the activations against 0.9e-7 here)
            auto bias = [&](float b) {
                const float p = b * x.sum[c];
                return t & 1u ? p : __fmaf_rn(b, x.sum[c], -p);
            };
            a[0] += __fmaf_rn(pick(sc.s0) * r, v0, bias(pick(sc.b0)));
            a[1] += __fmaf_rn(pick(sc.s1) * r, v1, bias(pick(sc.b1)));
        }
    };

    // the next piece: its codes and scales into registers, and its stage to the copies
    uint32_t st = 0, par = 0;
    Packed q;
    Scales sc;
    auto take = [&](bool there) {
        settle(there, st, par);
        load_q(st, q);
        load_s(st, sc);
        __syncwarp();
        if (issued != pieces) issue(st);
    };
    auto first_piece = [&] {  // once the loads of x are on their way
        if (!S::SHARING) fill(ahead);
        if (pieces) take(test_stage(0u, 0u));
    };

    // warps that share a position have pieces if the first of them has
    const uint32_t work = !PAIRED ? pieces : my_tiles > (tg & ~1u) ? slabs : 0u;
    uint4 gm = make_uint4(0u, 0u, 0u, 0u);  // norm weights of this lane's activations
    if (normed && work && (pos * 32u + lane) * 8u < K) gm = __ldg(reinterpret_cast<const uint4*>(A.pre.gamma) + pos * 32u + lane);
    pdl_wait_prior();  // x (and y) belong to the predecessor until here

    // A CTA without rows keeps its place until the next launch has taken its own: at the head of a chain it would be gone
    // first, and leave its SM to two of the next launch's
    if (S::SHARING && my_tiles == 0u)
        while (clock64() - born < LINGER_CYCLES) __nanosleep(100);

    // ---- the activations of this warp's position: one unit of every row and slab a lane
    __shared__ float nm_part[ROWS][WARPS], nm_inv[ROWS];
    const uint32_t cr = ROWS > 1 ? tg & 1u : 0u;             // the row that this warp converts, and its slabs c0 .. c0 + sets - 1
    const uint32_t below = PAIRED && ROWS == 1 ? (slabs + 1u) >> 1 : slabs;
    const uint32_t c0 = PAIRED && ROWS == 1 && (tg & 1u) ? below : 0u, sets = c0 ? slabs - below : below;
    uint32_t top = 0u;
    if (my_tiles && (work || normed)) {
        const uint32_t upr = K >> 3;
        // normed (one slab): the squares first (every unit once: of the first warps of a position), warps in order
        float4 xa4, xc4;
        float inv = 0.0f;
        if (normed) {
            const float4* x4 = reinterpret_cast<const float4*>(A.x);
            const uint32_t u = pos * 32u + lane;
            xa4 = xc4 = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (sets && u < upr) xa4 = ld_fresh(x4 + (cr * upr + u) * 2u), xc4 = ld_fresh(x4 + (cr * upr + u) * 2u + 1u);
            first_piece();
            float ss = 0.0f;
            ss = __fmaf_rn(xa4.x, xa4.x, ss), ss = __fmaf_rn(xa4.y, xa4.y, ss), ss = __fmaf_rn(xa4.z, xa4.z, ss), ss = __fmaf_rn(xa4.w, xa4.w, ss);
            ss = __fmaf_rn(xc4.x, xc4.x, ss), ss = __fmaf_rn(xc4.y, xc4.y, ss), ss = __fmaf_rn(xc4.z, xc4.z, ss), ss = __fmaf_rn(xc4.w, xc4.w, ss);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xFFFFFFFFu, ss, o);
            if (lane == 0) {
#pragma unroll
                for (uint32_t m = 0; m < (uint32_t)ROWS; ++m) nm_part[m][warp] = m == cr && tg == cr ? ss : 0.0f;
            }
            __syncthreads();
#pragma unroll
            for (uint32_t m = 0; m < (uint32_t)ROWS; ++m) {
                float tot = 0.0f;
#pragma unroll
                for (uint32_t w = 0; w < WARPS; ++w) tot += nm_part[m][w];
                const float in = rsqrtf(tot / (float)K + A.pre.eps);
                if (m == cr) inv = in;
                if (threadIdx.x == 0) nm_inv[m] = in;
            }
        }
        auto load = [&](uint32_t r) {
            const uint32_t u = ((c0 + r) * 8u + pos) * 32u + lane;
            uint4 v = make_uint4(0u, 0u, 0u, 0u);
            if (r < sets && u < upr) {
                if (normed) v = gemvtma::normed8(xa4, xc4, inv, gm);
                else v = ld_fresh(reinterpret_cast<const uint4*>(A.x) + (size_t)cr * upr + u);
            }
            return v;
        };
        auto stage = [&](uint32_t r, const uint4& v) {
            return stage_unit(v, r < sets, xw + cr * 4u * L.pitch + (c0 + r) * PK + lane * 8u, L.pitch, (lane & 7u) == 0u,
                              msw + (((c0 + r) * NG + (lane >> 3)) * ROWS + cr) * 16u);
        };
        if constexpr (RES) {
            const uint4 v = load(0u);
            if (!normed) first_piece();
            if (sets) top = stage(0u, v);
        } else {  // AHEAD loads in flight (all of them), PAIR units at a time (more would be straight code, which costs its fetches)
            constexpr int AHEAD = 4, PAIR = 2;
            static_assert(MAX_K <= AHEAD * 2u * SLAB, "a slab of the row for each");
            uint4 v[AHEAD];
#pragma unroll
            for (int h = 0; h < AHEAD; ++h) v[h] = load((uint32_t)h);
            first_piece();
#pragma unroll 1
            for (uint32_t r = 0; r < sets; r += PAIR) {
                top = max(top, max(stage(r, v[0]), stage(r + 1u, v[1])));
#pragma unroll
                for (int h = 0; h + PAIR < AHEAD; ++h) v[h] = v[h + PAIR];
            }
        }
    }
    top = __reduce_max_sync(0xFFFFFFFFu, top);
    if (lane == 0) {
#pragma unroll
        for (uint32_t m = 0; m < (uint32_t)ROWS; ++m) largest[warp][m] = m == cr ? top : 0u;
    }
    if constexpr (PAIRED) {
        if (work) asm volatile("bar.sync %0, 64;" ::"r"(region + 1u) : "memory");
    }
    __syncwarp();
    Acts xa;
    if constexpr (RES) {
        if (pieces) load_x(0u, xa);
    }

    // y is one launch's output; ARGMAX: key of the best element this thread has stored
    unsigned long long my_best = 0ull;
    auto store_out = [&](uint32_t m, uint32_t row, float v) { gemvtma::store_out<F>(A, m, row, v, my_best); };
    uint32_t j = tg, left = pieces, wanting = 0u;  // wanting: rows without digits
    for (uint32_t j0 = 0; j0 < my_tiles; j0 += batch) {
        const uint32_t jend = min(my_tiles, j0 + batch), buf = (j0 / batch) & 1u ? batch : 0u;  // two buffers: one meeting a batch
        uint32_t at = base + L.part + (((buf + j - j0) << pshift) + pos) * (ROWS * 128u) + lane * (ROWS * 4u);
#pragma unroll 1
        for (; j < jend && slabs; j += TG, at += WARPS * (ROWS * 128u)) {
#pragma unroll
            for (int p = 0; p < PAR; ++p) acc[p][0] = acc[p][1] = 0.0f;
#pragma unroll 1
            for (uint32_t s = 0; s < (RES ? 1u : slabs); ++s) {
                if constexpr (!RES) load_x(s, xa);
                Codes cur;
                Sums sums;
                if (++st == stages) st = 0u, par ^= 1u;
                const bool there = test_stage(st, par);
                unpack(q, cur);
                multiply(cur, xa, sums);
                const Scales now = sc;
                if (--left) take(there);
                apply(sums, now, xa);
            }
            // the digits' sums; lanes of even t go on with row prow, the others with row prow + 8
            auto meet = [&](const float (&a)[2]) { return (t & 1u ? a[1] : a[0]) + __shfl_xor_sync(0xFFFFFFFFu, t & 1u ? a[0] : a[1], 1); };
#pragma unroll
            for (int p = 0; p < PAR; ++p) {
                const float v = meet(acc[p]);
                asm volatile("st.shared.f32 [%0], %1;" ::"r"(at + (uint32_t)p * 4u), "f"(v) : "memory");
            }
        }
        __syncthreads();
        uint32_t tallest = 0u;  // of this lane's row
#pragma unroll
        for (uint32_t w = 0; w < WARPS; ++w) tallest = max(tallest, largest[w][ROWS == 1 ? 0u : t >> 1]);
        const bool none = no_digits(tallest);
        wanting = ROWS == 1 ? (none ? 1u : 0u) : (__any_sync(0xFFFFFFFFu, none && t < 2u) ? 1u : 0u) | (__any_sync(0xFFFFFFFFu, none && t >= 2u) ? 2u : 0u);
        for (uint32_t jj = j0 + warp; jj < jend; jj += WARPS) {  // a tile a warp: positions in a fixed tree, even and odd groups last
            const uint32_t from = base + L.part + ((buf + jj - j0) << pshift) * (ROWS * 128u) + lane * (ROWS * 4u);
            float v[PAR];
#pragma unroll
            for (int p = 0; p < PAR; ++p) {
                float h[8];
#pragma unroll
                for (uint32_t i = 0; i < 8u; ++i) {
                    h[i] = 0.0f;
                    if (i < P) asm volatile("ld.shared.f32 %0, [%1];" : "=f"(h[i]) : "r"(from + i * (ROWS * 128u) + (uint32_t)p * 4u));
                }
                v[p] = ((h[0] + h[1]) + (h[2] + h[3])) + ((h[4] + h[5]) + (h[6] + h[7]));
            }
            float y = ROWS == 1 ? v[0] + __shfl_xor_sync(0xFFFFFFFFu, v[0], 2) : v[0] + v[PAR - 1];
            const uint32_t m = ROWS == 1 ? 0u : t >> 1, r = prow + 8u * (t & 1u), tile = tile_of(jj);
            const bool live = !none && (ROWS > 1 || t < 2u) && (gated || tile * 16u + r < N);
            if (gated) {  // even t: gate of output prow, odd t: its up
                __syncwarp();
                const float up = __shfl_xor_sync(0xFFFFFFFFu, y, 1);
                if (live && ok && (t & 1u) == 0u) gemvtma::store_gated(A, m, tile * 8u + prow, y, up);
            } else if (live && ok) {
                store_out(m, tile * 16u + r, y);
            }
        }
    }

    // rows without digits: here, where nothing of the above is wanted any more (among the stores it would be spilled)
    if (__builtin_expect(wanting != 0u, 0)) my_best = plain_rows<ROWS, F>(A, wanting, smem_addr(nm_inv), my_best);

    if constexpr (POSTNORM_ || ARGMAX_ || SHARDED_) __syncthreads();
    if (abort_flag) {  // let copies still in flight land before the CTA's memory is released
        const long long t0 = clock64();
        while (clock64() - t0 < 2000000LL) __nanosleep(1000);
    }
    gemvtma::close_launch<F, (int)WARPS, (int)WARPS>(A, my_best);
}

// Launch plan: stages of a warp's ring (0: does not fit) and shared memory.
struct Plan {
    uint32_t grid, stages;
    size_t smem;
};
template <class S>
Plan plan_launch(uint32_t N, uint32_t K, bool normed) {
    Plan p;
    const uint32_t tiles = (N + 15u) / 16u;
    // Sharing its SMs: one CTA per SM, but for the SM that the norm kernel before a normed projection is on: its CTAs take
    // the room of one of ours there, and ours would join another SM's (a layer with its two norms at one row 21.7 us so, 18.3
    // with one CTA fewer; a chain of plain projections needs them all).
    p.grid = S::SHARING ? std::max(1u, (uint32_t)sm_count() - (normed ? 1u : 0u)) : std::min((uint32_t)sm_count(), tiles);
    const uint32_t tc = (tiles + p.grid - 1u) / p.grid, row_bytes = K / 2u, nslab = slabs_of(K);
    const uint32_t P = row_bytes >= SLAB ? 8u : (row_bytes + PIECE - 1u) / PIECE, pshift = P > 4u ? 3u : P > 2u ? 2u : P > 1u ? 1u : 0u;
    const uint32_t TG = (uint32_t)S::W >> pshift, batch = TG * S::BATCH, part = (tc > batch ? 2u * batch : tc) << pshift;
    if (nslab > 1u && tc > 1u) {  // takes() has none (see rings_of)
        p.stages = 0u;
        return p;
    }
    for (p.stages = std::min<uint32_t>(MAX_STAGES, (tc + TG - 1u) / TG * nslab); p.stages > 0u; --p.stages) {
        p.smem = layout<S>(K, p.stages, part).total;
        if (p.smem <= S::SMEM_LIMIT) break;
    }
    p.smem = std::max(p.smem, S::SMEM_FLOOR);
    return p;
}

template <class S, Fuse F, bool RES>
int launch_one(const void* q, Args a, cudaStream_t stream) {
    const Plan p = plan_launch<S>(a.N, a.K, a.pre.gamma != nullptr);
    if (!p.stages) return fail(MIORI_E_INVALID, "gemv: no plan for N=%u K=%u M=%u", a.N, a.K, a.M);
    a.stages = p.stages;
    CUtensorMap tq;
    const int rc = make_tmap_2d(&tq, q, CU_TENSOR_MAP_DATA_TYPE_UINT64, 8, (uint64_t)a.K / 16, a.N, PIECE / 8, a.gated ? 8 : 16,
                                CU_TENSOR_MAP_SWIZZLE_128B);
    if (rc) return rc;
    const cudaError_t e = launch<Split::SHARED>(gemv_digits_kernel<S, F, RES>, dim3(p.grid), dim3(S::THREADS), p.smem, stream, true, tq, a);
    if (e != cudaSuccess) return cuda_fail(e, "gemv_digits launch");
    return MIORI_OK;
}

template <class S, Fuse F>
int launch_k(const void* q, const Args& a, cudaStream_t stream) {
    return a.K / 2u <= SLAB ? launch_one<S, F, true>(q, a, stream) : launch_one<S, F, false>(q, a, stream);
}

// K that this kernel takes: whole pieces (a row of 6208 codes, with its last groups picked out one by one, took 11.3 us at
// 5967 rows, 7.6 in gemv_tma.cuh), up to where its launches still pay.
// Beyond one slab as long as there is one tile a CTA: what a layer's last projection is, which the others of a chain of
// early launches start beside (with this product in gemv_tma.cuh the four projections of a layer take 15.9 us at one row, 13.5
// with it here); with more, the conversion of x and the pieces take longer than there (8192 x 8192 at one row 11.5 us,
// 10.1).  So there the kernel, and with it a row's rounding, depends on N, as the order of its sums in gemv_tma.cuh does.
// Never with the norm in front: the squares are a trip to L2 of their own there (norm and 2048 x 4096 at one row and at two
// 5.2 and 6.1 us, 3.7 and 4.5 there; 2048 x 8192 8.0 and 9.2, 6.5 and 7.8).
inline bool takes(uint32_t N, uint32_t K, bool normed) {
    return K % PK == 0u && (K <= 2u * SLAB || (!normed && K <= MAX_K && (N + 15u) / 16u <= (uint32_t)sm_count()));
}

// Whether one row started early leaves half of its SMs to the next launch.  Beside a long stream that half is worth less than
// eight more warps.  Early launches with eight and with sixteen warps, us, in chains of their own, and each with one of 2048 outputs
// behind it, which has eight:
//   24576 x 2048 (170 KiB of codes an SM) 7.5 and 7.2, 9.5 and 10.3    28672 x 2048 (194) 8.5 and 7.5, 10.4 and 10.5
//   32768 x 2048 (226) 9.3 and 8.6, 11.2 and 10.9                      131072 x 2048 (908) 35.2 and 27.6, 36.8 and 29.7
//   49152 x 1024 (170) 7.5 and 7.0, 9.2 and 9.4                        65536 x 1024 (226) 9.4 and 8.3, 11.0 and 10.5
//   65536 x 512 (113) 5.3 and 5.4, 7.0 and 7.8                         131072 x 512 (226) 9.7 and 8.6, 11.4 and 10.7
constexpr uint32_t SHARING_CODES = 192 * 1024;
inline bool shares(uint32_t N, uint32_t K) { return (uint64_t)N * (K / 2u) <= (uint64_t)sm_count() * SHARING_CODES; }

// One or two rows, of a K that is taken.
template <class S>
int launch_form(const void* q, const Args& a, cudaStream_t stream) {
    if (a.best) {
        if constexpr (S::ROWS == 1) return launch_k<S, gemvtma::ARGMAX>(q, a, stream);
    }
    if (a.pa.world > 1) {
        if constexpr (!S::SHARING) return launch_k<S, gemvtma::SHARDED>(q, a, stream);
    }
    if (a.post.residual) return launch_k<S, gemvtma::POSTNORM>(q, a, stream);
    if (a.gated || a.pre.gamma) return launch_k<S, gemvtma::FUSED>(q, a, stream);
    return launch_k<S, gemvtma::NONE>(q, a, stream);
}
inline int launch_rows(const void* q, const void* s, const void* b, const void* x, void* y, uint32_t N, uint32_t K, uint32_t M, uint32_t flags,
                       cudaStream_t stream, const gemvtma::Shard& sh) {
    const bool placed = sh.pa.world > 1 || sh.best;  // y is a slice of an n_total-row output
    Args a;
    a.x = static_cast<const uint16_t*>(x), a.y = y;
    a.q = static_cast<const uint8_t*>(q), a.s = static_cast<const uint16_t*>(s), a.b = static_cast<const uint16_t*>(b);
    a.pre = sh.pre, a.post = sh.post;
    a.N = N, a.K = K, a.M = M, a.stages = 0u;
    a.out_bf16 = flags & MIORI_OUT_BF16 ? 1u : 0u, a.gated = sh.gated ? 1u : 0u, a.early = flags & MIORI_LAUNCH_PDL ? 1u : 0u;
    a.n_total = placed ? sh.n_total : N, a.row0 = placed ? sh.row0 : 0u, a.y_off = sh.y_off, a.best = sh.best, a.pa = sh.pa;
    const int rc = gemvtma::check_fuse(sh, 4, N, M, a.out_bf16 != 0u);
    if (rc) return rc;
    if (M == 2u) return launch_form<Shape<2, 16>>(q, a, stream);
    return a.early && sh.pa.world <= 1 && shares(N, K) ? launch_form<Shape<1, 8>>(q, a, stream) : launch_form<Shape<1, 16>>(q, a, stream);
}

}  // namespace gemvdigits
}  // namespace miori_b200
