// The decode GEMV's launches: which kernel takes a batch, and batches that need several.
#pragma once
#include "gemv_digits.cuh"
#include "gemv_tma.cuh"

namespace miori_b200 {
namespace gemvtma {

// ---- batches
//
// A row's bits must not depend on how many rows are in flight beside it, so everything that decides the order of
// its sums -- the shape and how many groups share a tile -- is chosen by a class of batch sizes and not by M:
// the class's largest batch has to fit, and where it does not, every batch of the class is dealt to launches of
// the next smaller class.  Classes: 1..4 rows (4-bit weights in groups of 64: 1..2, see below), up to 8, 16, 32.
template <int BITS, int GROUP>
struct Batch {
    // Three and four rows of 4-bit weights at group 64 gain nothing from slots (two, one step a pass): 16384 x
    // 2048 takes 8.0 us with them and 7.2 without; they run as eight do.
    static constexpr bool WIDE3 = BITS == 4 && GROUP == 64;
    static constexpr uint32_t class_of(uint32_t M) { return M <= 2u ? (WIDE3 ? 2u : 4u) : M <= 4u ? (WIDE3 ? 8u : 4u) : M <= 8u ? 8u : M <= 16u ? 16u : 32u; }
    static uint32_t kpar_of(uint32_t cls, uint32_t N, uint32_t K) {
        switch (cls) {
        case 1: return choose_kpar<Shape<BITS, GROUP, 1>>(N, K, 1);
        case 2: return choose_kpar<Shape<BITS, GROUP, 2>>(N, K, 2);
        case 4: return choose_kpar<Shape<BITS, GROUP, WIDE3 ? 8 : 4>>(N, K, 4);
        case 8: return choose_kpar<Shape<BITS, GROUP, 8>>(N, K, 8);
        case 16: return choose_kpar<Shape<BITS, GROUP, 16>>(N, K, 16);
        default: return choose_kpar<Shape<BITS, GROUP, 32>>(N, K, 32);
        }
    }
    // One launch of up to cls rows.  Below eight the shapes of fewer rows sum in the same order.
    static int launch(uint32_t cls, uint32_t kpar, const void* q, const void* s, const void* b, const void* x, void* y, uint32_t N,
                      uint32_t K, uint32_t M, uint32_t flags, cudaStream_t stream, const Shard& sh, bool wide_k) {
#define MIORI_GEMV(ROWS) return launch_shape<Shape<BITS, GROUP, ROWS>>(q, s, b, x, y, N, K, M, flags, stream, sh, kpar, wide_k)
        if (cls > 16u) MIORI_GEMV(32);
        if (cls > 8u) MIORI_GEMV(16);
        if (cls > 4u || (WIDE3 && cls > 2u)) MIORI_GEMV(8);
        if (M == 1u) MIORI_GEMV(1);
        if (M == 2u) MIORI_GEMV(2);
        if constexpr (!WIDE3) MIORI_GEMV(4);
#undef MIORI_GEMV
        return fail(MIORI_E_INVALID, "gemv: %u rows are not of the class of %u", M, cls);
    }
    static int run(const void* q, const void* s, const void* b, const void* x, void* y, uint32_t N, uint32_t K, uint32_t M,
                   uint32_t flags, cudaStream_t stream, Shard sh) {
        if constexpr (BITS == 4 && GROUP == 64) {
            // the class of one and two rows: exact integer sums (gemv_digits.cuh)
            if (M <= 2u && gemvdigits::takes(N, K, sh.pre.gamma != nullptr))
                return gemvdigits::launch_rows(q, s, b, x, y, N, K, M, flags, stream, sh);
        }
        uint32_t cls = class_of(M), kpar = 0;
        while (cls && (kpar = kpar_of(cls, N, K)) == 0u) cls >>= 1;
        const bool wide_k = cls == 0u;  // not even one row and its scales fit
        if (wide_k) {
            if (sh.gated || sh.post.residual || sh.best || sh.pa.world > 1) return 1;
            cls = 1u, kpar = choose_kpar<Shape<BITS, GROUP, 1>>(N, K, 1u, false);
            if (!kpar) return 1;
        }
        const uint32_t launches = (M + cls - 1u) / cls, rows = (M + launches - 1u) / launches;
        const uint32_t n_out = sh.gated ? N / 2u : sh.pa.world > 1 || sh.best ? sh.n_total : N;
        const size_t x_row = (size_t)K * (sh.pre.gamma ? 4 : 2), y_row = (size_t)n_out * ((flags & MIORI_OUT_BF16) ? 2 : 4);
        for (uint32_t m0 = 0; m0 < M; m0 += rows) {
            const int rc = launch(cls, kpar, q, s, b, static_cast<const uint8_t*>(x) + m0 * x_row, static_cast<uint8_t*>(y) + m0 * y_row,
                                  N, K, std::min(rows, M - m0), flags, stream, sh, wide_k);
            if (rc) return rc;
            sh.y_off += rows * y_row;
            if (sh.post.residual) sh.post.residual += (size_t)rows * N;
        }
        return MIORI_OK;
    }
};

// Launch, or return 1 if not even one row of K activations fits shared memory, or a fused form does not take the
// shape (nothing launched).
template <int BITS>
int try_launch(const void* q, const void* s, const void* b, const void* x, void* y, uint32_t N, uint32_t K, uint32_t M,
               uint32_t group, uint32_t flags, cudaStream_t stream, const Shard& sh = Shard()) {
    const bool fused = sh.pa.world > 1 || sh.best || sh.gated || sh.post.residual || sh.pre.gamma;
    if (fused && (K / group) % 8 != 0) return 1;  // what the fused entries promise to take
    return group == 64 ? Batch<BITS, 64>::run(q, s, b, x, y, N, K, M, flags, stream, sh)
                       : Batch<BITS, 32>::run(q, s, b, x, y, N, K, M, flags, stream, sh);
}

}  // namespace gemvtma
}  // namespace miori_b200
