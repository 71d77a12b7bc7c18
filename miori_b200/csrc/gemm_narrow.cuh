// A few output columns: C[M][N] = A[M][K] * B[N][K]^T for N <= 32 (the 16-wide gate projection).
//
// The tiled GEMM gives such a product one CTA per 128 rows, and that CTA's SM then fetches 32 KB per k-block at
// its own rate: 10.4 us at K = 2048 whatever M is.  Nothing here is worth a tensor-memory pipeline; what
// counts is the one trip to L2.  So a CTA takes ROWS = 16 or 32 rows and every column, its sixteen warps
// take every sixteenth piece of 32 k, and each lane loads its operands of mma.sync.m16n8k16 straight from
// global memory, 16 bytes a row (the k order inside a piece is the same permutation for A and B): at K =
// 2048 all loads of a warp are in flight at once.  B, the weights, is loaded before griddepcontrol.wait.
// The warps' sums meet in shared memory and are added in order, so a row does not depend on M.
// Measured in chains of dependent launches, tiled and this, us: N = 16, K = 2048, M = 1: 10.2 -> 1.8, 77: 10.4 ->
// 2.1, 1024: 10.6 -> 2.3, 4096: 10.9 -> 4.8, 32768: 41.6 -> 30.8 (4.4 TB/s); N = 32, K = 4096, M = 77: 17.8 -> 5.1.
#pragma once

namespace narrow {

constexpr int WARPS = 16, THREADS_N = WARPS * 32;

__device__ __forceinline__ void mma_bf16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// NT: sets of eight columns; MT: sets of sixteen rows of a CTA
template <int NT, int MT, bool OUT_BF16>
__global__ void __launch_bounds__(THREADS_N)
gemm_narrow_kernel(const uint16_t* __restrict__ A, const uint16_t* __restrict__ B, void* __restrict__ Cout, uint32_t M,
                   uint32_t N, uint32_t K, uint32_t lda, uint32_t ldb, uint32_t ldc) {
    constexpr int U = NT * MT <= 4 ? 4 : 2;  // pieces in flight per warp
    __shared__ float red[WARPS][16 * MT * 8 * NT];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3u;
    const uint32_t m0 = blockIdx.x * (16u * MT);
    // this lane's part of the rows it supplies; rows and columns past the end repeat the last one
    const uint16_t *a_row[2 * MT], *b_row[NT];
#pragma unroll
    for (int r = 0; r < 2 * MT; ++r) a_row[r] = A + (size_t)min(m0 + 8u * r + g, M - 1u) * lda;
#pragma unroll
    for (int j = 0; j < NT; ++j) b_row[j] = B + (size_t)min(8u * j + g, N - 1u) * ldb;
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    uint4 b[U][NT];
    auto k_of = [&](uint32_t trip, int u) { return ((trip * U + u) * WARPS + warp) * 32u + t * 8u; };
    auto load_b = [&](uint32_t trip) {
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int j = 0; j < NT; ++j)
                b[u][j] = k_of(trip, u) < K ? __ldg(reinterpret_cast<const uint4*>(b_row[j] + k_of(trip, u))) : zero;
    };
    pdl_launch_dependents();
    load_b(0u);
    pdl_wait_prior();

    float d[MT][NT][4];
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < NT; ++j) d[i][j][0] = d[i][j][1] = d[i][j][2] = d[i][j][3] = 0.0f;
    const uint32_t trips = (K + 32u * WARPS * U - 1u) / (32u * WARPS * U);
    for (uint32_t trip = 0; trip < trips; ++trip) {
        uint4 a[U][2 * MT];
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int r = 0; r < 2 * MT; ++r)
                a[u][r] = k_of(trip, u) < K ? ld_fresh(reinterpret_cast<const uint4*>(a_row[r] + k_of(trip, u))) : zero;
        if (trip) load_b(trip);
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int i = 0; i < MT; ++i)
#pragma unroll
                for (int j = 0; j < NT; ++j) {
                    const uint4 &lo = a[u][2 * i], &hi = a[u][2 * i + 1];
                    mma_bf16(d[i][j], lo.x, hi.x, lo.y, hi.y, b[u][j].x, b[u][j].y);
                    mma_bf16(d[i][j], lo.z, hi.z, lo.w, hi.w, b[u][j].z, b[u][j].w);
                }
    }
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int h = 0; h < 2; ++h)
                *reinterpret_cast<float2*>(&red[warp][(16 * i + 8 * h + g) * (8 * NT) + 8 * j + 2 * t]) =
                    make_float2(d[i][j][2 * h], d[i][j][2 * h + 1]);
    __syncthreads();
    for (uint32_t o = threadIdx.x; o < 16u * MT * 8u * NT; o += THREADS_N) {
        float v = red[0][o];
#pragma unroll
        for (int w = 1; w < WARPS; ++w) v += red[w][o];
        const uint32_t m = m0 + o / (8u * NT), n = o % (8u * NT);
        if (m < M && n < N) {
            if (OUT_BF16) static_cast<uint16_t*>(Cout)[(size_t)m * ldc + n] = (uint16_t)float_to_bf16_bits(v);
            else static_cast<float*>(Cout)[(size_t)m * ldc + n] = v;
        }
    }
}

template <int NT>
static int launch_nt(const uint16_t* A, uint32_t lda, const uint16_t* B, uint32_t ldb, void* C, uint32_t ldc, uint32_t M,
                     uint32_t N, uint32_t K, uint32_t flags, cudaStream_t stream) {
    const bool bf16 = (flags & MIORI_OUT_BF16) != 0, pdl = (flags & MIORI_LAUNCH_PDL) != 0;
    // 32 rows a CTA, so that B is read half as often, once 16 rows each make more than two waves
    constexpr int TALL = NT <= 2 ? 2 : 1;
    const bool tall = M > 2u * 16u * (uint32_t)sm_count() && TALL == 2;
    auto kern = tall ? (bf16 ? gemm_narrow_kernel<NT, TALL, true> : gemm_narrow_kernel<NT, TALL, false>)
                     : (bf16 ? gemm_narrow_kernel<NT, 1, true> : gemm_narrow_kernel<NT, 1, false>);
    const uint32_t rows = tall ? 32u : 16u;
    const cudaError_t e = launch(kern, dim3((M + rows - 1u) / rows), dim3(THREADS_N), 0, stream, pdl, A, B, C, M, N, K, lda, ldb, ldc);
    if (e != cudaSuccess) return cuda_fail(e, "gemm_narrow launch");
    return MIORI_OK;
}

// Whether a product of 16-byte aligned rows runs here.  Long ones go to the tiled kernel, which reads B once per
// 128 rows: with more than 16 columns beyond two waves of CTAs (N = 32, K = 4096, M = 8192: 21.7 us against
// 18.7), else where HBM bounds both (N = 8, K = 512, M = 32768: 11.9 and 12.3, M = 131072: 50.9 and 39.3).
inline bool takes(uint32_t M, uint32_t N, uint32_t K) {
    return K % 8 == 0 && N <= 32u && M <= (N <= 16u ? 32768u : 4096u);
}

static int launch_narrow(const void* A, uint32_t lda, const void* B, uint32_t ldb, void* C, uint32_t ldc, uint32_t M,
                         uint32_t N, uint32_t K, uint32_t flags, cudaStream_t stream) {
    const uint16_t *a = static_cast<const uint16_t*>(A), *b = static_cast<const uint16_t*>(B);
    if (N <= 8u) return launch_nt<1>(a, lda, b, ldb, C, ldc, M, N, K, flags, stream);
    if (N <= 16u) return launch_nt<2>(a, lda, b, ldb, C, ldc, M, N, K, flags, stream);
    return launch_nt<4>(a, lda, b, ldb, C, ldc, M, N, K, flags, stream);
}

}  // namespace narrow
