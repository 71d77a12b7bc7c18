// Up to 48 rows of activations against the bf16 cache: C[M][N] = A[M][K] * Bc[N][K]^T.
//
// What bounds such a product: a wide one, one tile a CTA, the cache's trip from HBM (16384 x 2048: 4.8 TB/s); a
// short one the launch and a chain of k-blocks, each of which takes 0.23 us whatever its bytes -- the one thread
// that waits, issues four MMAs and commits is what they queue for (one computed address more in its loop
// cost 25 ns a block).  The tiled GEMM's 128 x 128 tiles of C leave most SMs without one, so K is
// split, the partials travel through a workspace and a second kernel sums them, and each of the two pays
// the hand-over to the next.  Here one kernel does it: a CTA owns 128 weight rows and a slice of K, the
// slices of a tile are the CTAs of one cluster, and the partial sums meet in distributed shared memory.
//
//   * roles are swapped against the tiled kernel: the 128 weight rows are the MMA's M (the TMEM lanes), the
//     activation rows, padded to a multiple of 16, its N -- a batch of 32 rows costs 32 columns, not a
//     128-row operand three quarters empty, and an accumulator register is one (row, column) of C whose 32
//     lanes are 128 neighbouring bytes of a row of C;
//   * warp 0 issues TMA into a ring of {128 x 64 weights, M x 64 activations} stages (the weights of the first
//     ring fill before griddepcontrol.wait: they are immutable), warp 1 issues tcgen05.mma, warps 2..5 drain;
//   * with a cluster of cs CTAs, CTA r receives columns [r MP / cs, (r + 1) MP / cs) of every CTA's partial
//     tile into the memory of its ring (free by then), adds them in rank order and stores them.  The number
//     of slices depends on N and K only.
// Every wait is bounded; the cluster barriers are reached by every thread whatever its waits returned.
//
// Measured in chains of dependent launches over caches larger than L2, the split tiled GEMM and this, us:
// 32 rows, N x K: 2048 x 2048 8.1 -> 5.4, 3072 x 2048 8.9 -> 6.5, 8192 x 2048 12.4 -> 10.5, 16384 x 2048 (one
// slice) 15.8 -> 13.9, 2048 x 8192 12.9 -> 9.7, 8192 x 8192 29.5 -> 25.7 (5.2 TB/s).  The exchange
// grows with the rows: even at 64 (6.9 and 6.7 at 2048 x 2048, 10.8 and 11.3 at 6144 x 2048), behind at 77.
#pragma once

namespace skinny {

constexpr int TILE = 128;                     // weight rows per CTA
constexpr int W_BYTES = TILE * BK * 2;        // 16 KiB per k-block
constexpr int MAX_M = 48;
constexpr int MAX_STAGES = 10;
// Accumulators of a K slice, a share of its k-blocks each, which are added in fp32: the tensor core cuts its running
// sum off instead of rounding it, and the error grows with the chain, by about 2^-24 of the result a k-block.
// (Four and eight slices of eight k-blocks, 3072 x 2048 and 512 x 4096, against 64-bit sums: 4.7e-7 of the result
// with one, 2.3e-7 with two, 1.3e-7 with four; the split tiled kernel has 3.2e-7 and 2.4e-7.  16 rows of 3072 x 2048
// take 5.8, 5.9 and 6.2 us.)  One where K is not split: the bits are then the tiled kernels'.
constexpr int ACCS = 2;

struct Geo {
    uint32_t M, N, K;
    uint32_t mp;       // activation rows padded to a multiple of 16
    uint32_t cs;       // CTAs per cluster = K slices: 1, 2, 4 or 8
    uint32_t stages;
    uint32_t tmem_cols;
    uint32_t out_bf16;
};

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),
          "=r"(r[13]), "=r"(r[14]), "=r"(r[15]) : "r"(taddr) : "memory");
}

__global__ void __launch_bounds__(THREADS)
gemm_skinny_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x,
                   void* __restrict__ C, const Geo g) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t full_bars[MAX_STAGES], empty_bars[MAX_STAGES], done_bar;
    __shared__ uint32_t tmem_base_slot;
    __shared__ volatile uint32_t abort_flag;

    const uint32_t ring = (smem_addr(smem_raw) + 1023u) & ~1023u;
    const uint32_t x_bytes = g.mp * BK * 2u, stage_bytes = (uint32_t)W_BYTES + x_bytes;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint32_t rank = g.cs > 1u ? blockIdx.x % g.cs : 0u, tile = blockIdx.x / g.cs;
    const uint32_t k_blocks = (g.K + BK - 1) / BK;  // TMA zero-fills a ragged last block
    const uint32_t kb0 = rank * k_blocks / g.cs, nkb = (rank + 1u) * k_blocks / g.cs - kb0;

    pdl_launch_dependents();
    if (threadIdx.x == 0) {
        abort_flag = 0u;
        for (uint32_t s = 0; s < g.stages; ++s) {
            mbar_init(smem_addr(&full_bars[s]), 1);
            mbar_init(smem_addr(&empty_bars[s]), 1);
        }
        mbar_init(smem_addr(&done_bar), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        // the weights of the first ring fill: no other thread is needed for that
        for (uint32_t i = 0; i < min(g.stages, nkb); ++i) {
            mbar_expect_tx(smem_addr(&full_bars[i]), stage_bytes);
            tma_load_2d(ring + i * stage_bytes, &tmap_w, (int)((kb0 + i) * BK), (int)(tile * TILE), smem_addr(&full_bars[i]));
        }
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_addr(&tmem_base_slot)), "r"(g.tmem_cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_base_slot;

    pdl_wait_prior();  // A may be produced, and C read, by the preceding kernel

    bool ok = true;
    if (warp == 0) {
        if (lane == 0) {
            uint32_t s = 0, parity = 1u;
            for (uint32_t i = 0; i < nkb && ok; ++i) {
                const uint32_t bar = smem_addr(&full_bars[s]), dst = ring + s * stage_bytes;
                if (i >= g.stages) {
                    if (!(ok = mbar_wait(smem_addr(&empty_bars[s]), parity, &abort_flag, 0x31))) break;
                    mbar_expect_tx(bar, stage_bytes);
                    tma_load_2d(dst, &tmap_w, (int)((kb0 + i) * BK), (int)(tile * TILE), bar);
                }
                tma_load_2d(dst + W_BYTES, &tmap_x, (int)((kb0 + i) * BK), 0, bar);
                if (++s == g.stages) s = 0u, parity ^= 1u;
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            // D = f32, A = B = bf16, both K-major, shape 128 x mp
            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((g.mp >> 3) << 17) | ((uint32_t)(TILE >> 4) << 24);
            const uint32_t accs = g.cs > 1u ? (uint32_t)ACCS : 1u;
            uint32_t s = 0, parity = 0u, i = 0;
            for (uint32_t a = 0; a < accs; ++a) {
                const uint32_t acc = tmem + a * g.mp, i0 = i, i1 = (a + 1u) * nkb / accs;
                for (; i < i1 && ok; ++i) {
                    if (!(ok = mbar_wait(smem_addr(&full_bars[s]), parity, &abort_flag, 0x32))) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint64_t wdesc = umma_desc_sw128(ring + s * stage_bytes);
                    const uint64_t xdesc = umma_desc_sw128(ring + s * stage_bytes + W_BYTES);
#pragma unroll
                    for (uint32_t k = 0; k < BK / UMMA_K; ++k)
                        umma_f16(acc, wdesc + 2u * k, xdesc + 2u * k, idesc, ((i - i0) | k) != 0u);
                    umma_commit(smem_addr(&empty_bars[s]));
                    if (++s == g.stages) s = 0u, parity ^= 1u;
                }
            }
            if (ok) umma_commit(smem_addr(&done_bar));
        }
    } else {
        ok = mbar_wait(smem_addr(&done_bar), 0u, &abort_flag, 0x33);
        ok = __all_sync(0xFFFFFFFFu, ok);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    }
    __syncwarp();

    const uint32_t quad = warp & 3u, row = quad * 32u + lane;  // TMEM lane quarter of an epilogue warp
    const uint32_t n = tile * TILE + row;
    auto store = [&](uint32_t m, float v) {  // 32 lanes: neighbouring elements of a row of C
        if (m < g.M && n < g.N) {
            if (g.out_bf16) static_cast<uint16_t*>(C)[(size_t)m * g.N + n] = (uint16_t)float_to_bf16_bits(v);
            else static_cast<float*>(C)[(size_t)m * g.N + n] = v;
        }
    };
    if (g.cs == 1u) {
        if (warp >= 2u && ok) {
            for (uint32_t c = 0; c < g.mp; c += 16u) {
                uint32_t r[16];
                tmem_ld16(tmem + ((quad * 32u) << 16) + c, r);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (uint32_t j = 0; j < 16u; ++j) store(c + j, __uint_as_float(r[j]));
            }
        }
    } else {
        // every CTA of the cluster has finished its MMAs: the rings may be written to
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
        // partial sums travel as four columns of a row, 16 bytes a lane: [source CTA][column / 4][row]
        const uint32_t per4 = g.mp / g.cs / 4u;  // groups of four columns that one CTA receives
        if (warp >= 2u) {
            uint32_t owner = 0, cg = 0, to = 0;
            for (uint32_t c = 0; c < g.mp; c += 16u) {
                uint32_t part[ACCS][16], (&r)[16] = part[0];
#pragma unroll
                for (uint32_t a = 0; a < (uint32_t)ACCS; ++a) tmem_ld16(tmem + ((quad * 32u) << 16) + a * g.mp + c, part[a]);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (uint32_t a = 1; a < (uint32_t)ACCS; ++a)
#pragma unroll
                    for (uint32_t j = 0; j < 16u; ++j) r[j] = __float_as_uint(__uint_as_float(r[j]) + __uint_as_float(part[a][j]));
#pragma unroll
                for (uint32_t j = 0; j < 16u; j += 4u) {
                    if (cg == 0u)
                        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(to) : "r"(ring + (rank * per4 * TILE + row) * 16u), "r"(owner));
                    asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};"
                                 ::"r"(to + cg * (TILE * 16u)), "r"(r[j]), "r"(r[j + 1]), "r"(r[j + 2]), "r"(r[j + 3]) : "memory");
                    if (++cg == per4) cg = 0u, ++owner;
                }
            }
        }
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
        if (warp >= 2u && ok) {
            for (uint32_t cg = 0; cg < per4; ++cg) {
                float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 4
                for (uint32_t p = 0; p < g.cs; ++p) {
                    float4 w;
                    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                                 : "=f"(w.x), "=f"(w.y), "=f"(w.z), "=f"(w.w) : "r"(ring + ((p * per4 + cg) * TILE + row) * 16u));
                    v = p == 0u ? w : make_float4(v.x + w.x, v.y + w.y, v.z + w.z, v.w + w.w);
                }
                const uint32_t m = (rank * per4 + cg) * 4u;
                store(m, v.x), store(m + 1u, v.y), store(m + 2u, v.z), store(m + 3u, v.w);
            }
        }
    }

    // teardown: on abort give in-flight copies and MMAs time to land before freeing TMEM
    if (abort_flag) {
        const long long t0 = clock64();
        while (clock64() - t0 < 2000000LL) __nanosleep(1000);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(g.tmem_cols) : "memory");
    }
}

// K slices for an N x K cache: as many as the SMs hold clusters for, while a slice keeps four k-blocks.
inline uint32_t slices(uint32_t N, uint32_t K) {
    const uint32_t tiles = (N + TILE - 1) / TILE, k_blocks = (K + BK - 1) / BK, sms = (uint32_t)sm_count();
    uint32_t cs = 1;
    while (cs < 8u && tiles * cs * 2u <= sms && k_blocks >= cs * 8u) cs *= 2u;
    return cs;
}

// How many slices to run a product with, 0: on the tiled kernels.  K may be split only when `split`: without,
// a row's value is the tiled kernels' for every M, and one slice gives the same bits.  One wave of CTAs only
// (24576 x 2048, 192 of them: 27.9 us against 23.3 for the persistent tiled kernel).  Unsplit the gain is
// in the prologue and the epilogue alone: it is gone at 48 rows (2048 x 2048 11.3 and 11.8) and at K = 4096 (19.2
// and 19.5).
inline uint32_t plan(uint32_t M, uint32_t N, uint32_t K, bool split) {
    const uint32_t cs = split ? slices(N, K) : 1u;
    if ((N + TILE - 1) / TILE * cs > (uint32_t)sm_count()) return 0u;
    return cs > 1u ? (M <= (uint32_t)MAX_M ? cs : 0u) : (M <= 32u && K <= 2048u ? 1u : 0u);
}

static int launch_skinny(const void* A, const void* Bc, void* Cm, uint32_t M, uint32_t N, uint32_t K, uint32_t flags,
                         uint32_t cs, cudaStream_t stream) {
    Geo g;
    g.M = M, g.N = N, g.K = K, g.cs = cs;
    const uint32_t pad = std::max(16u, 4u * cs);  // whole groups of four columns for every CTA of a cluster
    g.mp = (M + pad - 1u) / pad * pad;
    g.tmem_cols = 32u;  // of the 512 of an SM, which shared memory lets at most three of these CTAs share
    while (g.tmem_cols < g.mp * (cs > 1u ? (uint32_t)ACCS : 1u)) g.tmem_cols *= 2u;
    g.out_bf16 = flags & MIORI_OUT_BF16 ? 1u : 0u;
    const uint32_t stage_bytes = W_BYTES + g.mp * BK * 2u, k_blocks = (K + BK - 1) / BK;
    // clusters of eight find a place on half SMs only (33 of them against 15 on whole ones)
    const size_t budget = cs == 8u ? 110 * 1024 : 200 * 1024, recv = cs > 1u ? (size_t)g.mp * TILE * 4 : 0;
    g.stages = std::min<uint32_t>({(uint32_t)MAX_STAGES, (uint32_t)(budget / stage_bytes), (k_blocks + cs - 1u) / cs});
    const size_t smem = std::max<size_t>((size_t)g.stages * stage_bytes, recv) + 1024;
    CUtensorMap tw, tx;
    int rc = make_tmap(&tw, Bc, N, K, TILE, 0);
    if (rc) return rc;
    rc = make_tmap(&tx, A, M, K, g.mp, 0);
    if (rc) return rc;
    cudaError_t e = set_up_kernel(reinterpret_cast<const void*>(gemm_skinny_kernel), Split::DRIVERS);
    if (e == cudaSuccess) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((N + TILE - 1) / TILE * cs);
        cfg.blockDim = dim3(THREADS);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = stream;
        cudaLaunchAttribute attr[2];
        unsigned na = 0;
        if (cs > 1u) {
            attr[na].id = cudaLaunchAttributeClusterDimension;
            attr[na].val.clusterDim.x = cs;
            attr[na].val.clusterDim.y = attr[na].val.clusterDim.z = 1;
            ++na;
        }
        if (flags & MIORI_LAUNCH_PDL) {
            attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
            attr[na].val.programmaticStreamSerializationAllowed = 1;
            ++na;
        }
        cfg.attrs = attr;
        cfg.numAttrs = na;
        e = cudaLaunchKernelEx(&cfg, gemm_skinny_kernel, tw, tx, Cm, g);
    }
    if (e != cudaSuccess) return cuda_fail(e, "gemm_skinny launch");
    return MIORI_OK;
}

}  // namespace skinny
