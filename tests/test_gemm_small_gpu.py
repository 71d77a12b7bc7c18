"""GEMMs of few rows (a cluster of CTAs per tile, K slices meeting in distributed shared memory) and of
few columns (operands straight from global memory), at the edges of their tiles, slices and ranges; tiles
of 192 columns on SM pairs."""
import ctypes as C

import pytest
import torch

import miori_b200
from miori_b200 import synth
from conftest import assert_close, u16

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
NARROW = 0x100  # force the tiled kernel with 128 x 128 tiles


def _bf16(rows, cols, seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return torch.randn((rows, cols), generator=g, device=DEV).to(torch.bfloat16)


@pytest.mark.parametrize("M,N,K", [(16, 3072, 2048), (48, 512, 4096), (1, 512, 4096)])
def test_split_sums_are_as_exact_as_the_tiled_kernels(M, N, K):
    """Chains of four k-blocks, each of which costs about 2^-24 of the result (2-norm over 2-norm, against 64 bits)."""
    A, B, ws = _bf16(M, K, 1), _bf16(N, K, 2), torch.empty(16, device=DEV)
    want = A.double() @ B.double().T
    got = miori_b200.gemm_bf16_cache(A, B.view(-1), N, workspace=ws).double()
    assert float((got - want).norm() / want.norm()) < 5 * 2.0 ** -24


def test_a_workspace_of_no_bytes_is_none():
    M, N, K = 32, 512, 4096
    A, B, ws = _bf16(M, K, 1), _bf16(N, K, 2), torch.empty(1 << 20, device=DEV)

    def product(nbytes):
        c = torch.empty((M, N), device=DEV)
        rc = miori_b200.lib.miori_gemm_bf16_cache_ws(A.data_ptr(), B.data_ptr(), c.data_ptr(), M, N, K, 0, ws.data_ptr(), nbytes,
                                                     torch.cuda.current_stream().cuda_stream)
        assert rc == 0
        return c
    unsplit = miori_b200.gemm_bf16_cache(A, B.view(-1), N)
    assert torch.equal(product(0), unsplit) and not torch.equal(product(4 << 20), unsplit)


# N, K: clusters of 8, 8, 4, 2, 1 and 1 CTAs; ragged last tiles, uneven slices, one k-block
@pytest.mark.parametrize("N,K", [(8, 4096), (1000, 4160), (2056, 2112), (5000, 1088), (136, 64), (16384, 192)])
@pytest.mark.parametrize("M", [1, 15, 17, 32, 48])
def test_few_rows(port, N, K, M):
    A, B = _bf16(M, K, M + K), _bf16(N, K, N + K)
    cache = B.view(-1)
    ws = torch.empty(16, device=DEV)  # its presence allows the split
    guard = torch.full((M * N + 64,), 777.0, device=DEV)
    split = guard[32:32 + M * N].view(M, N)
    miori_b200.gemm_bf16_cache(A, cache, N, out=split, workspace=ws)
    want = port.gemm_bf16(u16(A), u16(B))
    assert_close(split.cpu().numpy(), want, rel_max=1e-4, what=f"{M}x{N}x{K}")
    assert (guard[:32] == 777.0).all() and (guard[32 + M * N:] == 777.0).all()
    # rows do not depend on M, the bf16 epilogue rounds the fp32 result, unsplit is the tiled kernel's product
    assert torch.equal(miori_b200.gemm_bf16_cache(A[:(M + 1) // 2], cache, N, workspace=ws), split[:(M + 1) // 2])
    c16 = miori_b200.gemm_bf16_cache(A, cache, N, flags=miori_b200.OUT_BF16, workspace=ws)
    assert torch.equal(c16, split.to(torch.bfloat16))
    assert torch.equal(miori_b200.gemm_bf16_cache(A, cache, N), miori_b200.gemm_bf16_cache(A, cache, N, flags=NARROW))
    assert miori_b200.lib.miori_device_error_poll() == 0


@pytest.mark.parametrize("M,N,K", [(1, 1, 8), (15, 7, 40), (16, 8, 512), (17, 9, 520), (33, 16, 2056), (100, 17, 2048),
                                   (31, 31, 4104), (5, 32, 4096), (4737, 16, 64), (4800, 5, 1024)])
def test_few_columns(port, M, N, K):
    A, B = _bf16(M, K + 8, M + K)[:, :K], _bf16(N, K + 16, N + K)[:, :K]
    C = torch.full((M + 2, 48), -7.0, device=DEV)
    miori_b200.gemm_bf16_strided(A, B, out=C[1:M + 1, :N])
    want = port.gemm_bf16(u16(A.contiguous()), u16(B.contiguous()))
    assert_close(C[1:M + 1, :N].cpu().numpy(), want, rel_max=1e-4, what=f"{M}x{N}x{K}")
    assert (C[0] == -7.0).all() and (C[M + 1] == -7.0).all() and (C[1:M + 1, N:] == -7.0).all()
    assert torch.equal(miori_b200.gemm_bf16_strided(A[:1], B), C[1:2, :N])
    c16 = torch.zeros((M, 64), dtype=torch.bfloat16, device=DEV)
    miori_b200.gemm_bf16_strided(A, B, flags=miori_b200.OUT_BF16, out=c16[:, :N])
    assert torch.equal(c16[:, :N], C[1:M + 1, :N].to(torch.bfloat16))


@pytest.mark.parametrize("M,N,K", [(1024, 3072, 128), (1500, 2056, 192), (2047, 3080, 64), (600, 8192, 320)])
def test_pair_tiles_of_192_columns(port, M, N, K):
    tile, ctas, splits = C.c_uint32(), C.c_uint32(), C.c_uint32()
    assert miori_b200.lib.miori_gemm_plan(M, N, K, 0, C.byref(tile), C.byref(ctas), C.byref(splits)) == 0
    assert (tile.value, ctas.value) == (192, 2), "the planner changed: pick shapes that run on these tiles"
    A, B = _bf16(M, K, M + K), _bf16(N, K, N + K)
    guard = torch.full((M + 2, N), 777.0, device=DEV)
    miori_b200.gemm_bf16_cache(A, B.view(-1), N, out=guard[1:M + 1])
    assert_close(guard[1:M + 1].cpu().numpy(), port.gemm_bf16(u16(A), u16(B)), rel_max=1e-4, what=f"{M}x{N}x{K}")
    assert (guard[0] == 777.0).all() and (guard[M + 1] == 777.0).all()
    assert torch.equal(miori_b200.gemm_bf16_cache(A, B.view(-1), N, flags=NARROW), guard[1:M + 1])
    c16 = miori_b200.gemm_bf16_cache(A, B.view(-1), N, flags=miori_b200.OUT_BF16)
    assert torch.equal(c16, guard[1:M + 1].to(torch.bfloat16))
    assert miori_b200.lib.miori_device_error_poll() == 0


@pytest.mark.parametrize("N,K", [(512, 2048), (2048, 2048), (16384, 2048)])
@pytest.mark.parametrize("M", [8, 32, 77, 256])
def test_early_launch_reads_the_cache_built_before_it(N, K, M):
    """A product launched early right behind the build of its cache, or with another early launch between, reads
    what the build wrote.  Replayed as a graph, so that nothing but the device orders them."""
    ws = [synth.make_weight(N, K, 4, 64, seed=i, device=DEV) for i in (1, 2)]
    x = synth.make_activation(M, K, seed=3, device=DEV)
    cache = torch.empty(N * K, dtype=torch.bfloat16, device=DEV)
    xf, g = torch.randn((1, 2048), device=DEV), torch.ones(2048, dtype=torch.bfloat16, device=DEV)
    product = miori_b200.gemv_bf16_cache if M == 8 else miori_b200.gemm_bf16_cache
    want = []
    for w in ws:
        miori_b200.dequant4_cache(*w, group=64, out=cache)
        torch.cuda.synchronize()
        want.append(product(x, cache, N))
    graph, got = torch.cuda.CUDAGraph(), []
    with torch.cuda.graph(graph):
        for i in range(16):
            miori_b200.dequant4_cache(*ws[i % 2], group=64, out=cache)
            if i % 4 >= 2:
                miori_b200.rmsnorm(xf, g, 1e-5, flags=miori_b200.LAUNCH_PDL)
            got.append(product(x, cache, N, flags=miori_b200.LAUNCH_PDL))
    for _ in range(3):
        graph.replay()
        torch.cuda.synchronize()
        assert [i for i, y in enumerate(got) if not torch.equal(y, want[i % 2])] == []
