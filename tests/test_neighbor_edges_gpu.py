"""RMSNorm, post-norm + residual, SiLU x up, arg-max and the cache build where their dispatch changes: rows
beyond one trip of the block, sizes that are no multiple of the vector, bases off the 16-byte boundary,
ties and NaNs, the smallest and largest grids."""
import numpy as np
import pytest
import torch

import miori_b200
from miori_b200 import synth
from conftest import assert_close, u16, u32

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _steps(a, b):
    def key(v):
        v = v.astype(np.int32)
        return np.where(v & 0x8000, 0x8000 - (v & 0x7FFF), v + 0x8000)
    return np.abs(key(a) - key(b))


def _shifted(t, shift):
    """The tensor on the GPU, `shift` elements into an allocation."""
    room = torch.zeros(t.numel() + 8, dtype=t.dtype, device=DEV)
    view = room[shift:shift + t.numel()].view(t.shape)
    view.copy_(t)
    return view


@pytest.mark.parametrize("rows,n", [(1, 1), (2, 7), (3, 1023), (2, 2048), (2, 2052), (5, 4096), (2, 4100), (1, 8192), (2, 8196), (1, 20001)])
@pytest.mark.parametrize("shift", [0, 1])
def test_norms(port, rows, n, shift):
    g = torch.Generator().manual_seed(rows + n)
    x, src = torch.randn((rows, n), generator=g), torch.randn((rows, n), generator=g) * 2.0
    w = (torch.randn(n, generator=g) * 0.2 + 1.0).to(torch.bfloat16)
    y = miori_b200.rmsnorm(_shifted(x, shift), _shifted(w, shift), 1e-5)
    d = _steps(u16(y), port.rmsnorm(x.numpy(), u16(w), 1e-5))
    assert d.max() <= 1 and (d != 0).mean() < 0.02 + 1.0 / n
    out = miori_b200.post_norm_add(_shifted(x, shift), _shifted(src, shift), _shifted(w, shift), 1e-5)
    assert_close(out.cpu().numpy(), port.post_norm_add(x.numpy(), src.numpy(), u16(w), 1e-5), rel_max=1e-6, what="post_norm_add")


@pytest.mark.parametrize("n", [1, 3, 8, 1021, 4096, 300003])
@pytest.mark.parametrize("shift", [0, 1])
def test_silu(port, n, shift):
    g = torch.Generator().manual_seed(n)
    gate, up = torch.randn(n, generator=g) * 4.0, torch.randn(n, generator=g)
    d = _steps(u16(miori_b200.silu_mul(_shifted(gate, shift), _shifted(up, shift))), port.silu_mul(gate.numpy(), up.numpy()))
    assert d.max() <= 1 and (d != 0).mean() < 0.01 + 1.0 / n


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_argmax_special_values(dtype):
    for n in (5, 9000):
        v = torch.full((n,), float("-inf"), dtype=dtype, device=DEV)
        assert int(miori_b200.argmax(v)[0]) == 0          # all tie
        v[n - 2:] = -3.0
        assert int(miori_b200.argmax(v)[0]) == n - 2
        v.fill_(float("nan"))
        v[3] = -1.0
        idx, val = miori_b200.argmax(v)                  # NaN never wins
        assert int(idx) == 3 and float(val) == -1.0


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("n", [5, 9000])
def test_argmax_zeros_tie_and_keep_their_sign(dtype, n):
    for zeros in ((-0.0, 0.0), (0.0, -0.0)):
        v = torch.full((n,), -2.0, dtype=dtype, device=DEV)
        v[n - 3], v[n - 1] = zeros
        idx, val = miori_b200.argmax(v)
        assert int(idx) == n - 3 and float(val).hex() == zeros[0].hex()


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("N,K,group", [(1, 32, 32), (3, 96, 32), (7, 2048, 64), (149, 1440, 32), (20000, 320, 64), (33, 8192, 64)])
def test_cache_build(port, bits, N, K, group):
    q, s, b = synth.make_weight(N, K, bits, group, seed=N + K)
    fn = miori_b200.dequant4_rowmajor if bits == 4 else miori_b200.dequant8_rowmajor
    guard = torch.full((N + 2, K), 7.0, dtype=torch.bfloat16, device=DEV)
    fn(q.to(DEV), s.to(DEV), b.to(DEV), group=group, out=guard[1:N + 1])
    assert np.array_equal(u16(guard[1:N + 1]), port.dequant_rowmajor(bits, u32(q), u16(s), u16(b), group))
    assert (guard[0] == 7.0).all() and (guard[N + 1] == 7.0).all()
