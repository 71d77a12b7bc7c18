"""The weight-streaming GEMV where it can go wrong: ragged rows (scales copied in part by hand), K that
ends inside a step, a run or a slab, scale rows without a 16-byte pitch, groups that share a tile, every
number-of-rows shape, more rows than one launch holds."""
import numpy as np
import pytest
import torch

import miori_b200
from miori_b200 import synth
from conftest import TOL_EXACT_PATH, assert_close, u16, u32

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
OPS = {4: miori_b200.gemv4, 8: miori_b200.gemv8}


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("N,K,group", [(1, 32, 32), (15, 64, 64), (33, 96, 32), (17, 160, 32), (100, 1440, 32), (70, 2112, 64),
                                       (2500, 2048, 64), (40, 3456, 64), (31, 4128, 32), (700, 8192, 64), (48, 6144, 32),
                                       (9473, 320, 64)])
@pytest.mark.parametrize("M", [1, 2, 3, 5, 9, 17])
def test_edges(port, bits, N, K, group, M):
    q, s, b = synth.make_weight(N, K, bits, group, seed=N + K + M)
    x = synth.make_activation(M, K, seed=M)
    guard = torch.full((M * N + 64,), 777.0, device=DEV)
    y = guard[32:32 + M * N].view(M, N)
    OPS[bits](q.to(DEV), s.to(DEV), b.to(DEV), x.to(DEV), group=group, out=y)
    torch.cuda.synchronize()
    want = port.gemv(bits, u32(q), u16(s), u16(b), u16(x), group)
    assert_close(y.cpu().numpy(), want, rel_max=TOL_EXACT_PATH, what=f"gemv{bits} N={N} K={K} g={group} M={M}")
    assert (guard[:32] == 777.0).all() and (guard[32 + M * N:] == 777.0).all()
    assert miori_b200.lib.miori_device_error_poll() == 0


@pytest.mark.parametrize("bits,group", [(4, 32), (4, 64), (8, 32), (8, 64)])
def test_activation_range_per_group(port, bits, group):
    """Activations are scaled to fp16 by their group's power of two: groups of very different size, zeros,
    and a group with an outlier next to small values."""
    N, K = 64, 1024
    q, s, b = synth.make_weight(N, K, bits, group, seed=3)
    x = synth.make_activation(2, K, seed=4).float()
    scale = torch.exp2((torch.arange(K) // group % 5 - 2).float() * 12)
    x = x * scale
    x[0, :group] = 0.0
    x[1, 5] = 3.0e4
    x = x.to(torch.bfloat16)
    want = port.gemv(bits, u32(q), u16(s), u16(b), u16(x), group)
    got = OPS[bits](q.to(DEV), s.to(DEV), b.to(DEV), x.to(DEV), group=group).cpu().numpy()
    assert_close(got, want, rel_max=TOL_EXACT_PATH, what="groups of different size")
    for k in (-60, 90):
        xs = (x.float() * 2.0 ** k).to(torch.bfloat16)
        assert np.array_equal(OPS[bits](q.to(DEV), s.to(DEV), b.to(DEV), xs.to(DEV), group=group).cpu().numpy(),
                              got * np.float32(2.0 ** k))


@pytest.mark.parametrize("M", [1, 2, 3, 4])
def test_rows_of_one_class_are_bit_identical(M):
    N, K = 96, 4096
    for bits, group in ((4, 32), (8, 32), (8, 64)):
        q, s, b = (t.to(DEV) for t in synth.make_weight(N, K, bits, group, seed=bits))
        x = synth.make_activation(4, K, seed=9, device=DEV)
        full = OPS[bits](q, s, b, x, group=group)
        assert torch.equal(OPS[bits](q, s, b, x[:M].contiguous(), group=group), full[:M])


@pytest.mark.parametrize("M,K", [(32, 8192), (13, 16384), (5, 24576)])
def test_more_rows_than_a_launch_holds(port, M, K):
    N = 40
    q, s, b = synth.make_weight(N, K, 4, 64, seed=K)
    x = synth.make_activation(M, K, seed=M)
    want = port.gemv(4, u32(q), u16(s), u16(b), u16(x), 64)
    got = miori_b200.gemv4(q.to(DEV), s.to(DEV), b.to(DEV), x.to(DEV), group=64, flags=miori_b200.LAUNCH_PDL).cpu().numpy()
    assert_close(got, want, rel_max=TOL_EXACT_PATH, what=f"M={M} K={K}")


@pytest.mark.parametrize("N,K", [(40, 256), (2048, 2048), (5000, 2048)])
def test_plain_launch_reads_what_the_launch_before_it_wrote(N, K):
    """Without the early-start flag a launch may have its weights, its cache or its activations written by
    whatever precedes it on the stream, kernels that let their dependents start early included."""
    ws = [synth.make_weight(N, K, 4, 64, seed=i, device=DEV) for i in range(3)]
    x = synth.make_activation(1, K, seed=9, device=DEV)
    want = [miori_b200.gemv4(*w, x, group=64) for w in ws]
    caches = [miori_b200.dequant4_cache(*w, group=64) for w in ws]
    torch.cuda.synchronize()
    live = [t.clone() for t in ws[0]]
    warm = torch.empty((1, N), device=DEV)
    for it in range(30):
        i = it % 3
        miori_b200.gemv4(*ws[i], x, group=64, flags=miori_b200.LAUNCH_PDL, out=warm)
        for t, src in zip(live, ws[i]):
            t.copy_(src)
        got = miori_b200.gemv4(*live, x, group=64)
        again = miori_b200.dequant4_cache(*live, group=64)
        assert torch.equal(got, want[i]) and torch.equal(again, caches[i]), it


def _weights64(q, s, b, bits, group):
    shift = torch.arange(32 // bits, device=q.device, dtype=torch.int64) * bits
    codes = ((q.to(torch.int64).unsqueeze(-1) >> shift) & (2 ** bits - 1)).reshape(q.shape[0], -1)
    return codes.double() * s.double().repeat_interleave(group, 1) + b.double().repeat_interleave(group, 1)


@pytest.mark.parametrize("bits", [4, 8])
@pytest.mark.parametrize("group", [32, 64])
@pytest.mark.parametrize("N,K", [(2048, 2048), (256, 8192)])
@pytest.mark.parametrize("M", [1, 2, 4, 8, 16, 32])
def test_error_is_that_of_fp32_sums(bits, group, N, K, M):
    """Against 64-bit sums, 2-norm over 2-norm.  Products are exact; a group's sum and its bias term, each about
    1.5 times the result, and the sum over groups take a rounding of 2^-24 each, and the result one: under 4 of
    them.  (Whatever the tensor core cuts off has to stay below that.)"""
    q, s, b = synth.make_weight(N, K, bits, group, seed=N + K, device=DEV)
    x = synth.make_activation(M, K, seed=M, device=DEV)
    want = x.double() @ _weights64(q, s, b, bits, group).T
    got = OPS[bits](q, s, b, x, group=group).double()
    assert float((got - want).norm() / want.norm()) < 4 * 2.0 ** -24


# shapes where the number of groups that share a tile, or of launches that a batch is dealt to, would change inside the class
@pytest.mark.parametrize("bits,group,N,K,lo,hi", [
    (4, 64, 2048, 8192, 3, 8), (4, 64, 256, 8192, 9, 16), (4, 32, 256, 8192, 5, 8), (4, 64, 1024, 16384, 3, 8), (4, 64, 1024, 16384, 1, 2),
    (8, 64, 2048, 4096, 9, 16), (8, 32, 64, 16384, 1, 4), (4, 64, 256, 3072, 17, 32), (4, 32, 48, 6144, 9, 16), (8, 64, 48, 8192, 17, 32)])
def test_a_row_does_not_depend_on_the_batch_of_its_class(bits, group, N, K, lo, hi):
    q, s, b = synth.make_weight(N, K, bits, group, seed=K, device=DEV)
    x = synth.make_activation(hi, K, seed=9, device=DEV)
    full = OPS[bits](q, s, b, x, group=group)
    for M in range(lo, hi):
        assert torch.equal(OPS[bits](q, s, b, x[:M].contiguous(), group=group), full[:M]), M


@pytest.mark.parametrize("group,K,M", [(32, 32768, 2), (64, 8192, 9), (64, 16384, 4)])
def test_fused_forms_of_batches_dealt_to_several_launches(group, K, M):
    """Bit for bit the unfused pair, also where a launch does not hold the batch."""
    N = 64
    q, s, b = synth.make_weight(N, K, 4, group, seed=K, device=DEV)
    x = synth.make_activation(M, K, seed=M, device=DEV)
    v = miori_b200.gemv4(q, s, b, x, group=group)
    want = miori_b200.silu_mul(v[:, :N // 2].contiguous(), v[:, N // 2:].contiguous())
    assert torch.equal(miori_b200.gemv4_silu(q, s, b, x, group=group), want)
    if M <= 4:
        res, w = torch.randn((M, N), device=DEV), synth.make_activation(1, N, seed=1, device=DEV).reshape(-1)
        counter = torch.zeros(1, dtype=torch.int32, device=DEV)
        got = miori_b200.gemv4_post_norm_add(q, s, b, x, res, w, 1e-5, counter, group=group)
        assert torch.equal(got, miori_b200.post_norm_add(res, v, w, 1e-5)) and int(counter) == 0
        xf, g = x.float() * 3.0, synth.make_activation(1, K, seed=2, device=DEV).reshape(-1)
        y = miori_b200.gemv4_rmsnorm(q, s, b, xf, g, 1e-5, group=group)
        z = miori_b200.silu_mul(y[:, :N // 2].contiguous(), y[:, N // 2:].contiguous())
        assert torch.equal(miori_b200.gemv4_rmsnorm_silu(q, s, b, xf, g, 1e-5, group=group), z)


@pytest.mark.parametrize("bits,group,K", [(4, 32, 51200), (8, 32, 56320), (4, 64, 75776), (8, 64, 74752), (8, 32, 50432)])
@pytest.mark.parametrize("N,M", [(24, 1), (2500, 1), (40, 3)])
def test_rows_whose_scales_do_not_fit_beside_them(bits, group, K, N, M):
    q, s, b = synth.make_weight(N, K, bits, group, seed=K, device=DEV)
    w = _weights64(q, s, b, bits, group)
    x = synth.make_activation(M, K, seed=M, device=DEV)
    guard = torch.full((M * N + 64,), 777.0, device=DEV)
    y = guard[32:32 + M * N].view(M, N)
    OPS[bits](q, s, b, x, group=group, out=y)
    want = x.double() @ w.T
    assert float((y.double() - want).norm() / want.norm()) < 8 * 2.0 ** -24  # as above, and four times as many groups
    assert (guard[:32] == 777.0).all() and (guard[32 + M * N:] == 777.0).all()
    if K // group % 8 == 0:
        g = synth.make_activation(1, K, seed=2, device=DEV).reshape(-1)
        xf = x.float() * 3.0
        xn = (xf.double() * (xf.double().pow(2).mean(1, keepdim=True) + 1e-5).rsqrt() * g.double()).to(torch.bfloat16)
        got = (miori_b200.gemv4_rmsnorm if bits == 4 else miori_b200.gemv8_rmsnorm)(q, s, b, xf, g, 1e-5, group=group).double()
        want = xn.double() @ w.T
        assert float((got - want).norm() / want.norm()) < 1e-4  # single roundings of the normalised activations may tip over
    assert miori_b200.lib.miori_device_error_poll() == 0


# one and two rows of 4-bit weights in groups of 64: rows of one to eight 128-byte pieces and of several slabs, whole and not, one
# tile, as many as CTAs, one more, and several batches of a CTA's tiles
@pytest.mark.parametrize("K", [256, 512, 768, 1024, 1280, 1792, 2048, 2304, 3840, 4096, 7936, 8192])
@pytest.mark.parametrize("N", [1, 17, 2368, 2371, 40000])
def test_integer_sums_of_one_and_two_rows(K, N):
    if N * K > 1 << 27:
        pytest.skip("covered by shorter rows")
    q, s, b = synth.make_weight(N, K, 4, 64, seed=N + K, device=DEV)
    x = synth.make_activation(2, K, seed=K, device=DEV)
    x[1, K // 2:] *= 2.0 ** -9   # groups of different size
    guard = torch.full((2 * N + 64,), 777.0, device=DEV)
    y = guard[32:32 + 2 * N].view(2, N)
    miori_b200.gemv4(q, s, b, x, group=64, flags=miori_b200.LAUNCH_PDL, out=y)
    groups = x.double().view(2, -1, 64)
    parts = torch.einsum("mgk,ngk->mng", groups, _weights64(q, s, b, 4, 64).view(N, -1, 64))
    bias = torch.einsum("mg,ng->mng", groups.sum(-1), b.double())
    want, size = parts.sum(-1), (parts.abs() + 2 * bias.abs()).square().sum(-1).sqrt()
    # a group's sum is exact; that of its codes and its bias term (which cancel), and the sum over groups, round by 2^-24 of
    # what they come to, some three times a group and at random
    for m in (0, 1):
        assert float((y[m].double() - want[m]).norm() / size[m].norm()) < 4 * 2.0 ** -24
        assert torch.equal(miori_b200.gemv4(q, s, b, x[m:m + 1].contiguous(), group=64), y[m:m + 1])
    assert (guard[:32] == 777.0).all() and (guard[32 + 2 * N:] == 777.0).all()
    assert torch.equal(miori_b200.gemv4(q, s, b, x, group=64, flags=miori_b200.OUT_BF16), y.to(torch.bfloat16))
    assert miori_b200.lib.miori_device_error_poll() == 0


@pytest.mark.parametrize("K", [256, 2048, 8192])
@pytest.mark.parametrize("bad", [float("inf"), float("-inf"), float("nan")])
def test_rows_with_values_that_are_not_finite(K, bad):
    N = 100
    q, s, b = synth.make_weight(N, K, 4, 64, seed=K, device=DEV)
    x = synth.make_activation(2, K, seed=K, device=DEV)
    want = miori_b200.gemv4(q, s, b, x, group=64)
    x[1, K - 3] = bad
    got = miori_b200.gemv4(q, s, b, x, group=64)
    assert torch.equal(got[0], want[0]) and not torch.isfinite(got[1]).any()
    assert not torch.isfinite(miori_b200.gemv4(q, s, b, x[1:].contiguous(), group=64)).any()


@pytest.mark.parametrize("K", [256, 2048, 4096])
@pytest.mark.parametrize("shift", [-118, -100, -96, 100, 118])
def test_rows_next_to_nothing_and_huge_ones(K, shift):
    """bf16 goes down to 2^-126 with all its bits, and up to 2^127: what the weights make of that is in fp32's range."""
    N = 64
    q, s, b = synth.make_weight(N, K, 4, 64, seed=K, device=DEV)
    x = synth.make_activation(2, K, seed=K, device=DEV).clamp(-4.0, 4.0)
    x = torch.where(x.abs() < 2.0 ** -7, torch.full_like(x, 2.0 ** -7), x)  # no subnormals after the shift
    x[1] = x[1] * (2.0 if shift < 0 else 0.5)
    want = x.double() @ _weights64(q, s, b, 4, 64).T
    got = miori_b200.gemv4(q, s, b, (x.float() * 2.0 ** shift).to(torch.bfloat16), group=64).double() * 2.0 ** -shift
    # sums of a whole row in order at worst: K roundings, growing as their square root
    assert float((got - want).norm() / want.norm()) < 2.0 ** -24 * 4 * K ** 0.5


def test_rows_of_zeros_and_groups_of_zeros():
    N, K = 48, 1024
    q, s, b = synth.make_weight(N, K, 4, 64, seed=1, device=DEV)
    x = synth.make_activation(2, K, seed=2, device=DEV)
    x[0] = 0.0
    x[1, 64:960] = 0.0
    got = miori_b200.gemv4(q, s, b, x, group=64)
    want = x.double() @ _weights64(q, s, b, 4, 64).T
    assert (got[0] == 0).all() and float((got[1].double() - want[1]).norm() / want[1].norm()) < 4 * 2.0 ** -24


def test_fused_forms_of_activations_that_are_not_finite():
    N, K = 64, 2048
    q, s, b = synth.make_weight(N, K, 4, 64, seed=3, device=DEV)
    x = synth.make_activation(2, K, seed=4, device=DEV).float()
    x[1, 7] = float("nan")
    g = synth.make_activation(1, K, seed=2, device=DEV).reshape(-1)
    y = miori_b200.gemv4_rmsnorm(q, s, b, x, g, 1e-5, group=64)
    pair = miori_b200.gemv4(q, s, b, miori_b200.rmsnorm(x, g, 1e-5), group=64)
    assert torch.isfinite(y[0]).all() and torch.equal(y[1], pair[1])  # the norm's rounding to bf16 is for finite values
    z = miori_b200.gemv4_silu(q, s, b, x.to(torch.bfloat16), group=64)
    v = miori_b200.gemv4(q, s, b, x.to(torch.bfloat16), group=64)
    assert torch.equal(z[0], miori_b200.silu_mul(v[:, :N // 2].contiguous(), v[:, N // 2:].contiguous())[0])


@pytest.mark.parametrize("K", [512, 1536, 2048, 2560, 4096, 6656, 8192])
@pytest.mark.parametrize("N", [16, 2368, 5008])
def test_launches_of_one_and_two_rows_agree(K, N):
    """One row started early runs eight warps a CTA, one that waits and two rows run sixteen: the same bits in every form."""
    q, s, b = synth.make_weight(N, K, 4, 64, seed=N + K, device=DEV)
    x, h, res = synth.make_activation(2, K, seed=K, device=DEV), torch.randn((2, K), device=DEV), torch.randn((2, N), device=DEV)
    g, gn = (synth.make_activation(1, n, seed=n, device=DEV).reshape(-1) for n in (K, N))
    counter = torch.zeros(1, dtype=torch.int32, device=DEV)
    forms = [lambda r, f: miori_b200.gemv4(q, s, b, x[r], group=64, flags=f)]
    if K % 512 == 0:  # what the fused entries take
        forms += [lambda r, f: miori_b200.gemv4_rmsnorm(q, s, b, h[r], g, 1e-5, group=64, flags=f),
                  lambda r, f: miori_b200.gemv4_silu(q, s, b, x[r], group=64, flags=f),
                  lambda r, f: miori_b200.gemv4_rmsnorm_silu(q, s, b, h[r], g, 1e-5, group=64, flags=f),
                  lambda r, f: miori_b200.gemv4_post_norm_add(q, s, b, x[r], res[r], gn, 1e-5, counter, group=64, flags=f)]
    for i, form in enumerate(forms):
        both = form(slice(0, 2), 0)
        assert torch.isfinite(both.float()).all()
        assert torch.equal(form(slice(0, 2), miori_b200.LAUNCH_PDL), both), i
        for r in (0, 1):
            for f in (0, miori_b200.LAUNCH_PDL):
                assert torch.equal(form(slice(r, r + 1), f), both[r:r + 1]), (i, r, f)
    assert miori_b200.lib.miori_device_error_poll() == 0


@pytest.mark.parametrize("flags", [0, miori_b200.LAUNCH_PDL])
@pytest.mark.parametrize("K", [512, 2048, 3072, 8192])
def test_every_form_of_rows_next_to_nothing(K, flags):
    """Rows of activations below 2^-98 through the forms that carry a neighbour: the sums of the plain product."""
    N = 144
    q, s, b = synth.make_weight(N, K, 4, 64, seed=K, device=DEV)
    s, b = s * 2.0 ** 100, b * 2.0 ** 100  # outputs of ordinary size
    w = _weights64(q, s, b, 4, 64)
    x = synth.make_activation(2, K, seed=1, device=DEV)
    x[1] *= 2.0 ** -100
    x[0] *= 2.0 ** -90
    assert float(x[1].abs().max()) < 2.0 ** -97 and float(x[0].abs().max()) > 2.0 ** -98
    v = miori_b200.gemv4(q, s, b, x, group=64, flags=flags)
    want = x.double() @ w.T
    for m in (0, 1):  # a row's terms in order at worst, growing as the root of their number
        assert float((v[m].double() - want[m]).norm() / want[m].norm()) < 2.0 ** -24 * 4 * K ** 0.5
    z = miori_b200.silu_mul(v[:, :N // 2].contiguous(), v[:, N // 2:].contiguous())
    assert torch.equal(miori_b200.gemv4_silu(q, s, b, x, group=64, flags=flags), z) and (z[1] != 0).any()
    res, gn = torch.randn((2, N), device=DEV), synth.make_activation(1, N, seed=1, device=DEV).reshape(-1)
    counter = torch.zeros(1, dtype=torch.int32, device=DEV)
    got = miori_b200.gemv4_post_norm_add(q, s, b, x, res, gn, 1e-5, counter, group=64, flags=flags)
    assert torch.equal(got, miori_b200.post_norm_add(res, v, gn, 1e-5)) and int(counter) == 0
    for m in (0, 1):
        one = slice(m, m + 1)
        assert torch.equal(miori_b200.gemv4(q, s, b, x[one], group=64, flags=flags), v[one])
        assert torch.equal(miori_b200.gemv4_silu(q, s, b, x[one], group=64, flags=flags), z[one])
        assert torch.equal(miori_b200.gemv4_post_norm_add(q, s, b, x[one], res[one], gn, 1e-5, counter, group=64, flags=flags), got[one])
    # the norm in front: normalised rows that small, and single roundings of them may tip over
    h, g = torch.randn((2, K), device=DEV), (synth.make_activation(1, K, seed=2, device=DEV) * 2.0 ** -101).reshape(-1)
    want = miori_b200.rmsnorm(h, g, 1e-5).double() @ w.T
    y = miori_b200.gemv4_rmsnorm(q, s, b, h, g, 1e-5, group=64, flags=flags)
    assert float((y.double() - want).norm() / want.norm()) < 1e-3
    z = miori_b200.silu_mul(y[:, :N // 2].contiguous(), y[:, N // 2:].contiguous())
    assert torch.equal(miori_b200.gemv4_rmsnorm_silu(q, s, b, h, g, 1e-5, group=64, flags=flags), z) and (z != 0).any()
    assert torch.equal(miori_b200.gemv4_rmsnorm(q, s, b, h[1:], g, 1e-5, group=64, flags=flags), y[1:])
    assert miori_b200.lib.miori_device_error_poll() == 0


@pytest.mark.parametrize("K", [512, 2048, 8192])
def test_gated_outputs_of_a_row_that_is_not_finite(K):
    N = 144
    q, s, b = synth.make_weight(N, K, 4, 64, seed=3, device=DEV)
    x = synth.make_activation(2, K, seed=4, device=DEV)
    want = miori_b200.gemv4_silu(q, s, b, x, group=64)
    x[1, 7] = float("inf")
    z = miori_b200.gemv4_silu(q, s, b, x, group=64)
    v = miori_b200.gemv4(q, s, b, x, group=64)
    assert torch.equal(z[0], want[0]) and not torch.isfinite(v[1]).any()
    pair = miori_b200.silu_mul(v[1:, :N // 2].contiguous(), v[1:, N // 2:].contiguous())
    assert torch.equal(z[1:].view(torch.int16), pair.view(torch.int16))


def test_greedy_pick_of_a_row_next_to_nothing():
    from miori_b200.peers import PeerGroup
    N, K = 1000, 2048
    q, s, b = synth.make_weight(N, K, 4, 64, seed=5, device=DEV)
    s, b = s * 2.0 ** 100, b * 2.0 ** 100
    x = (synth.make_activation(1, K, seed=1, device=DEV).float() * 2.0 ** -110).to(torch.bfloat16)
    want = miori_b200.gemv4(q, s, b, x, group=64)[0]
    grp = PeerGroup(0, 1, 1 << 16, torch.device("cuda", 0))
    try:
        off_y, off_b = grp.alloc(N * 4), grp.alloc(grp.gemv_argmax_bytes())
        for flags in (0, miori_b200.LAUNCH_PDL):
            grp.gemv_argmax(4, q, s, b, x, off_y, off_b, 0, N, group=64, flags=flags)
            torch.cuda.synchronize()
            assert torch.equal(grp.tensor(off_y, (1, N))[0], want)
            assert grp.gemv_argmax_result(off_b) == (int(want.argmax()), float(want.max()))
    finally:
        grp.close()


@pytest.mark.parametrize("exponent", [6, 12, 20])
@pytest.mark.parametrize("code", [0, 1, 3, 8])
@pytest.mark.parametrize("K", [2048, 4096])
def test_outliers_whose_weights_are_zero(exponent, code, K):
    """One activation of 2^exponent a group, the others normal, and its weight exactly zero: code * s + b = 0.  An activation
    is held to 2^-25 of its group's largest, and that is all that is to be seen.  The rows of a batch of three, whose operands are
    fp16, are exact there for code 0 alone, where nothing of the outlier meets a sum: for the others they are further off."""
    N = 256
    gen = torch.Generator(device=DEV)
    gen.manual_seed(exponent)
    at = torch.randint(0, 64, (K // 64,), generator=gen, device=DEV) + torch.arange(0, K, 64, device=DEV)
    codes = torch.randint(0, 16, (N, K), generator=gen, device=DEV)
    codes[:, at] = code
    q = (codes.view(N, K // 8, 8) << (4 * torch.arange(8, device=DEV))).sum(-1)
    q = torch.where(q >= 2 ** 31, q - 2 ** 32, q).to(torch.int32)
    s = torch.randint(1, 16, (N, K // 64), generator=gen, device=DEV).to(torch.bfloat16) * 2.0 ** -10
    b = -code * s  # exact: four bits times four
    x = torch.randn((3, K), generator=gen, device=DEV).to(torch.bfloat16)
    x[:, at] = 2.0 ** exponent
    want = x.double() @ _weights64(q, s, b, 4, 64).T
    reach = (codes.double() * s.double().repeat_interleave(64, 1)).sum(1) * 2.0 ** (exponent - 25)
    # a group's sum of its codes and its bias term meet the outlier's code * s * 2^exponent each, and round it some three times
    rounding = 6 * 2.0 ** -24 * ((code * s.double()).sum(1) * 2.0 ** exponent + 64 * s.double().sum(1))
    for M in (1, 2):
        got = miori_b200.gemv4(q, s, b, x[:M].contiguous(), group=64).double()
        assert ((got - want[:M]).abs() <= reach + rounding).all()
    if code:
        wide = miori_b200.gemv4(q, s, b, x, group=64).double()
        assert float((got - want[:2]).norm()) < float((wide[:2] - want[:2]).norm())


@pytest.mark.parametrize("K", [256, 1536, 2048])
@pytest.mark.parametrize("more", [0, 1])
def test_early_rows_about_the_length_at_which_they_stop_sharing_an_sm(K, more):
    """192 KiB of codes an SM and one row of the tensor more: eight warps a CTA, sixteen beyond, the same bits."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    N = sms * 192 * 1024 // (K // 2) + more
    q, s, b = synth.make_weight(N, K, 4, 64, seed=K, device=DEV)
    x = synth.make_activation(2, K, seed=K, device=DEV)
    both = miori_b200.gemv4(q, s, b, x, group=64)
    want = x.double() @ _weights64(q, s, b, 4, 64).T
    assert float((both - want).norm() / want.norm()) < 2.0 ** -24 * 4 * K ** 0.5  # a row's terms in order at worst, at random
    for r in (0, 1):
        assert torch.equal(miori_b200.gemv4(q, s, b, x[r:r + 1], group=64, flags=miori_b200.LAUNCH_PDL), both[r:r + 1])
    assert miori_b200.lib.miori_device_error_poll() == 0


@pytest.mark.parametrize("K,values", [(8192, (2.0 ** 24, 1.0, 1.0, -2.0 ** 24)), (6144, (2.0 ** 24, 1.0, -2.0 ** 24)), (6144, (1.0, 2.0 ** 24, -2.0 ** 24))])
@pytest.mark.parametrize("flags", [0, miori_b200.LAUNCH_PDL])
def test_slabs_of_a_row_are_added_in_order(K, values, flags):
    """2048 activations at a time, from the first on: 2^24 + 1 is 2^24 in fp32, with the ones by themselves the sums were others."""
    N = 48
    x = torch.zeros((2, K), dtype=torch.bfloat16, device=DEV)
    x[:, ::2048] = torch.tensor(values, device=DEV).to(torch.bfloat16)
    q = torch.full((N, K // 8), 0x11111111, dtype=torch.int32, device=DEV)
    s = torch.ones((N, K // 64), dtype=torch.bfloat16, device=DEV)
    b = torch.zeros_like(s)
    want = torch.zeros((), device=DEV)
    for v in values:
        want = want + v
    for M in (1, 2):
        assert (miori_b200.gemv4(q, s, b, x[:M].contiguous(), group=64, flags=flags) == want).all()
