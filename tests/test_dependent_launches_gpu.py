"""Launches that start early and read what the launch before them writes: buffers that are written again and again,
as a decode step does, give what the same calls give one at a time."""
import pytest
import torch

import miori_b200 as mb
from miori_b200 import synth

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
EPS = 1e-5
HID, QKV, FF = 2048, 3072, 8192


@pytest.mark.parametrize("group", [32, 64])
@pytest.mark.parametrize("M", [1, 2, 3, 5, 8, 13, 16, 24, 32, 40, 130])
def test_step_of_early_launches_equals_its_calls_one_at_a_time(M, group):
    layers = 6
    shapes = ((QKV, HID), (HID, HID), (2 * FF, HID), (HID, FF))
    w = [[synth.make_weight(N, K, 4, group, seed=10 * l + i, device=DEV) for i, (N, K) in enumerate(shapes)] for l in range(layers)]
    cache = [[mb.dequant4_cache(*t, group=group) for t in ws] for ws in w]
    head = synth.make_weight(8192, HID, 8, group, seed=1, device=DEV)
    gamma = torch.ones(HID, dtype=torch.bfloat16, device=DEV)
    table, tokens = synth.make_weight(500, HID, 8, group, seed=2, device=DEV), torch.arange(M, device=DEV, dtype=torch.int32)
    gate_w = synth.make_activation(16, HID, seed=3, device=DEV)
    need = [mb.gemm_workspace(M, N, K, DEV) for N, K in shapes]
    ws = max((t for t in need if t is not None), key=lambda t: t.numel(), default=None)
    bf, f32 = torch.bfloat16, torch.float32
    emb, xn, act = (torch.empty((M, n), dtype=bf, device=DEV) for n in (HID, HID, FF))
    qkv, proj, h, mid, gates = (torch.empty((M, n), dtype=f32, device=DEV) for n in (QKV, HID, HID, HID, 16))
    gu, logits = torch.empty((M, 2 * FF), dtype=f32, device=DEV), torch.empty((M, 8192), dtype=bf, device=DEV)

    def linear(l, i, x, out, flags):
        if M <= 32:
            mb.linear4(*w[l][i], cache[l][i], x, group=group, flags=flags, out=out, workspace=ws)
        else:
            mb.gemm_bf16_cache(x, cache[l][i], shapes[i][0], flags=flags, out=out, workspace=ws)

    def step(flags, between):
        seen = []

        def keep(*ts):  # every layer's values, read by a launch that is not early
            seen.extend(t.clone() for t in ts)

        mb.embed8(*table, tokens, group=group, flags=flags, out=emb)
        between()
        h.copy_(emb)
        for l in range(layers):
            calls = [lambda: mb.rmsnorm(h, gamma, EPS, flags=flags, out=xn), lambda: linear(l, 0, xn, qkv, flags),
                     lambda: mb.gemm_bf16_strided(xn, gate_w, flags=flags, out=gates),
                     lambda: linear(l, 1, xn, proj, flags), lambda: mb.post_norm_add(h, proj, gamma, EPS, flags=flags, out=mid),
                     lambda: mb.rmsnorm(mid, gamma, EPS, flags=flags, out=xn), lambda: linear(l, 2, xn, gu, flags),
                     lambda: mb.silu_mul(gu.view(2, M, FF)[0], gu.view(2, M, FF)[1], flags=flags, out=act)]
            if M <= 16 and l % 2:
                calls[6:] = [lambda: mb.gemv4_silu(*w[l][2], xn, group=group, flags=flags, out=act)]
            calls += [lambda: linear(l, 3, act, proj, flags), lambda: mb.post_norm_add(mid, proj, gamma, EPS, flags=flags, out=h)]
            for call in calls:
                call()
                between()
            if l % 3 == 2:
                keep(h, mid, xn, qkv, gates, act)
        mb.rmsnorm(h, gamma, EPS, flags=flags, out=xn)
        between()
        if M <= 32:
            mb.gemv8(*head, xn, group=group, flags=flags | mb.OUT_BF16, out=logits)
            between()
            keep(logits, *mb.argmax(logits[M - 1], flags=flags))
        return seen

    want = step(0, torch.cuda.synchronize)
    for it in range(20):
        got = step(mb.LAUNCH_PDL, lambda: None)
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(got, want)), it
    assert mb.lib.miori_device_error_poll() == 0


@pytest.mark.parametrize("bits,group", [(4, 32), (4, 64), (8, 64)])
@pytest.mark.parametrize("M", [1, 2, 3, 4])
def test_fused_launches_that_start_early_equal_their_calls_one_at_a_time(M, bits, group):
    """The forms that carry a neighbour: the norm reads rows that the launch before wrote, in place."""
    layers = 6
    shapes = ((QKV, HID), (HID, HID), (2 * FF, HID), (HID, FF))
    w = [[synth.make_weight(N, K, bits, group, seed=10 * l + i, device=DEV) for i, (N, K) in enumerate(shapes)] for l in range(layers)]
    gamma, h0 = torch.ones(HID, dtype=torch.bfloat16, device=DEV), torch.randn((M, HID), device=DEV)
    counter = torch.zeros(1, dtype=torch.int32, device=DEV)
    qkv, proj, h, mid = (torch.empty((M, n), device=DEV) for n in (QKV, HID, HID, HID))
    gu, act, attn = torch.empty((M, 2 * FF), device=DEV), *(torch.empty((M, n), dtype=torch.bfloat16, device=DEV) for n in (FF, HID))

    def step(flags, between):
        kw, seen = dict(group=group, flags=flags), []
        h.copy_(h0)
        for l in range(layers):
            a, b, c, d = w[l]
            normed = mb.gemv4_rmsnorm if bits == 4 else mb.gemv8_rmsnorm
            calls = [lambda: normed(*a, h, gamma, EPS, out=qkv, **kw),
                     lambda: mb.silu_mul(qkv.view(-1)[:M * HID].view(M, HID), qkv.view(-1)[M * HID // 2:][:M * HID].view(M, HID), flags=flags, out=attn)]
            if bits == 4 and l % 2:
                calls += [lambda: mb.gemv4_post_norm_add(*b, attn, h, gamma, EPS, counter, out=mid, **kw),
                          lambda: mb.gemv4_rmsnorm_silu(*c, mid, gamma, EPS, out=act, **kw),
                          lambda: mb.gemv4_post_norm_add(*d, act, mid, gamma, EPS, counter, out=h, **kw)]
            else:
                plain = mb.gemv4 if bits == 4 else mb.gemv8
                calls += [lambda: plain(*b, attn, out=proj, **kw), lambda: mb.post_norm_add(h, proj, gamma, EPS, flags=flags, out=mid),
                          lambda: normed(*c, mid, gamma, EPS, out=gu, **kw),
                          lambda: mb.silu_mul(gu.view(2, M, FF)[0], gu.view(2, M, FF)[1], flags=flags, out=act),
                          lambda: plain(*d, act, out=proj, **kw), lambda: mb.post_norm_add(mid, proj, gamma, EPS, flags=flags, out=h)]
            for call in calls:
                call()
                between()
            if l % 3 == 2:
                seen.extend(t.clone() for t in (h, mid, qkv, act))
        return seen

    want = step(0, torch.cuda.synchronize)
    for it in range(20):
        got = step(mb.LAUNCH_PDL, lambda: None)
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(got, want)), it
    assert int(counter) == 0 and mb.lib.miori_device_error_poll() == 0
