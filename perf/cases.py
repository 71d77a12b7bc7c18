"""The work a program built on this package has it do, as cases that can be timed and compared.

Sizes are those of the benchmark's model (hidden 2048, fused QKV 3072, feed-forward 8192, a head of
128000 or 131072 rows, 24 layers) and generic ones around them, odd and ragged ones included.  Every
case goes through the package's public operators.  A kind of work is one of

  projection     one packed projection called by itself: `gemv4` / `gemv8`, the output allocated by the
                 call.  Stand-alone probes, adapters, single layers; the smallest call is all latency.
  head           the 8-bit LM head over the vocabulary, then the greedy pick of every slot.
  stack          the projections of a whole decode step for a fixed number of slots, recorded once as a
                 CUDA graph (what an engine with fixed slots keeps) and replayed: `linear4` with the
                 bf16 cache at hand, which routes by the number of rows.
  step           one decode step issued call by call, as an engine that encodes every step does:
                 embedding, norms, projections, activation, residuals, head; attention left out.
  cache_build    the packed -> bf16 conversion that start-up runs for every projection.
  prefill_layer  one layer over the tokens of one or several prompts: norms, cache GEMMs, the 16-wide gate
                 projection, activation, residuals; attention left out.
  gemm           one cache GEMM over packed prompts.
"""
import math

import torch

import miori_b200 as mb
from miori_b200 import synth

DEV = "cuda:0"
EPS = 1e-5
HID, QKV, FF, GATE = 2048, 3072, 8192, 16
LAYER = ((QKV, HID), (HID, HID), (2 * FF, HID), (HID, FF))  # (N, K) of a layer's four projections
LARGEST_GEMM = 32768 * 16384 * 2048


def listed():
    return [
        # one slot, one projection: a few microseconds of work behind one call
        {"name": "projection-1row", "kind": "projection", "bits": 4, "N": 2048, "K": 2048, "M": 1, "group": 64, "bf16": False},
        # a ragged projection for a handful of rows in the reference's own group size: odd N, a K
        # whose scale rows are no multiple of 16 bytes
        {"name": "projection-ragged", "kind": "projection", "bits": 4, "N": 5003, "K": 1440, "M": 6, "group": 32, "bf16": True},
        # greedy decoding of one stream: the head is the longest single read of a step
        {"name": "head-1slot", "kind": "head", "N": 131072, "K": 2048, "M": 1, "group": 64},
        # four slots against the reference's vocabulary in its group size
        {"name": "head-4slots", "kind": "head", "N": 128000, "K": 2048, "M": 4, "group": 32},
        # decode of one stream, eight slots, and the widest batch
        {"name": "stack-1slot", "kind": "stack", "layers": 24, "M": 1, "group": 64},
        {"name": "stack-8slots", "kind": "stack", "layers": 24, "M": 8, "group": 64},
        {"name": "stack-32slots", "kind": "stack", "layers": 24, "M": 32, "group": 64},
        # a whole step of one stream issued eagerly, with every neighbour of the projections
        {"name": "step-1slot", "kind": "step", "layers": 24, "N": 131072, "M": 1, "group": 64},
        # start-up: the widest projection of a layer
        {"name": "cache-build", "kind": "cache_build", "bits": 4, "N": 16384, "K": 2048, "group": 64},
        # one short prompt, and packed prompts of a thousand tokens, through a layer
        {"name": "prefill-77tokens", "kind": "prefill_layer", "M": 77},
        {"name": "prefill-1024tokens", "kind": "prefill_layer", "M": 1024},
        # large packed prefill: the widest projection over 32768 tokens
        {"name": "gemm-32768tokens", "kind": "gemm", "M": 32768, "N": 16384, "K": 2048, "bf16": True},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("projection", "projection", "head", "stack", "stack", "step", "cache_build", "prefill_layer", "gemm"))
    group = rng.choice((32, 64))
    if kind == "projection":
        return {"kind": kind, "bits": rng.choice((4, 4, 8)), "N": _log(rng, 256, 32768), "K": group * max(1, _log(rng, 512, 8192) // group),
                "M": _log(rng, 1, 32), "group": group, "bf16": rng.random() < 0.5}
    if kind == "head":
        return {"kind": kind, "N": _log(rng, 8192, 131072), "K": 64 * _log(rng, 16, 64), "M": _log(rng, 1, 16), "group": group}
    if kind == "stack":
        return {"kind": kind, "layers": rng.randint(4, 24), "M": _log(rng, 1, 32), "group": group}
    if kind == "step":
        return {"kind": kind, "layers": rng.randint(4, 24), "N": _log(rng, 8192, 131072), "M": _log(rng, 1, 16), "group": group}
    if kind == "cache_build":
        K = group * max(1, _log(rng, 256, 8192) // group)
        return {"kind": kind, "bits": rng.choice((4, 4, 8)), "N": min(_log(rng, 256, 32768), (1 << 26) // K), "K": K, "group": group}
    if kind == "prefill_layer":
        return {"kind": kind, "M": _log(rng, 33, 4096)}
    N, K = 8 * _log(rng, 32, 2048), 64 * _log(rng, 8, 128)
    return {"kind": kind, "M": min(_log(rng, 33, 32768), LARGEST_GEMM // (N * K)), "N": N, "K": K, "bf16": rng.random() < 0.5}


# ---------------------------------------------------------------------------------- inputs

class _Seeds:
    """Distinct generator seeds for the tensors of one state."""

    def __init__(self, seed):
        self.next = int(seed) * 4096

    def __call__(self):
        self.next += 1
        return self.next


def _normal(seed, *shape):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return torch.randn(shape, generator=g, device=DEV)


def _gamma(seed, n):
    return (1.0 + 0.1 * _normal(seed, n)).to(torch.bfloat16)


def _weights(sd, N, K, bits, group):
    return synth.make_weight(N, K, bits, group, seed=sd(), device=DEV)


def _cache(w, group):
    return mb.dequant4_cache(*w, group=group)


class _State:
    pass


def prepare(case, seed):
    sd, st, kind = _Seeds(seed), _State(), case["kind"]
    st.case = case
    M, group = case.get("M"), case.get("group", 64)
    if kind == "projection":
        st.w = _weights(sd, case["N"], case["K"], case["bits"], group)
        st.x = synth.make_activation(M, case["K"], seed=sd(), device=DEV)
    elif kind == "head":
        st.w = _weights(sd, case["N"], case["K"], 8, group)
        st.x = synth.make_activation(M, case["K"], seed=sd(), device=DEV)
        st.logits = torch.empty((M, case["N"]), dtype=torch.bfloat16, device=DEV)
    elif kind == "stack":
        _prepare_stack(st, sd, case["layers"], M, group)
    elif kind == "step":
        _prepare_step(st, sd, case["layers"], case["N"], M, group)
    elif kind == "cache_build":
        st.w = _weights(sd, case["N"], case["K"], case["bits"], group)
        st.out = torch.empty(case["N"] * case["K"], dtype=torch.bfloat16, device=DEV)
        if case["bits"] == 8:
            st.out = st.out.view(case["N"], case["K"])
    elif kind == "prefill_layer":
        _prepare_prefill(st, sd, M)
    else:
        st.cache = _cache(_weights(sd, case["N"], case["K"], 4, 64), 64)
        st.x = synth.make_activation(M, case["K"], seed=sd(), device=DEV)
        st.ws = mb.gemm_workspace(M, case["N"], case["K"], DEV)
        st.y = torch.empty((M, case["N"]), dtype=torch.bfloat16 if case["bf16"] else torch.float32, device=DEV)
    return st


def _prepare_stack(st, sd, layers, M, group):
    st.w = [[_weights(sd, N, K, 4, group) for N, K in LAYER] for _ in range(layers)]
    st.cache = [[_cache(w, group) if M > 4 else None for w in ws] for ws in st.w]  # up to four rows run on the packed weights
    st.x = [synth.make_activation(M, K, seed=sd(), device=DEV) for _, K in LAYER]
    st.y = [torch.empty((layers, M, N), device=DEV) for N, _ in LAYER]
    need = [mb.gemm_workspace(M, N, K, DEV) for N, K in LAYER]
    st.ws = max((w for w in need if w is not None), key=lambda w: w.numel(), default=None)

    def one_pass():
        for l, (ws, cs) in enumerate(zip(st.w, st.cache)):
            for i in range(len(LAYER)):
                mb.linear4(*ws[i], cs[i], st.x[i], group=group, flags=mb.LAUNCH_PDL, out=st.y[i][l], workspace=st.ws)

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        one_pass()  # first use of every kernel, outside the capture
    torch.cuda.current_stream().wait_stream(side)
    st.graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(st.graph):
        one_pass()


def _prepare_step(st, sd, layers, vocab, M, group):
    st.table = _weights(sd, vocab, HID, 8, group)  # the embedding and the head share it
    st.w = [[_weights(sd, N, K, 4, group) for N, K in LAYER] for _ in range(layers)]
    st.cache = [[_cache(w, group) if M > 4 else None for w in ws] for ws in st.w]
    st.gamma = [[_gamma(sd(), HID) for _ in range(4)] for _ in range(layers)]
    st.gamma_out = _gamma(sd(), HID)
    g = torch.Generator(device=DEV)
    g.manual_seed(sd())
    st.tokens = torch.randint(0, vocab, (M,), generator=g, device=DEV, dtype=torch.int32)
    st.attn = synth.make_activation(M, HID, seed=sd(), device=DEV)  # stands in for the attention's output
    bf, f32 = torch.bfloat16, torch.float32
    st.emb, st.xn = torch.empty((M, HID), dtype=bf, device=DEV), torch.empty((M, HID), dtype=bf, device=DEV)
    st.qkv = torch.empty((layers, M, QKV), dtype=f32, device=DEV)
    st.h = torch.empty((2 * layers + 1, M, HID), dtype=f32, device=DEV)
    st.proj = torch.empty((M, HID), dtype=f32, device=DEV)
    st.act = torch.empty((M, FF), dtype=bf, device=DEV)
    st.logits = torch.empty((M, vocab), dtype=bf, device=DEV)
    need = [mb.gemm_workspace(M, N, K, DEV) for N, K in LAYER]
    st.ws = max((w for w in need if w is not None), key=lambda w: w.numel(), default=None)


def _prepare_prefill(st, sd, M):
    st.cache = [_cache(_weights(sd, N, K, 4, 64), 64) for N, K in LAYER]
    half = mb.lib.miori_cache_bytes(FF, HID) // 2
    st.w1, st.w3 = st.cache[2][:half], st.cache[2][half:]  # gate rows, then up rows: shards of the cache
    st.gate_w = (0.02 * _normal(sd(), GATE, HID)).to(torch.bfloat16)
    st.gamma = [_gamma(sd(), HID) for _ in range(4)]
    st.h0 = _normal(sd(), M, HID)
    st.attn = synth.make_activation(M, HID, seed=sd(), device=DEV)
    bf = torch.bfloat16
    st.xn = torch.empty((M, HID), dtype=bf, device=DEV)
    st.qkv, st.gates = torch.empty((M, QKV), device=DEV), torch.empty((M, GATE), device=DEV)
    st.proj = torch.empty((M, HID), device=DEV)
    st.h1, st.h2 = torch.empty((M, HID), device=DEV), torch.empty((M, HID), device=DEV)
    st.g, st.u = torch.empty((M, FF), device=DEV), torch.empty((M, FF), device=DEV)
    st.act = torch.empty((M, FF), dtype=bf, device=DEV)
    need = [mb.gemm_workspace(M, N, K, DEV) for N, K in ((QKV, HID), (HID, HID), (FF, HID), (HID, FF))]
    st.ws = max((w for w in need if w is not None), key=lambda w: w.numel(), default=None)


# ---------------------------------------------------------------------------------- one pass

def run(st):
    return _RUN[st.case["kind"]](st, st.case)


def _run_projection(st, c):
    fn = mb.gemv4 if c["bits"] == 4 else mb.gemv8
    return fn(*st.w, st.x, group=c["group"], flags=mb.OUT_BF16 if c["bf16"] else mb.OUT_F32)


def _run_head(st, c):
    mb.gemv8(*st.w, st.x, group=c["group"], flags=mb.LAUNCH_PDL | mb.OUT_BF16, out=st.logits)
    picks = [mb.argmax(st.logits[m], flags=mb.LAUNCH_PDL) for m in range(c["M"])]
    return [st.logits, [i for i, _ in picks], [v for _, v in picks]]


def _run_stack(st, c):
    st.graph.replay()
    return st.y


def _run_step(st, c):
    M, group, pdl = c["M"], c["group"], mb.LAUNCH_PDL
    mb.embed8(*st.table, st.tokens, group=group, out=st.emb)
    st.h[0].copy_(st.emb)
    for l, (wq, wo, wgu, wd) in enumerate(st.w):
        g0, g1, g2, g3 = st.gamma[l]
        h, mid, out, qkv = st.h[2 * l], st.h[2 * l + 1], st.h[2 * l + 2], st.qkv[l]
        cq, co, _, cd = st.cache[l]
        if M <= 4:  # the norms and the activation ride in the projections' launches
            mb.gemv4_rmsnorm(*wq, h, g0, EPS, group=group, flags=pdl, out=qkv)
            mb.gemv4(*wo, st.attn, group=group, flags=pdl, out=st.proj)
            mb.post_norm_add(h, st.proj, g1, EPS, flags=pdl, out=mid)
            mb.gemv4_rmsnorm_silu(*wgu, mid, g2, EPS, group=group, flags=pdl, out=st.act)
            mb.gemv4(*wd, st.act, group=group, flags=pdl, out=st.proj)
        else:
            mb.rmsnorm(h, g0, EPS, flags=pdl, out=st.xn)
            mb.linear4(*wq, cq, st.xn, group=group, flags=pdl, out=qkv, workspace=st.ws)
            mb.linear4(*wo, co, st.attn, group=group, flags=pdl, out=st.proj, workspace=st.ws)
            mb.post_norm_add(h, st.proj, g1, EPS, flags=pdl, out=mid)
            mb.rmsnorm(mid, g2, EPS, flags=pdl, out=st.xn)
            mb.gemv4_silu(*wgu, st.xn, group=group, flags=pdl, out=st.act)
            mb.linear4(*wd, cd, st.act, group=group, flags=pdl, out=st.proj, workspace=st.ws)
        mb.post_norm_add(mid, st.proj, g3, EPS, flags=pdl, out=out)
    mb.rmsnorm(st.h[2 * c["layers"]], st.gamma_out, EPS, flags=pdl, out=st.xn)
    mb.gemv8(*st.table, st.xn, group=group, flags=pdl | mb.OUT_BF16, out=st.logits)
    return [st.h, st.qkv, st.logits]


def _run_cache_build(st, c):
    return (mb.dequant4_cache if c["bits"] == 4 else mb.dequant8_rowmajor)(*st.w, group=c["group"], out=st.out)


def _run_prefill(st, c):
    pdl, ws = mb.LAUNCH_PDL, st.ws
    mb.rmsnorm(st.h0, st.gamma[0], EPS, flags=pdl, out=st.xn)
    mb.gemm_bf16_cache(st.xn, st.cache[0], QKV, flags=pdl, out=st.qkv, workspace=ws)
    mb.gemm_bf16_strided(st.xn, st.gate_w, flags=pdl, out=st.gates)
    mb.gemm_bf16_cache(st.attn, st.cache[1], HID, flags=pdl, out=st.proj, workspace=ws)
    mb.post_norm_add(st.h0, st.proj, st.gamma[1], EPS, flags=pdl, out=st.h1)
    mb.rmsnorm(st.h1, st.gamma[2], EPS, flags=pdl, out=st.xn)
    mb.gemm_bf16_cache(st.xn, st.w1, FF, flags=pdl, out=st.g, workspace=ws)
    mb.gemm_bf16_cache(st.xn, st.w3, FF, flags=pdl, out=st.u, workspace=ws)
    mb.silu_mul(st.g, st.u, flags=pdl, out=st.act)
    mb.gemm_bf16_cache(st.act, st.cache[3], HID, flags=pdl, out=st.proj, workspace=ws)
    mb.post_norm_add(st.h1, st.proj, st.gamma[3], EPS, flags=pdl, out=st.h2)
    return [st.qkv, st.gates, st.h1, st.act, st.h2]


def _run_gemm(st, c):
    return mb.gemm_bf16_cache(st.x, st.cache, c["N"], flags=mb.OUT_BF16 if c["bf16"] else mb.OUT_F32, out=st.y, workspace=st.ws)


_RUN = {"projection": _run_projection, "head": _run_head, "stack": _run_stack, "step": _run_step,
        "cache_build": _run_cache_build, "prefill_layer": _run_prefill, "gemm": _run_gemm}


# ---------------------------------------------------------------------------------- what a pass needs

def _packed(N, K, bits, group):
    return N * K * bits // 8 + N * (K // group) * 4


def work(case):
    kind, M, group = case["kind"], case.get("M", 1), case.get("group", 64)
    if kind in ("projection", "head"):
        N, K = case["N"], case["K"]
        out = 4 if kind == "projection" and not case["bf16"] else 2
        return {"bytes": _packed(N, K, case.get("bits", 8), group) + 2 * M * K + out * M * N, "flops": 2 * M * N * K}
    if kind in ("stack", "step"):
        # activations pass between neighbours of a layer on the chip's own memory; what is returned is written
        by = case["layers"] * sum(_packed(N, K, 4, group) for N, K in LAYER)
        fl = case["layers"] * sum(2 * M * N * K for N, K in LAYER)
        if kind == "stack":
            by += sum(2 * M * K + case["layers"] * 4 * M * N for N, K in LAYER)
        else:
            by += _packed(case["N"], HID, 8, group) + 2 * M * case["N"] + 4 * M * (case["layers"] * (2 * HID + QKV) + HID)
            fl += 2 * M * case["N"] * HID
        return {"bytes": by, "flops": fl}
    if kind == "cache_build":
        return {"bytes": _packed(case["N"], case["K"], case["bits"], group) + 2 * case["N"] * case["K"], "flops": 2 * case["N"] * case["K"]}
    if kind == "prefill_layer":
        weights = sum(2 * N * K for N, K in LAYER) + 2 * GATE * HID
        acts = M * (4 * HID + 2 * HID) + M * (4 * QKV + 4 * GATE + 4 * HID + 2 * FF + 4 * HID)  # read, then written
        return {"bytes": weights + acts, "flops": sum(2 * M * N * K for N, K in LAYER) + 2 * M * GATE * HID}
    N, K = case["N"], case["K"]
    return {"bytes": 2 * N * K + 2 * M * K + (2 if case["bf16"] else 4) * M * N, "flops": 2 * M * N * K}


def tolerance(case):
    kind, M = case["kind"], case.get("M", 1)
    if kind == "cache_build":
        return "exact"
    if kind == "projection":
        # 4-bit batches above four rows may round the weights to bf16, as the cache does
        return {"rel": 5e-3} if case["bf16"] or (case["bits"] == 4 and M > 4) else {"rel": 1e-5, "max": 1e-4}
    if kind == "stack":
        return {"rel": 5e-3} if M > 4 else {"rel": 1e-5, "max": 1e-4}
    if kind == "head":
        return {"rel": 5e-3}  # bf16 logits
    if kind in ("step", "prefill_layer"):
        return {"rel": 1e-2}  # activations rounded to bf16 between the operators
    return {"rel": 5e-3} if case["bf16"] else {"rel": 1e-5, "max": 1e-4}
