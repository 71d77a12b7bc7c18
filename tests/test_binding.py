"""The operators' native call path: argument handling (no GPU), outputs given and allocated (GPU)."""
import inspect

import pytest
import torch

import miori_b200
from miori_b200 import ops, synth


def test_arguments_are_checked_before_the_library_is_called():
    q = torch.zeros((16, 8), dtype=torch.int32)
    s = torch.zeros((16, 2), dtype=torch.bfloat16)
    x = torch.zeros((1, 64), dtype=torch.bfloat16)
    with pytest.raises(TypeError, match="missing required argument 'x'"):
        ops.gemv4(q, s, s)
    with pytest.raises(TypeError, match="unexpected keyword argument 'grup'"):
        ops.gemv4(q, s, s, x, grup=64)
    with pytest.raises(TypeError, match="multiple values for argument 'q'"):
        ops.gemv4(q, s, s, x, q=q)
    with pytest.raises(TypeError, match="at most 7"):
        ops.gemv4(q, s, s, x, 32, 0, None, 1)
    with pytest.raises(TypeError, match="tensor"):
        ops.gemv4(q, s, s, 3.0)
    assert str(inspect.signature(ops.gemv4)) == "(q, s, b, x, group=32, flags=0, out=None)"


@pytest.mark.parametrize("name", ["rmsnorm", "post_norm_add", "silu_mul", "embed8", "argmax", "dequant4_cache",
                                  "gemm_bf16_cache", "gemm_bf16_strided", "linear4", "gemv4_silu"])
def test_no_operator_takes_cpu_tensors(name):
    t = torch.zeros((16, 64), dtype=torch.bfloat16)
    sig = inspect.signature(getattr(ops, name))
    need = sum(p.default is p.empty for p in sig.parameters.values())
    args = [1e-5 if p == "eps" else 16 if p == "N" else t for p in list(sig.parameters)[:need]]
    with pytest.raises(ValueError, match="no CPU path"):
        getattr(ops, name)(*args)


def _fakes():
    """CUDA tensors without memory."""
    from torch._subclasses import FakeTensorMode
    with FakeTensorMode():
        return {"q": torch.empty((16, 8), dtype=torch.int32, device="cuda"), "s": torch.empty((16, 2), dtype=torch.bfloat16, device="cuda"),
                "x": torch.empty((1, 64), dtype=torch.bfloat16, device="cuda"), "y": torch.empty((1, 16), device="cuda"),
                "strided": torch.empty((4, 32), device="cuda")[:, :16], "f": torch.empty((1, 64), device="cuda")}


def test_tensors_without_storage_raise():
    """Reading such a tensor's pointer throws inside the C function: an exception as from torch's own operators."""
    f = _fakes()
    for call in (lambda: ops.gemv4(f["q"], f["s"], f["s"], f["x"], group=32, out=f["y"]),
                 lambda: ops.gemm_bf16_cache(f["x"], f["x"], 16, out=f["y"]),
                 lambda: ops.gemm_bf16_cache(f["x"], f["x"], 16, out=f["y"], workspace=f["y"]),
                 lambda: ops.silu_mul(f["f"], f["f"], out=f["f"]), lambda: ops.post_norm_add(f["f"], f["f"], f["x"], 1e-5, out=f["f"]),
                 lambda: ops.rmsnorm(f["f"], f["x"], "1e-5", out=f["f"])):
        with pytest.raises(RuntimeError):
            call()
    with pytest.raises(IndexError):
        ops.gemv4(f["q"][0], f["s"], f["s"], f["x"], out=f["y"])


def test_outputs_and_workspaces_are_checked():
    f = _fakes()
    host = torch.zeros((1, 16))
    args = (f["q"], f["s"], f["s"], f["x"])
    with pytest.raises(ValueError, match="out: a CUDA tensor"):
        ops.gemv4(*args, out=host)
    with pytest.raises(ValueError, match="out: a CUDA tensor"):
        ops.gemm_bf16_strided(f["x"], f["x"], out=torch.zeros((1, 1)))
    with pytest.raises(ValueError, match="out: 64 bytes needed, the tensor has 32"):
        ops.gemv4(*args, out=f["y"][:, :8])
    with pytest.raises(ValueError, match="out: a contiguous tensor"):
        ops.gemv4(f["q"], f["s"], f["s"], f["x"].expand(4, 64).clone(), out=f["strided"])
    with pytest.raises(ValueError, match="out: 128 bytes needed"):
        ops.rmsnorm(f["f"], f["x"], 1e-5, out=f["y"])
    with pytest.raises(ValueError, match="workspace: a CUDA tensor"):
        ops.gemm_bf16_cache(f["x"], f["x"], 16, out=f["y"], workspace=host)


@pytest.mark.gpu
def test_out_of_memory_is_torchs():
    A = torch.zeros((64, 64), dtype=torch.bfloat16, device="cuda:0")
    with pytest.raises(torch.OutOfMemoryError):
        ops.gemm_bf16_cache(A, A, 2 ** 32 - 8)  # an output of a terabyte


@pytest.mark.gpu
def test_given_and_allocated_outputs():
    dev = "cuda:0"
    q, s, b = synth.make_weight(48, 256, 4, 64, seed=1, device=dev)
    x = synth.make_activation(3, 256, seed=2, device=dev)
    y = ops.gemv4(q, s, b, x, 64)
    out = torch.empty((3, 48), device=dev)
    assert ops.gemv4(q=q, s=s, b=b, x=x, group=64, out=out) is out
    assert torch.equal(y, out) and y.dtype == torch.float32
    assert ops.gemv4(q, s, b, x[0], group=64).shape == (1, 48)
    assert ops.gemv4(q, s, b, x, group=64, flags=miori_b200.OUT_BF16).dtype == torch.bfloat16
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        z = ops.gemv4(q, s, b, x, group=64)
    side.synchronize()
    assert torch.equal(z, y)
    with pytest.raises(miori_b200.MioriError, match="group must be"):
        ops.gemv4(q, s, b, x, group=48)
    with pytest.raises(ValueError, match="words per row"):
        ops.gemv8(q, s, b, x, group=64)


def test_a_binding_of_another_torch_is_rebuilt(monkeypatch):
    from miori_b200 import build
    assert not build._binding_stale([])
    monkeypatch.setattr(build, "_torch_tag", lambda: "built against torch 0.0;")
    assert build._binding_stale([])
