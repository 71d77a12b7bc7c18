"""Kernels are set up once in every context a thread launches from: in a second one on the same device, and in the first
again afterwards."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = """
import ctypes as C
import torch
import miori_b200 as mb
from miori_b200 import synth
cuda = C.CDLL("libcuda.so.1")
def ok(rc): assert rc == 0, rc
N, K = 2048, 2048
q, s, b = synth.make_weight(N, K, 4, 64, seed=1, device="cuda:0")
x = synth.make_activation(8, K, seed=2, device="cuda:0")
host = [t.cpu().contiguous() for t in (q, s, b, x)]
want = {M: mb.gemv4(q, s, b, x[:M].contiguous(), group=64).cpu() for M in (1, 2, 8)}  # set up here first
ctx, old = C.c_void_p(), C.c_void_p()
ok(cuda.cuCtxCreate_v2(C.byref(ctx), 0, 0))  # and current
dev = []
for t in host:
    p = C.c_uint64()
    ok(cuda.cuMemAlloc_v2(C.byref(p), C.c_size_t(t.numel() * t.element_size())))
    ok(cuda.cuMemcpyHtoD_v2(p, C.c_void_p(t.data_ptr()), C.c_size_t(t.numel() * t.element_size())))
    dev.append(p)
y = C.c_uint64()
ok(cuda.cuMemAlloc_v2(C.byref(y), C.c_size_t(8 * N * 4)))
for M in (1, 2, 8):
    rc = mb.lib.miori_gemv4(*(p.value for p in dev), y.value, N, K, M, 64, 0, None)
    assert rc == 0, mb.lib.miori_last_error()
    got = torch.empty((M, N))
    ok(cuda.cuMemcpyDtoH_v2(C.c_void_p(got.data_ptr()), y, C.c_size_t(M * N * 4)))
    assert torch.equal(got, want[M]), M
for p in dev + [y]:
    ok(cuda.cuMemFree_v2(p))
ok(cuda.cuCtxPopCurrent_v2(C.byref(old)))
for M in (1, 2, 8):
    assert torch.equal(mb.gemv4(q, s, b, x[:M].contiguous(), group=64).cpu(), want[M])
ok(cuda.cuCtxDestroy_v2(ctx))
print("contexts ok")
"""


def test_second_context_on_the_device():
    r = subprocess.run([sys.executable, "-c", PROGRAM], cwd=ROOT, capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and "contexts ok" in r.stdout, r.stdout[-2000:] + r.stderr[-3000:]
