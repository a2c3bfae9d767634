"""CPU checks of the native module behind capi.py's tensor calls: what it refuses, it refuses with a Python exception."""
import os
import subprocess
import sys

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

# Fake CUDA tensors reach the native argument checks without a GPU.
FAKE = """
import torch
from torch._subclasses.fake_tensor import FakeTensorMode
from jjjetson_ops_b200 import capi as c

def f32(*shape):
    return torch.empty(shape, device="cuda")

def u8(n, *batch):
    return torch.empty(batch + (n,), dtype=torch.uint8, device="cuda")

K, N, M = 256, 64, 2
nw, nq = c.q4_0_bytes(N, K), c.q8_1_bytes(K, M)
"""


def _raised(calls, setup=""):
    """The names of the exceptions that the calls raise, in a process of its own that has to outlive all of them."""
    code = FAKE + setup + "for call in %r:\n    with FakeTensorMode():\n        try:\n            eval(call)\n            print('nothing')\n" \
        "        except Exception as e:\n            print('RuntimeError' if isinstance(e, RuntimeError) else type(e).__name__)\n" % (calls,)
    r = subprocess.run([sys.executable, "-W", "ignore", "-c", code], capture_output=True, text=True, cwd=ROOT, timeout=300)
    assert r.returncode == 0, (r.returncode, r.stdout, r.stderr[-2000:])
    return r.stdout.split()


def test_tensor_without_storage_is_a_runtime_error(native_lib):
    """A tensor whose data pointer torch refuses to give: an exception, not the end of the process."""
    calls = [
        "torch.vmap(lambda v: c.quantize_q8_1(v, out=u8(nq)))(f32(3, M, K))",
        "torch.vmap(lambda v: c.mul_mat_q4_0_q8_1(u8(nw), v, K, N, M, out=f32(M, N)))(u8(nq, 3))",
        "torch.vmap(lambda v: c.linear_q4_0(v, f32(M, K), N, ws=u8(nq), out=f32(M, N)))(u8(nw, 3))",
        "torch.vmap(lambda v: c.linear_q4_0_multi([v], [N], xq=u8(nq), K=K, M=M, outs=[f32(M, N)]))(u8(nw, 3))",
        "torch.vmap(lambda v: c.rms_norm_q8_1(f32(M, K), f32(K), 1e-6, xq=v))(u8(nq, 3))",
        "torch.vmap(lambda v: c.swiglu_q8_1(f32(M, K), v, xq=u8(nq)))(f32(3, M, K))",
    ]
    assert _raised(calls) == ["RuntimeError"] * len(calls)


def test_lists_that_change_during_the_call(native_lib):
    """A row count whose conversion empties the caller's lists: the call works on what the lists held."""
    setup = """
ws_list, N_list, outs = [], [], []

class Rows:
    def __int__(self):
        for l in (ws_list, N_list, outs):
            l.clear()
        return 2**70  # refused, with OverflowError, once the lists are gone

def multi(*rows):
    ws_list[:], N_list[:], outs[:] = [u8(nw) for _ in rows], rows, [f32(M, N) for _ in rows]
    return c.linear_q4_0_multi(ws_list, N_list, xq=u8(nq), K=K, M=M, outs=outs)

class Small(Rows):
    def __int__(self):
        super().__int__()
        return N
"""
    assert _raised(["multi(Rows(), N, N)", "multi(Small(), N, Rows())"], setup) == ["OverflowError"] * 2


def test_refused_arguments(native_lib):
    """Wrong type, layout, device, dimensions or counts: ValueError, as before the calls were native."""
    calls = [
        "c.quantize_q8_1(f32(M, K).half(), out=u8(nq))",
        "c.quantize_q8_1(f32(K, M).t(), out=u8(nq))",
        "c.quantize_q8_1(f32(M, K), out=f32(nq))",
        "c.quantize_q8_1(f32(1, M, K), out=u8(nq))",
        "c.mul_mat_q4_0_q8_1(f32(nw), u8(nq), K, N, M, out=f32(M, N))",
        "c.mul_mat_q4_0_q8_1(u8(nw), u8(nq).cpu(), K, N, M, out=f32(M, N))",
        "c.mul_mat_q4_0_q8_1(u8(nw), u8(nq), K, N, M, out=f32(M, 2 * N)[:, ::2])",
        "c.linear_q4_0(u8(nw), f32(M * K), N, ws=u8(nq), out=f32(M, N))",
        "c.linear_q4_0(None, f32(M, K), N, ws=u8(nq), out=f32(M, N))",
        "c.linear_q4_0_multi([u8(nw)], [N, N], xq=u8(nq), K=K, M=M, outs=[f32(M, N)])",
        "c.linear_q4_0_multi([u8(nw)] * 17, [N] * 17, xq=u8(nq), K=K, M=M, outs=[f32(M, N)] * 17)",
        "c.rms_norm_q8_1(f32(M, K), f32(K), 1e-6, xq=[0])",
        "c.rms_norm_q8_1(f32(M, K), f32(K).double(), 1e-6, xq=u8(nq))",
        "c.swiglu_q8_1(f32(M, K), f32(K, M).t(), xq=u8(nq))",
    ]
    assert _raised(calls) == ["ValueError"] * len(calls)
