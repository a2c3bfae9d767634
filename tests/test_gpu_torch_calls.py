"""The native module behind capi.py's tensor calls, with the library's functions replaced by ones that tell what they saw."""
import ctypes
import subprocess
import threading
import time

import pytest

pytestmark = pytest.mark.gpu

# Stands in for every function of the library: succeeds once another thread has raised the flag, fails after 2 s.
SOURCE = """
#include <time.h>
static volatile int flag;
void set_flag(int v) { flag = v; }
int wait_for_flag() {
    const struct timespec ms = {0, 1000000};
    for (int i = 0; i < 2000; ++i) {
        if (flag) return 0;
        nanosleep(&ms, 0);
    }
    return 99;
}
"""
NAMES = ["jq_quantize_q8_1_device", "jq_mul_mat_q4_0_q8_1_device_ex", "jq_linear_q4_0_device", "jq_linear_q4_0_multi_device",
         "jq_rms_norm_q8_1_device", "jq_swiglu_q8_1_device"]


def _address(f):
    return ctypes.cast(f, ctypes.c_void_p).value


@pytest.fixture(scope="module")
def waiting(native_lib, cuda_device, tmp_path_factory):
    from jjjetson_ops_b200 import _torch_calls

    lib = str(tmp_path_factory.mktemp("waiting") / "libwaiting.so")
    subprocess.run(["gcc", "-std=gnu11", "-shared", "-fPIC", "-x", "c", "-", "-o", lib], input=SOURCE, text=True, check=True)
    w = ctypes.CDLL(lib)
    _torch_calls.bind({n: _address(w.wait_for_flag) for n in NAMES})
    yield w
    _torch_calls.bind({n: _address(getattr(native_lib.lib(), n)) for n in NAMES})


@pytest.mark.parametrize("name", ["quantize", "mul_mat", "linear", "multi", "rms_norm", "swiglu"])
def test_other_threads_run_during_a_call(native_lib, cuda_device, waiting, name):
    """A launch can take long (a full queue, a kernel's first use): Python threads go on meanwhile."""
    import torch

    c, K, N, M = native_lib, 256, 64, 2
    w = torch.zeros(c.q4_0_bytes(N, K), dtype=torch.uint8, device=cuda_device)
    xq = torch.zeros(c.q8_1_bytes(K, M), dtype=torch.uint8, device=cuda_device)
    x, y, v = (torch.zeros(s, device=cuda_device) for s in ((M, K), (M, N), (K,)))
    call = {
        "quantize": lambda: c.quantize_q8_1(x, out=xq),
        "mul_mat": lambda: c.mul_mat_q4_0_q8_1(w, xq, K, N, M, out=y),
        "linear": lambda: c.linear_q4_0(w, x, N, ws=xq, out=y),
        "multi": lambda: c.linear_q4_0_multi([w], [N], xq=xq, K=K, M=M, outs=[y]),
        "rms_norm": lambda: c.rms_norm_q8_1(x, v, 1e-6, xq=xq),
        "swiglu": lambda: c.swiglu_q8_1(x, x, xq=xq),
    }[name]
    waiting.set_flag(0)

    def raise_it():
        time.sleep(0.05)
        waiting.set_flag(1)

    other = threading.Thread(target=raise_it)
    other.start()
    try:
        call()  # JqError (status 99) if the other thread could not run
    finally:
        other.join()
