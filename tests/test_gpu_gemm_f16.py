"""GPU parity of the fp16-operand tcgen05 GEMM (JQ_KERNEL_GEMM_F16), called through the C ABI.

This kernel rounds every scaled operand ((q4 - 8) * d4 and q8 * d8) to fp16 before the tensor core
multiplies them with fp32 accumulation, so its bar is not the integer kernels' 1e-5: it is
max|y - ref| / max|ref| <= 1e-3 against the oracle's reference-formula multiply on the same
quantized inputs (about 3e-4 is expected) and <= 1e-3 against dequantise-then-matmul in float64
when the quantizer stored s = d * sum(q).
"""
import subprocess
import sys

import numpy as np
import pytest

from launch_forms import ROOT, gemm_f16_form

pytestmark = pytest.mark.gpu

TOL_F16_FORMULA = 1e-3  # operands rounded to fp16 (2^-11 relative each), fp32 accumulation
TOL_DEQUANT = 1e-3      # the accuracy target against dequantise-then-matmul


@pytest.fixture(scope="module")
def env(native_lib, oracle, cuda_device):
    import torch

    class Env:
        c = native_lib
        O = oracle
        dev = cuda_device
        t = torch

        def up(self, a):
            return torch.from_numpy(np.ascontiguousarray(a)).to(cuda_device)

    e = Env()
    yield e
    assert native_lib.device_fault(clear=True) == 0  # no kernel gave up on a bounded wait


def _check(env, wq, x, K, N, M, order, s_mode, rows=None):
    c = env.c
    xq = env.O.quantize_q8_1(x, order, s_mode)
    y = c.mul_mat_q4_0_q8_1(env.up(wq), env.up(xq), K, N, M, order, c.KERNEL_GEMM_F16).cpu().numpy()
    assert y.shape == (M, N) and np.isfinite(y).all()
    if rows is not None:
        wq = np.ascontiguousarray(wq.reshape(N, -1)[rows])
        y = y[:, rows]
        N = len(rows)
    e_ref = env.O.err_max_rel(y, env.O.mul_mat_ref(wq, xq, K, N, M, order))
    assert e_ref <= TOL_F16_FORMULA, e_ref
    if s_mode == c.S_D_SUM_Q:
        e_deq = env.O.err_max_rel(y, env.O.mul_mat_deq_f64(wq, xq, K, N, M, order))
        assert e_deq <= TOL_DEQUANT, e_deq
    return e_ref


@pytest.mark.parametrize("K,N,M", [(2560, 40, 20), (256, 64, 9), (512, 200, 33), (1024, 129, 130), (768, 256, 128),
                                   (4096, 384, 17), (1280, 1, 1), (11008, 50, 40), (1792, 300, 257)])
@pytest.mark.parametrize("order", [0, 1])
@pytest.mark.parametrize("s_mode", [0, 1])
def test_gemm_f16_small_and_ragged_shapes(env, K, N, M, order, s_mode):
    rng = np.random.default_rng(K + 3 * N + 7 * M)
    w = (rng.standard_normal((N, K), dtype=np.float32) * np.float32(0.02)).astype(np.float32)
    x = rng.standard_normal((M, K), dtype=np.float32)
    if K >= 256:
        x[:, 5] *= 20.0          # an outlier channel
        x[M // 2, 128:160] = 0.0  # an all-zero group: d = 0
    _check(env, env.O.quantize_q4_0(w), x, K, N, M, order, s_mode)


def test_gemm_f16_refuses_odd_super_block_counts(env):
    """The tensor copies need a weight-row pitch that is a multiple of 16 bytes: K % 256 == 0."""
    c = env.c
    w = env.t.zeros(c.q4_0_bytes(8, 384), dtype=env.t.uint8, device=env.dev)
    xq = env.t.zeros(c.q8_1_bytes(384, 16), dtype=env.t.uint8, device=env.dev)
    with pytest.raises(c.JqError) as ei:
        c.mul_mat_q4_0_q8_1(w, xq, 384, 8, 16, c.ORDER_COL_KSUPER, c.KERNEL_GEMM_F16)
    assert ei.value.status == c.ERR_UNSUPPORTED


def test_gemm_f16_prefill_config(env):
    """K = N = 4096, M = 512: the prefill configuration, oracle on a sample of the weight rows."""
    from jjjetson_ops_b200 import synth

    c = env.c
    w, x, lin = synth.make_linear_case(3, 0, 512)
    wq = c.quantize_q4_0(env.up(w)).cpu().numpy()
    rows = np.sort(np.random.default_rng(33).choice(lin.N, size=256, replace=False))
    for order in (c.ORDER_COL_KSUPER, c.ORDER_KSUPER_COL):
        _check(env, wq, x, lin.K, lin.N, 512, order, c.S_D_SUM_Q, rows=rows)


def test_gemm_f16_matches_integer_kernel_closely(env):
    """Same inputs through the integer GEMM and the fp16-operand GEMM: they differ only by the
    operand rounding."""
    c = env.c
    rng = np.random.default_rng(91)
    K, N, M = 2048, 512, 256
    w = (rng.standard_normal((N, K), dtype=np.float32) * np.float32(0.02)).astype(np.float32)
    x = rng.standard_normal((M, K), dtype=np.float32)
    d_w = env.up(env.O.quantize_q4_0(w))
    d_xq = env.up(env.O.quantize_q8_1(x, c.ORDER_COL_KSUPER, c.S_D_SUM_Q))
    y_int = c.mul_mat_q4_0_q8_1(d_w, d_xq, K, N, M, c.ORDER_COL_KSUPER, c.KERNEL_GEMM_MMA).cpu().numpy()
    y_f16 = c.mul_mat_q4_0_q8_1(d_w, d_xq, K, N, M, c.ORDER_COL_KSUPER, c.KERNEL_GEMM_F16).cpu().numpy()
    assert env.O.err_max_rel(y_f16, y_int) <= TOL_F16_FORMULA


# More tiles than SMs, so that pairs of CTAs share 256 x 256 tiles: the last pair's second CTA without rows (18690 = 73 * 256
# + 2) or with one, its columns a few or all but one; one stage pair, and more stages than the ring holds.  With 300 tiles on 148
# SMs and a short K single CTAs are as quick: several waves of those.
@pytest.mark.parametrize("K,N,M,form", [(256, 18690, 130, "pair"), (768, 18690, 255, "pair"), (1280, 18817, 256, "pair"), (512, 8960, 400, "pair"),
                                        (512, 9473, 400, 1)])
@pytest.mark.parametrize("order", [0, 1])
def test_gemm_f16_pairs_of_ctas(env, K, N, M, form, order):
    assert gemm_f16_form(K, [N], M) == form
    rng = np.random.default_rng(K + N + M + order)
    w = (rng.standard_normal((N, K), dtype=np.float32) * np.float32(0.02)).astype(np.float32)
    x = rng.standard_normal((M, K), dtype=np.float32)
    rows = np.unique(np.concatenate([rng.choice(N, size=96, replace=False), [0, 127, 128, 255, 256, N - 2, N - 1]]))
    _check(env, env.O.quantize_q4_0(w), x, K, N, M, order, env.c.S_SUM_X, rows)


# K in one to eight parts, equal and with a shorter last one, added up over shared memory by the CTAs of a cluster
@pytest.mark.parametrize("K,N,M,parts", [(512, 130, 64, 1), (768, 200, 66, 1), (2048, 4096, 200, 2), (2304, 4096, 256, 2), (2304, 300, 65, 3),
                                         (1024, 129, 200, 4), (2048, 257, 9, 4), (1536, 1, 130, 6), (2816, 300, 65, 6), (4096, 300, 65, 8)])
def test_gemm_f16_parts_of_k(env, K, N, M, parts):
    assert gemm_f16_form(K, [N], M) == parts
    rng = np.random.default_rng(K + N + M)
    w = (rng.standard_normal((N, K), dtype=np.float32) * np.float32(0.02)).astype(np.float32)
    rows = None if N <= 300 else np.unique(np.concatenate([rng.choice(N, size=96, replace=False), [0, 127, 128, N - 1]]))
    _check(env, env.O.quantize_q4_0(w), rng.standard_normal((M, K), dtype=np.float32), K, N, M, env.c.ORDER_KSUPER_COL, env.c.S_SUM_X, rows)


def test_gemm_f16_parts_of_k_on_two_streams(env):
    """Launches that split K on two streams at once: each keeps its parts to itself."""
    c, t = env.c, env.t
    g = t.Generator(device=env.dev)
    g.manual_seed(12)
    problems = []
    for K, N, M in [(4096, 2048, 100), (2048, 1003, 70)]:
        assert gemm_f16_form(K, [N], M) > 1
        w = c.quantize_q4_0(t.randn((N, K), generator=g, device=env.dev).mul_(0.02))
        xqs = [c.quantize_q8_1(t.randn((M, K), generator=g, device=env.dev)) for _ in range(8)]
        want = [c.mul_mat_q4_0_q8_1(w, xq, K, N, M, kernel=c.KERNEL_GEMM_F16) for xq in xqs]
        problems.append((K, N, M, w, xqs, want, [t.empty_like(y) for y in want], t.cuda.Stream(env.dev)))
    t.cuda.synchronize()
    for i in range(8):
        for K, N, M, w, xqs, _, got, stream in problems:
            with t.cuda.stream(stream):
                c.mul_mat_q4_0_q8_1(w, xqs[i], K, N, M, kernel=c.KERNEL_GEMM_F16, out=got[i])
    t.cuda.synchronize()
    for p in problems:
        assert all(t.equal(a, b) for a, b in zip(p[5], p[6]))


@pytest.mark.parametrize("K,rows,M,form", [(512, [300, 1, 128, 257], 64, 1), (256, [9400, 9290], 130, "pair"), (4096, [128, 200], 100, 8),
                                           (4096, [1024, 1024, 1024], 128, 4)])
def test_gemm_f16_several_matrices(env, K, rows, M, form):
    """Several matrices in one launch (single CTAs, pairs, split K): each row against separate calls, whose sums over K may
    be split elsewhere (fp32 additions in another order)."""
    assert gemm_f16_form(K, rows, M) == form
    c = env.c
    rng = np.random.default_rng(K + M)
    ws = [c.quantize_q4_0(env.up((rng.standard_normal((n, K), dtype=np.float32) * np.float32(0.02)))) for n in rows]
    xq = c.quantize_q8_1(env.up(rng.standard_normal((M, K), dtype=np.float32)), c.ORDER_COL_KSUPER, c.S_D_SUM_Q)
    outs = c.linear_q4_0_multi(ws, rows, xq=xq, K=K, M=M)
    for w, n, y in zip(ws, rows, outs):
        want = c.mul_mat_q4_0_q8_1(w, xq, K, n, M, c.ORDER_COL_KSUPER, c.KERNEL_GEMM_F16)
        assert env.O.err_max_rel(y.cpu().numpy(), want.cpu().numpy()) <= 1e-5


@pytest.mark.parametrize("K,N,M", [(4096, 4096, 128), (11008, 4096, 128), (8192, 300, 70), (2048, 1000, 64)])
def test_gemm_f16_split_k_is_ordered(env, K, N, M):
    """Few output tiles and a long K: the kernel splits K over the CTAs of a cluster, which add up their parts in a
    fixed order.  Right against the oracle (a sample of rows at the large sizes), and bit-equal from run to run."""
    c = env.c
    rng = np.random.default_rng(K + N + M)
    w = (rng.standard_normal((N, K), dtype=np.float32) * np.float32(0.02)).astype(np.float32)
    x = rng.standard_normal((M, K), dtype=np.float32)
    wq = env.O.quantize_q4_0(w)
    rows = None if N <= 1000 else np.sort(rng.choice(N, size=96, replace=False))
    _check(env, wq, x, K, N, M, c.ORDER_COL_KSUPER, c.S_D_SUM_Q, rows)
    xq = env.up(env.O.quantize_q8_1(x, c.ORDER_COL_KSUPER, c.S_D_SUM_Q))
    d_w = env.up(wq)
    runs = [c.mul_mat_q4_0_q8_1(d_w, xq, K, N, M, c.ORDER_COL_KSUPER, c.KERNEL_GEMM_F16).cpu().numpy() for _ in range(4)]
    for y in runs[1:]:
        assert np.array_equal(y, runs[0])
    exact = c.mul_mat_q4_0_q8_1(d_w, xq, K, N, M, c.ORDER_COL_KSUPER, c.KERNEL_GEMM_MMA).cpu().numpy()
    assert env.O.err_max_rel(runs[0], exact) <= TOL_F16_FORMULA


FIRST_CALL = """
import torch
from jjjetson_ops_b200 import capi as c
dev = torch.device("cuda:0")
g = torch.Generator(device=dev)
g.manual_seed(3)
for K, N, M in [(2048, 2048, 128), (256, 18690, 130)]:
    w = c.quantize_q4_0(torch.randn((N, K), generator=g, device=dev) * 0.02)
    xq = c.quantize_q8_1(torch.randn((M, K), generator=g, device=dev))
    y = torch.zeros((M, N), device=dev)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        c.mul_mat_q4_0_q8_1(w, xq, K, N, M, out=y)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, c.mul_mat_q4_0_q8_1(w, xq, K, N, M)), (K, N, M)
print("captured")
"""


def test_gemm_f16_first_call_in_a_capture(env):
    """A process whose first use of the kernel is recorded into a graph: the form is the one of an eager call, bit for bit."""
    assert gemm_f16_form(2048, [2048], 128) == 4 and gemm_f16_form(256, [18690], 130) == "pair"
    r = subprocess.run([sys.executable, "-c", FIRST_CALL], capture_output=True, text=True, cwd=ROOT, timeout=300)
    assert r.returncode == 0 and "captured" in r.stdout, r.stderr[-2000:]


@pytest.mark.parametrize("K,rows,M", [(4096, [4096], 512), (4096, [1024], 64), (8192, [8192], 1024), (1024, [512, 128, 128], 100)])
def test_trace_stamps_of_a_launch_are_ordered(env, K, rows, M):
    """jq_trace_enable: single CTAs, a split K, pairs, several matrices.  Each of the first stages has its stamps in order, and the next
    launch none."""
    c, t = env.c, env.t
    x = t.randn((M, K), device=env.dev)
    ws = [c.quantize_q4_0(t.randn((n, K), device=env.dev)) for n in rows]
    want = c.linear_q4_0_multi(ws, rows, x=x)
    xq = c.quantize_q8_1(x, c.ORDER_COL_KSUPER, c.S_D_SUM_Q)
    buf = t.zeros((2, 512, 8), dtype=t.int64, device=env.dev)
    t.cuda.synchronize()
    c.check(c.lib().jq_trace_enable(buf.data_ptr(), 1))
    got = [c.linear_q4_0_multi(ws, rows, xq=xq, K=K, M=M) for _ in range(2)]
    c.check(c.lib().jq_trace_enable(None, 0))
    t.cuda.synchronize()
    assert all(t.equal(a, b) for g in got for a, b in zip(g, want))
    stamps = buf.cpu().numpy()
    assert not stamps[1].any()
    weights, activations, mma = stamps[0, :64], stamps[0, 64:128], stamps[0, 128:192]
    n = int((mma[:, 0] != 0).sum())  # the first CTA's stages
    assert n >= 2 and (mma[:n, :2] != 0).all() and (np.diff(mma[:n, :2].reshape(-1)) >= 0).all()
    for who in (weights, activations):
        own = [i for i in range(64) if who[i].any()]
        assert own == list(range(0, n, 3))
        assert (np.diff(who[own][:, [0, 1, 3, 4, 5]].reshape(-1)) >= 0).all() and (who[own, 4] <= mma[own, 0]).all()  # converted before it is seen
