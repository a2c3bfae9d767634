"""GPU parity of the small-batch multiply, which the automatic choice takes for 3 to 63 columns (where the decode kernels
refuse the shape) and for any batch when K is an odd multiple of 128.

The bar against the oracle's reference-formula multiply is the integer kernels' 1e-5: block sums are exact, only the
order of the fp32 additions differs (K / 32 <= 344 terms of relative rounding 2^-24 each, 2.1e-5 at the very worst and
a few 1e-7 as a rule).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-5


@pytest.fixture(scope="module")
def env(native_lib, oracle, cuda_device):
    import torch

    class Env:
        c, O, t, dev = native_lib, oracle, torch, cuda_device

    yield Env()
    assert native_lib.device_fault(clear=True) == 0


def _problem(K, N, M):
    rng = np.random.default_rng(5 * K + 3 * N + M)
    w = (rng.standard_normal((N, K), dtype=np.float32) * np.float32(0.02)).astype(np.float32)
    return w, rng.standard_normal((M, K), dtype=np.float32)


# Row tiles of 32 and (from 17 columns on, with enough of them) 64, column tiles of 8 to 32 in equal groups, stages of 512
# or 256 values with a shorter last one; more stages than the ring holds; an odd K with every remainder of four.
@pytest.mark.parametrize("K,N,M", [(128, 1, 1), (128, 31, 3), (384, 33, 9), (640, 32, 33), (1408, 65, 45), (896, 100, 130), (4224, 20, 2),
                                   (256, 31, 9), (512, 33, 16), (768, 64, 17), (6400, 40, 8), (6400, 10, 3), (4608, 97, 32),
                                   (256, 9500, 24), (512, 4800, 63), (1280, 9473, 31), (11008, 35, 63)])
@pytest.mark.parametrize("order", [0, 1])
def test_small_batch_shapes(env, K, N, M, order):
    c, O = env.c, env.O
    w, x = _problem(K, N, M)
    wq = O.quantize_q4_0(w)
    xq = O.quantize_q8_1(x, order, c.S_SUM_X)
    d_w, d_x = env.t.from_numpy(wq).to(env.dev), env.t.from_numpy(xq).to(env.dev)
    y = env.t.full((M, N), float("nan"), device=env.dev)
    c.mul_mat_q4_0_q8_1(d_w, d_x, K, N, M, order, out=y)
    assert O.err_max_rel(y.cpu().numpy(), O.mul_mat_ref(wq, xq, K, N, M, order)) <= TOL


@pytest.mark.parametrize("K", [512, 640])
@pytest.mark.parametrize("shift", [2, 8])
def test_small_batch_weights_off_alignment(env, K, shift):
    """Weights that are not 16-byte aligned go to another kernel: same answer."""
    c, O = env.c, env.O
    N, M = 70, 20
    w, x = _problem(K, N, M)
    wq = O.quantize_q4_0(w)
    xq = O.quantize_q8_1(x, O.ORDER_COL_KSUPER, c.S_SUM_X)
    buf = env.t.zeros(wq.nbytes + 16, dtype=env.t.uint8, device=env.dev)
    d_w = buf[shift:shift + wq.nbytes]
    d_w.copy_(env.t.from_numpy(wq.reshape(-1)))
    y = c.mul_mat_q4_0_q8_1(d_w, env.t.from_numpy(xq).to(env.dev), K, N, M)
    assert O.err_max_rel(y.cpu().numpy(), O.mul_mat_ref(wq, xq, K, N, M)) <= TOL


@pytest.mark.parametrize("K,M", [(512, 12), (6400, 5), (640, 7), (512, 40)])
def test_small_batch_several_matrices(env, K, M):
    """Several matrices in one launch give the bits of separate calls."""
    c, O = env.c, env.O
    rows = [40, 1, 96, 33]
    x = _problem(K, 1, M)[1]
    ws = [env.t.from_numpy(O.quantize_q4_0(_problem(K, n, M + i)[0])).to(env.dev) for i, n in enumerate(rows)]
    xq = env.t.from_numpy(O.quantize_q8_1(x, O.ORDER_COL_KSUPER, c.S_D_SUM_Q)).to(env.dev)
    outs = c.linear_q4_0_multi(ws, rows, xq=xq, K=K, M=M)
    for w, n, y in zip(ws, rows, outs):
        assert env.t.equal(y, c.mul_mat_q4_0_q8_1(w, xq, K, n, M))


@pytest.mark.parametrize("K,N,M,generic", [(8320, 756, 1, True), (8320, 757, 1, False), (10880, 31, 1, True), (8320, 64, 2, False),
                                           (8064, 64, 1, False), (10752, 64, 1, False)])
def test_one_column_of_a_long_odd_k(env, K, N, M, generic):
    """Which side of its line a shape is on shows in the bits: the kernels add in different orders."""
    c, O = env.c, env.O
    w, x = _problem(K, N, M)
    wq = O.quantize_q4_0(w)
    xq = O.quantize_q8_1(x, O.ORDER_COL_KSUPER, c.S_SUM_X)
    d_w, d_x = env.t.from_numpy(wq).to(env.dev), env.t.from_numpy(xq).to(env.dev)
    y = c.mul_mat_q4_0_q8_1(d_w, d_x, K, N, M)
    assert O.err_max_rel(y.cpu().numpy(), O.mul_mat_ref(wq, xq, K, N, M)) <= TOL
    assert env.t.equal(y, c.mul_mat_q4_0_q8_1(d_w, d_x, K, N, M, kernel=c.KERNEL_GENERIC)) == generic


def _error_against_64_bits(t, w, xq, y, K, rows):
    """2-norm of the difference over 2-norm of sum(d4 * (sumi * d8 - 8 * s8)) in 64 bits, over some weight rows."""
    M = y.shape[0]
    wb = w.view(-1, K // 32, 18)[rows]
    d4 = wb[:, :, :2].contiguous().view(t.float16).view(len(rows), K // 32).double()
    q4 = t.cat([wb[:, :, 2:] & 15, wb[:, :, 2:] >> 4], dim=2).double()
    xb = xq.view(M, K // 128, 144)
    ds = xb[:, :, :16].contiguous().view(t.float16).view(M, K // 32, 2).double()
    q8 = xb[:, :, 16:].contiguous().view(t.int8).view(M, K // 32, 32).double()
    want = (q8 * ds[:, :, :1]).reshape(M, K) @ (q4 * d4[:, :, None]).reshape(len(rows), K).T - 8.0 * ds[:, :, 1] @ d4.T
    return float((y[:, rows].double() - want).norm() / want.norm())


# Odd K: 32 and 64 rows per CTA, a CTA alone on its SM; running sums in one level and in two; parts as a tree and compensated.
@pytest.mark.parametrize("K,N,M", [(4224, 9600, 24), (4224, 4800, 32), (2688, 9600, 63), (1408, 600, 9), (1408, 9600, 45), (4224, 9600, 4),
                                   (4224, 600, 16), (1920, 9600, 31), (640, 4900, 5)])
def test_small_batch_is_as_exact_as_the_generic_kernel(env, K, N, M):
    """Odd multiples of 128, which the generic kernel took before: the sums over K round off no more than its 32 lanes do.  An
    eighth for the spread of the measure: at least 600 rows x 4 columns, whose squares' mean is known to some 5 %."""
    c, t = env.c, env.t
    g = t.Generator(device=env.dev)
    g.manual_seed(K + N + M)
    w = c.quantize_q4_0(t.randn((N, K), generator=g, device=env.dev).mul_(0.02))
    xq = c.quantize_q8_1(t.randn((M, K), generator=g, device=env.dev), s_mode=c.S_D_SUM_Q)
    rows = t.randperm(N, generator=g, device=env.dev)[:600]
    y = c.mul_mat_q4_0_q8_1(w, xq, K, N, M)
    before = c.mul_mat_q4_0_q8_1(w, xq, K, N, M, kernel=c.KERNEL_GENERIC)
    assert _error_against_64_bits(t, w, xq, y, K, rows) <= 1.125 * _error_against_64_bits(t, w, xq, before, K, rows)


@pytest.mark.parametrize("K,N,M", [(4224, 4800, 45), (8192, 9600, 24), (11008, 600, 8)])
def test_small_batch_wait_that_runs_out(env, K, N, M):
    """Waits of one poll: the kernel gives up, after its copies have landed, and says so (unless every copy was quick enough);
    launches right behind it on the same SMs are not disturbed."""
    c, O, t = env.c, env.O, env.t
    w, x = _problem(K, N, M)
    wq = O.quantize_q4_0(w)
    xq = O.quantize_q8_1(x, O.ORDER_COL_KSUPER, c.S_SUM_X)
    d_w, d_x = t.from_numpy(wq).to(env.dev), t.from_numpy(xq).to(env.dev)
    right = c.mul_mat_q4_0_q8_1(d_w, d_x, K, N, M)
    assert O.err_max_rel(right[:, :64].cpu().numpy(), O.mul_mat_ref(wq[:64], xq, K, 64, M)) <= TOL
    small = [c.quantize_q4_0(t.randn((256, 512), device=env.dev)), c.quantize_q8_1(t.randn((4, 512), device=env.dev))]
    small_right = c.mul_mat_q4_0_q8_1(*small, 512, 256, 4)
    t.cuda.synchronize()
    for _ in range(8):
        c.set_option(c.OPT_WAIT_POLL_LIMIT, 1)
        try:
            y = c.mul_mat_q4_0_q8_1(d_w, d_x, K, N, M)
        finally:
            c.set_option(c.OPT_WAIT_POLL_LIMIT, 0)
        after = [c.mul_mat_q4_0_q8_1(*small, 512, 256, 4), c.mul_mat_q4_0_q8_1(d_w, d_x, K, N, M)]
        t.cuda.synchronize()
        fault = c.device_fault(clear=True)
        assert fault == 1 or (fault == 0 and t.equal(y, right))
        assert t.equal(after[0], small_right) and t.equal(after[1], right)
