"""GPU parity of the small-batch multiply, which the automatic choice takes for 3 to 63 columns (where the decode kernels
refuse the shape) and for any batch when K is an odd multiple of 128.

The bar against the oracle's reference-formula multiply is the integer kernels' 1e-5: block sums are exact, only the
order of the fp32 additions differs (K / 32 <= 344 terms of relative rounding 2^-24 each, 2.1e-5 at the very worst and
a few 1e-7 as a rule).
"""
import numpy as np
import pytest

from launch_forms import small_batch_form, small_batch_tile

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


# Row tiles of 32 (one CTA per SM, sixteen warps along K) and (from 17 columns on, with enough of them) 64, column tiles of 8 to 32
# in equal groups, stages of 1024 or 256 values with a shorter last one; an odd K with every remainder of eight.
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


# The other forms: eight warps, two CTAs per SM, with 32 and 64 rows each, at even and odd K; a ring that goes round several times.
@pytest.mark.parametrize("K,N,M,form", [
    (640, 4900, 5, (True, 1, 32, False)), (1408, 4801, 16, (True, 2, 32, False)), (2688, 9473, 20, (True, 3, 32, False)),
    (1152, 4740, 30, (True, 4, 32, False)), (384, 9473, 24, (True, 3, 64, False)), (1152, 9473, 31, (True, 4, 64, False)),
    (6400, 4900, 8, (False, 1, 32, False)), (512, 5000, 12, (False, 2, 32, False)), (512, 5000, 24, (False, 3, 32, False)),
    (3072, 4740, 30, (False, 4, 32, False)), (4096, 9473, 24, (False, 3, 64, False)), (4352, 9473, 31, (False, 4, 64, False))])
@pytest.mark.parametrize("order", [0, 1])
def test_small_batch_two_ctas_per_sm(env, K, N, M, form, order):
    assert small_batch_form(K, [N], M) == form
    c, O = env.c, env.O
    w, x = _problem(K, N, M)
    d_w = c.quantize_q4_0(env.t.from_numpy(w).to(env.dev))
    wq = d_w.cpu().numpy().reshape(N, -1)
    rows = np.unique(np.concatenate([np.random.default_rng(N).choice(N, size=120, replace=False), [0, 31, 32, 63, 64, N - 2, N - 1]]))
    xq = O.quantize_q8_1(x, order, c.S_SUM_X)
    y = env.t.full((M, N), float("nan"), device=env.dev)
    c.mul_mat_q4_0_q8_1(d_w, env.t.from_numpy(xq).to(env.dev), K, N, M, order, out=y)
    assert not env.t.isnan(y).any()
    assert O.err_max_rel(y.cpu().numpy()[:, rows], O.mul_mat_ref(np.ascontiguousarray(wq[rows]), xq, K, len(rows), M, order)) <= TOL


# One CTA per SM with 64, 96 and 128 rows, at the ends of what makes one wave; all columns of 33 to 63 in one; two and three CTAs per SM.
@pytest.mark.parametrize("K,N,M,tile", [
    (6400, 9472, 8, (64, 1, 16, 1)), (512, 5185, 16, (64, 2, 16, 1)), (1280, 9408, 17, (64, 3, 16, 1)), (4096, 4672, 64, (64, 4, 16, 1)),
    (512, 5184, 16, (32, 2, 8, 2)), (512, 4672, 64, (32, 4, 8, 2)), (1280, 4800, 17, (32, 3, 8, 2)),
    (6400, 9473, 3, (96, 1, 24, 1)), (768, 14208, 9, (96, 2, 24, 1)), (6400, 14209, 8, (32, 1, 8, 2)), (1280, 18944, 16, (32, 2, 8, 2)),
    (6400, 18945, 8, (32, 1, 8, 3)), (1280, 18945, 16, (32, 2, 8, 3)),
    (512, 9472, 24, (64, 3, 8, 2)), (512, 9473, 24, (96, 3, 12, 1)), (1024, 14208, 31, (96, 4, 12, 1)), (512, 14209, 17, (128, 3, 16, 1)),
    (2304, 18944, 32, (128, 4, 16, 1)), (256, 18945, 24, (64, 3, 8, 2)), (512, 18945, 27, (64, 4, 8, 2)), (512, 7104, 33, (96, 3, 12, 1)),
    (512, 9473, 33, (96, 5, 12, 1)), (4096, 14208, 48, (96, 6, 12, 1)), (512, 9480, 49, (96, 7, 12, 1)), (1280, 14145, 63, (96, 8, 12, 1)),
    (512, 14209, 40, (128, 5, 16, 1)), (2304, 18944, 41, (128, 6, 16, 1)), (512, 14209, 49, (64, 4, 8, 2)), (256, 18945, 40, (64, 3, 8, 2))])
@pytest.mark.parametrize("order", [0, 1])
def test_small_batch_tiles(env, K, N, M, tile, order):
    assert small_batch_tile(K, [N], M) == tile
    c, O = env.c, env.O
    w, x = _problem(K, N, M)
    d_w = c.quantize_q4_0(env.t.from_numpy(w).to(env.dev))
    wq = d_w.cpu().numpy().reshape(N, -1)
    last = N // tile[0] * tile[0]
    rows = np.unique(np.concatenate([np.random.default_rng(N).choice(N, size=120, replace=False),
                                     [0, 31, 32, tile[0] - 1, tile[0], last - 1, min(last, N - 1), N - 2, N - 1]]))
    xq = O.quantize_q8_1(x, order, c.S_SUM_X)
    y = env.t.full((M, N), float("nan"), device=env.dev)
    c.set_option(c.OPT_PREFILL_EXACT, 1)  # 64 columns
    try:
        c.mul_mat_q4_0_q8_1(d_w, env.t.from_numpy(xq).to(env.dev), K, N, M, order, out=y)
    finally:
        c.set_option(c.OPT_PREFILL_EXACT, 0)
    assert not env.t.isnan(y).any()
    assert O.err_max_rel(y.cpu().numpy()[:, rows], O.mul_mat_ref(np.ascontiguousarray(wq[rows]), xq, K, len(rows), M, order)) <= TOL


# With JQ_OPT_PREFILL_EXACT, both sides of the lines between this kernel and the integer GEMM: 280 tiles of 128 x 128, K / 4 of them, one wave
# here (296 tiles of 64 x 32), and the estimates beyond
@pytest.mark.parametrize("K,N,M,here", [(2048, 17920, 140, True), (2048, 17921, 140, False), (256, 8192, 64, True), (256, 8193, 64, False),
                                        (256, 1216, 479, True), (256, 1217, 479, False), (1024, 2304, 950, False), (1024, 2305, 950, True),
                                        (1024, 3776, 950, True), (1024, 3777, 950, False), (512, 130, 64, True), (1280, 333, 77, True)])
def test_exact_prefill_kernel(env, K, N, M, here):
    c, O, t = env.c, env.O, env.t
    g = t.Generator(device=env.dev)
    g.manual_seed(K + N + M)
    w = c.quantize_q4_0(t.randn((N, K), generator=g, device=env.dev).mul_(0.02))
    xq = c.quantize_q8_1(t.randn((M, K), generator=g, device=env.dev), s_mode=c.S_D_SUM_Q)
    c.set_option(c.OPT_PREFILL_EXACT, 1)
    try:
        y = c.mul_mat_q4_0_q8_1(w, xq, K, N, M)
    finally:
        c.set_option(c.OPT_PREFILL_EXACT, 0)
    gemm = c.mul_mat_q4_0_q8_1(w, xq, K, N, M, kernel=c.KERNEL_GEMM_MMA)
    assert t.equal(y, gemm) != here and O.err_max_rel(y.cpu().numpy(), gemm.cpu().numpy()) <= TOL
    rows = t.randperm(N, generator=g, device=env.dev)[:600]
    assert _error_against_64_bits(t, w, xq, y, K, rows) <= 1.125 * _error_against_64_bits(t, w, xq, gemm, K, rows)


@pytest.mark.parametrize("K,rows,M,same_form", [(512, [40, 1, 96, 33], 12, True), (6400, [40, 1, 96, 33], 5, True), (640, [40, 1, 96, 33], 7, True),
                                                (512, [40, 1, 96, 33], 40, True), (4096, [2000, 2000, 2000], 16, False),
                                                (4096, [4096, 4096, 4096], 20, False), (1408, [4096, 64], 45, False)])
def test_small_batch_several_matrices(env, K, rows, M, same_form):
    """Several matrices in one launch against separate calls: the same bits where both are divided in the same way.  Where the
    launch has more tiles than each matrix alone, K may be shared by fewer warps, and the fp32 additions are in another order."""
    forms = [small_batch_form(K, [n], M) for n in rows]
    assert all(f == small_batch_form(K, rows, M) for f in forms) == same_form
    c, O = env.c, env.O
    x = _problem(K, 1, M)[1]
    ws = [c.quantize_q4_0(env.t.from_numpy(_problem(K, n, M + i)[0]).to(env.dev)) for i, n in enumerate(rows)]
    xq = env.t.from_numpy(O.quantize_q8_1(x, O.ORDER_COL_KSUPER, c.S_D_SUM_Q)).to(env.dev)
    outs = c.linear_q4_0_multi(ws, rows, xq=xq, K=K, M=M)
    for w, n, y in zip(ws, rows, outs):
        apart = c.mul_mat_q4_0_q8_1(w, xq, K, n, M)
        if same_form:
            assert env.t.equal(y, apart)
        else:
            assert O.err_max_rel(y.cpu().numpy(), apart.cpu().numpy()) <= TOL


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


# The decode kernel for 3 to 8 columns on ready blocks: warps with all, some and none of their blocks (8 of 8, 12 of 16 warps); ends of rows
# and columns; both orders; against the same kernel with the quantizer inside, which sums in the same order: the same bits.
@pytest.mark.parametrize("K,N,M", [(256, 1, 3), (768, 17, 4), (2048, 2400, 8), (2304, 15, 3), (3072, 2401, 5), (4096, 2370, 8), (4096, 16, 4),
                                   (4352, 33, 3), (5376, 2369, 7), (6144, 40, 8), (4608, 31, 6)])
@pytest.mark.parametrize("order", [0, 1])
def test_decode_batch_on_ready_blocks(env, K, N, M, order):
    c, O, t = env.c, env.O, env.t
    w, x = _problem(K, N, M)
    wq = O.quantize_q4_0(w)
    xq = O.quantize_q8_1(x, order, c.S_SUM_X)
    d_w, d_x = t.from_numpy(wq).to(env.dev), t.from_numpy(xq).to(env.dev)
    y = t.full((M, N), float("nan"), device=env.dev)
    c.mul_mat_q4_0_q8_1(d_w, d_x, K, N, M, order, kernel=c.KERNEL_GEMV_MMA, out=y)
    assert O.err_max_rel(y.cpu().numpy(), O.mul_mat_ref(wq, xq, K, N, M, order)) <= TOL
    if M <= 4 and K <= 4096:
        assert t.equal(y, c.linear_q4_0(d_w, t.from_numpy(x).to(env.dev), N, s_mode=c.S_SUM_X))


@pytest.mark.parametrize("K,N,M", [(4224, 4800, 45), (8192, 9600, 24), (11008, 600, 8), (4096, 9600, 1), (4096, 9600, 6)])
def test_poll_limit_of_one_waits_for_copies(env, K, N, M):
    """The shortest limit that can be set: a kernel does not give up on its own copies, and so cannot end before them."""
    c, t = env.c, env.t
    g = t.Generator(device=env.dev)
    g.manual_seed(K + M)
    w = c.quantize_q4_0(t.randn((N, K), generator=g, device=env.dev))
    xq = c.quantize_q8_1(t.randn((M, K), generator=g, device=env.dev))
    right = c.mul_mat_q4_0_q8_1(w, xq, K, N, M)
    c.set_option(c.OPT_WAIT_POLL_LIMIT, 1)
    try:
        results = [c.mul_mat_q4_0_q8_1(w, xq, K, N, M) for _ in range(8)]
        t.cuda.synchronize()
    finally:
        c.set_option(c.OPT_WAIT_POLL_LIMIT, 0)
    assert c.device_fault(clear=True) == 0 and all(t.equal(y, right) for y in results)
