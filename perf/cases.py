"""The work this library is used for, as cases that can be timed and compared.

Four kinds of case, each going through a public entry point the way a host program calls it:

  linear    ``capi.linear_q4_0``: fp32 activations -> Q8_1 -> multiply -> fp32, called from Python on the current
            stream with the workspace and the output kept by the caller.  ``exact`` sets JQ_OPT_PREFILL_EXACT.
  decoder   the linears of a decoder and the kernels that feed them (RMSNorm, SwiGLU; attention itself is not part of
            this library, the query projection stands in for its output).  ``graph``: a decode step recorded once as a
            CUDA graph and replayed, the way a decode loop runs; else called eagerly, as for a prompt.
  mmq       the reference-named module ``mm_q4_0_q8_1_me``: weights, activations and result in host arrays.
  resident  ``capi.ResidentWeights``: weights kept on the device, pinned host activations in, pinned host result out.

Shapes are those of the benchmark's five configurations, plus ragged ones.  The multiply takes K % 128 == 0 and any N
and M.  Weights are N(0, 0.02) quantized to Q4_0, activations N(0, 1) with one channel in a hundred scaled by 20.
"""
import numpy as np
import torch

from jjjetson_ops_b200 import capi, import_reference_modules

EPS = 1e-6
MOST_WORK = 2048 * 8192 * 28672  # M * N * K of the largest case


def listed():
    return [
        # one token through one attention-sized projection: the smallest call, all latency
        _linear("proj_4096x4096_m1", 4096, 4096, 1),
        # one token through a 70B-class feed-forward matrix: a pure weight stream
        _linear("ffn_8192x28672_m1", 8192, 28672, 1),
        # a decode step for one sequence: four 7B-shape layers and the vocabulary projection, as one graph
        _decoder("decode_7b_m1", 4096, 11008, 4096, 32000, 4, 1, True),
        # a decode step for eight sequences at once
        _decoder("decode_7b_m8", 4096, 11008, 4096, 32000, 2, 8, True),
        # a few dozen columns: batched decode, or a handful of draft tokens per sequence being verified
        _linear("ffn_4096x11008_m24", 4096, 11008, 24),
        # ragged: a hidden size that is an odd multiple of 128, an odd number of rows, an odd batch
        _linear("ragged_1408x1003_m45", 1408, 1003, 45),
        # a short prompt through one 7B-shape layer, called eagerly
        _decoder("prompt_7b_m128", 4096, 11008, 4096, 0, 1, 128, False),
        # prefill of a longer prompt, one projection
        _linear("prefill_4096x4096_m512", 4096, 4096, 512),
        # the same for a caller that needs the integer block sums exact
        _linear("prefill_exact_4096x4096_m512", 4096, 4096, 512, True),
        # the largest call: a prefill chunk through the 70B-class feed-forward matrix
        _linear("prefill_8192x28672_m2048", 8192, 28672, 2048),
        # the reference's own host call, weights and all
        {"name": "mmq_host_4096x4096_m1", "kind": "mmq", "K": 4096, "N": 4096, "M": 1},
        # host activations against resident weights, one token at a time
        {"name": "resident_4096x11008_m1", "kind": "resident", "K": 4096, "N": 11008, "M": 1},
    ]


def _linear(name, K, N, M, exact=False):
    return {"name": name, "kind": "linear", "K": K, "N": N, "M": M, "exact": exact}


def _decoder(name, hidden, inner, kv, vocab, layers, M, graph):
    return {"name": name, "kind": "decoder", "hidden": hidden, "inner": inner, "kv": kv, "vocab": vocab, "layers": layers,
            "M": M, "graph": graph}


def _spread(rng, lo, hi):
    """A whole number in [lo, hi], even over the logarithm."""
    return int(round(lo * (hi / lo) ** rng.random()))


def _multiple(rng, lo, hi, of):
    return max(lo, min(hi, _spread(rng, lo, hi) // of * of))


def draw(rng):
    kind = rng.choice(["linear"] * 6 + ["exact", "decoder", "decoder", "mmq", "resident"])
    if kind == "decoder":
        hidden = _multiple(rng, 1024, 4096, 256)
        inner = hidden * rng.choice([2, 3, 4]) - 256 * rng.randrange(4)
        kv = max(128, hidden // rng.choice([1, 4, 8]))
        if rng.random() < 0.5:
            c = _decoder("", hidden, inner, kv, _spread(rng, 4000, 32000), rng.randint(1, 4), _spread(rng, 1, 32), True)
        else:
            c = _decoder("", hidden, inner, kv, 0, 1, _spread(rng, 16, 512), False)
    elif kind == "mmq":
        c = {"kind": "mmq", "K": _multiple(rng, 256, 8192, 128), "N": _spread(rng, 64, 8192), "M": _spread(rng, 1, 32)}
    elif kind == "resident":
        c = {"kind": "resident", "K": _multiple(rng, 1024, 8192, 256), "N": _spread(rng, 512, 28672), "M": _spread(rng, 1, 16)}
    else:
        M = _spread(rng, 64 if kind == "exact" else 1, 2048)
        if rng.random() < 0.2:  # K an odd multiple of 128, as some models' hidden and inner sizes are
            K, M = 128 + _multiple(rng, 256, 5376, 256), min(M, 256)
        else:
            K = _multiple(rng, 256, 11008, 256)
        N = _spread(rng, 64, 32000)
        N = max(64, min(N, MOST_WORK // (M * K)))
        c = _linear("", K, N, M, kind == "exact")
    c.pop("name", None)
    return c


# ---- inputs ----------------------------------------------------------------------------------------------------
def _device():
    return torch.device("cuda", torch.cuda.current_device())


def _weights(gen, N, K):
    w = torch.randn((N, K), generator=gen, device=gen.device)
    return capi.quantize_q4_0(w.mul_(0.02))


def _activations(gen, M, K):
    x = torch.randn((M, K), generator=gen, device=gen.device)
    outliers = torch.randperm(K, generator=gen, device=gen.device)[: max(1, K // 100)]
    x[:, outliers] *= 20.0
    return x


def _blocks(K, M):
    return torch.zeros(capi.q8_1_bytes(K, M), dtype=torch.uint8, device=_device())


def prepare(case, seed):
    capi.set_option(capi.OPT_STATIC_WEIGHTS, 1)  # what an inference engine sets once: weights are never rewritten
    dev = _device()
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    s = dict(case)
    if case["kind"] == "decoder":
        return _prepare_decoder(s, gen)
    K, N, M = case["K"], case["N"], case["M"]
    w, x = _weights(gen, N, K), _activations(gen, M, K)
    if case["kind"] == "linear":
        s.update(w=w, x=x, ws=_blocks(K, M), y=torch.zeros((M, N), device=dev))
    elif case["kind"] == "mmq":
        s.update(mmq=import_reference_modules()[1].mmq, w=w.reshape(-1).cpu().numpy(), x=x.cpu().numpy(),
                 ws=np.zeros(capi.q8_1_bytes(K, M), dtype=np.uint8), y=np.zeros((M, N), dtype=np.float32), dims=[K, M, 1, 1])
    else:
        s.update(rw=capi.ResidentWeights(w.cpu().numpy(), N, K), x=x.cpu().pin_memory(), y=torch.zeros((M, N)).pin_memory())
    return s


def _prepare_decoder(s, gen):
    dev, M, H, I, KV = gen.device, s["M"], s["hidden"], s["inner"], s["kv"]

    def norm():
        return 1.0 + 0.1 * torch.randn(H, generator=gen, device=dev)

    s["stack"] = [dict(q=_weights(gen, H, H), k=_weights(gen, KV, H), v=_weights(gen, KV, H), o=_weights(gen, H, H),
                       gate=_weights(gen, I, H), up=_weights(gen, I, H), down=_weights(gen, H, I), norm1=norm(), norm2=norm())
                  for _ in range(s["layers"])]
    s["embedded"] = torch.randn((M, H), generator=gen, device=dev)
    for name, width in (("res", H), ("q", H), ("k", KV), ("v", KV), ("o", H), ("gate", I), ("up", I), ("down", H)):
        s["y_" + name] = torch.zeros((M, width), device=dev)
    s.update(hq=_blocks(H, M), oq=_blocks(H, M), iq=_blocks(I, M))
    if s["vocab"]:
        s.update(norm_f=norm(), head=_weights(gen, s["vocab"], H), y_logits=torch.zeros((M, s["vocab"]), device=dev))
    if s["graph"]:
        stream = torch.cuda.Stream(dev)
        stream.wait_stream(torch.cuda.current_stream(dev))
        with torch.cuda.stream(stream):
            _decoder_step(s)
        torch.cuda.current_stream(dev).wait_stream(stream)
        s["recorded"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(s["recorded"], stream=stream):
            _decoder_step(s)
    return s


# ---- one pass --------------------------------------------------------------------------------------------------
def _decoder_step(s):
    H, I, KV, M, res = s["hidden"], s["inner"], s["kv"], s["M"], s["y_res"]
    res.copy_(s["embedded"])
    for i, w in enumerate(s["stack"]):
        if i == 0:
            capi.rms_norm_q8_1(res, w["norm1"], EPS, xq=s["hq"])
        else:
            capi.rms_norm_q8_1(s["y_down"], w["norm1"], EPS, residual=res, xq=s["hq"])
        capi.linear_q4_0_multi([w["q"], w["k"], w["v"]], [H, KV, KV], xq=s["hq"], K=H, M=M, outs=[s["y_q"], s["y_k"], s["y_v"]])
        capi.linear_q4_0(w["o"], s["y_q"], H, ws=s["oq"], out=s["y_o"])
        capi.rms_norm_q8_1(s["y_o"], w["norm2"], EPS, residual=res, xq=s["hq"])
        capi.linear_q4_0_multi([w["gate"], w["up"]], [I, I], xq=s["hq"], K=H, M=M, outs=[s["y_gate"], s["y_up"]])
        capi.swiglu_q8_1(s["y_gate"], s["y_up"], xq=s["iq"])
        capi.mul_mat_q4_0_q8_1(w["down"], s["iq"], I, H, M, out=s["y_down"])
    if s["vocab"]:
        capi.rms_norm_q8_1(s["y_down"], s["norm_f"], EPS, residual=res, xq=s["hq"])
        capi.mul_mat_q4_0_q8_1(s["head"], s["hq"], H, s["vocab"], M, out=s["y_logits"])


def run(state):
    s = state
    if s["kind"] == "linear":
        if s["exact"]:
            capi.set_option(capi.OPT_PREFILL_EXACT, 1)
        capi.linear_q4_0(s["w"], s["x"], s["N"], ws=s["ws"], out=s["y"])
        if s["exact"]:
            capi.set_option(capi.OPT_PREFILL_EXACT, 0)
        return s["y"], s["ws"]
    if s["kind"] == "decoder":
        if s["graph"]:
            s["recorded"].replay()
        else:
            _decoder_step(s)
        return [s[n] for n in ("y_res", "y_k", "y_v", "y_down")] + ([s["y_logits"]] if s["vocab"] else [])
    if s["kind"] == "mmq":
        s["mmq"](s["w"], s["x"], s["ws"], s["y"], s["dims"], s["N"], s["K"])
        return s["y"], s["ws"]
    s["rw"].linear(s["x"].data_ptr(), s["y"].data_ptr(), s["M"])
    return s["y"]


# ---- what a pass cannot do without ----------------------------------------------------------------------------------
def work(case):
    M = case["M"]
    if case["kind"] == "decoder":
        H, I, KV, V, L = (case[n] for n in ("hidden", "inner", "kv", "vocab", "layers"))
        weights = L * (2 * H * H + 2 * KV * H + 3 * I * H) + V * H
        values = L * 2 * H + M * (3 * H + 2 * KV + V)  # norm vectors; embedded, res, down, k, v, logits
        return {"bytes": weights * 18 // 32 + 4 * values, "flops": 2 * M * weights}
    K, N = case["K"], case["N"]
    blocks = 0 if case["kind"] == "resident" else capi.q8_1_bytes(K, M)
    return {"bytes": capi.q4_0_bytes(N, K) + 4 * M * (K + N) + blocks, "flops": 2 * M * N * K}


def tolerance(case):
    M = case["M"]
    if case["kind"] == "decoder":
        # A last-bit difference in an activation can move it across a rounding boundary of the int8 quantizer: one step
        # is about 0.02 of the row's deviation.  Sums in fp32 (2e-7) move 2e-5 of the values, which adds 1e-4 per
        # quantization; operands rounded to fp16 (3e-4, batches of 64 and more) move 2.5 % of them, 4e-3 each.
        return {"rel": 2e-3 if M < 64 else 1e-2}
    if M >= 64 and case["K"] % 256 == 0 and not case.get("exact"):
        return {"rel": 1e-3}  # scaled operands rounded to fp16
    return {"rel": 1e-5}      # exact integer block sums, fp32 accumulation
