"""The work that users of this library have it do, as cases to be timed.

A case is a dict of plain values; `kind` says which public entry point it goes through:

  matmul    y [m, N] = x [m, K] . W on a BCQ container (lutgemm_b200.matmul, or matmul_f32 where f32 is true)
  linear    the same through the torch module BCQLinear, activations [1, m, K]: the prefill of a prompt
  stack     the linears of a decoder's decode step, every layer's four matvecs in one launch (MatvecSequence)
  quantize  a dense weight to bit planes and scales, greedy start + alternating refinement (bcq_quantize_device)
  convert   uniform (RTN) codes to bit planes, scales and offset (uniform_to_bcq_device)

Values and distributions are those of the benchmark configurations (lutgemm_b200/synth.py): activations fp16 N(0, 1),
fair sign bits, scales |N(0, 0.02)|; uniform layers have scales |N(0, 0.01)| and zero points and codes in [0, 2^q).
"""
import math

import torch

import lutgemm_b200 as L
from lutgemm_b200.torch_op import BCQLinear
from lutgemm_b200.tp_seq import stack_program


def _matmul(name, N, K, q, g, m, bias=False, f32=False):
    return dict(name=name, kind="matmul", N=N, K=K, q=q, g=g, m=m, bias=bias, f32=f32)


def listed():
    return [
        # decode, one token: a small square projection, where launch and latency count
        _matmul("matvec_4096", 4096, 4096, 3, 128, 1),
        # decode, one token: the attention output projection of a large decoder (the headline shape)
        _matmul("matvec_12288", 12288, 12288, 3, 128, 1),
        # decode, one token: the up projection of its feed-forward part at 4 planes, the largest single matvec
        _matmul("matvec_ffn_q4", 49152, 12288, 4, 128, 1),
        # decode, one token: the down projection of a uniformly quantised model, offset included
        _matmul("matvec_uniform_q4", 8192, 28672, 4, 128, 1, bias=True),
        # decode, one token: sizes that are multiples of nothing large, in a group size that is no power of two
        _matmul("matvec_ragged", 11004, 4128, 3, 96, 1),
        # decode, a handful of sequences: the up projection of a uniformly quantised model
        _matmul("batch_4", 28672, 8192, 4, 128, 4, bias=True),
        # decode, a small batch at 2 planes
        _matmul("batch_16", 8192, 8192, 2, 64, 16),
        # decode, a large batch at 2 planes
        _matmul("batch_128", 8192, 8192, 2, 64, 128),
        # prefill of a long prompt through the torch module, uniformly quantised weights
        dict(name="prefill_2048", kind="linear", N=8192, K=8192, q=4, g=128, m=2048, bias=True),
        # decode step of two decoder layers, hidden 12288, feed-forward 49152, in one launch
        dict(name="stack_2_layers", kind="stack", hidden=12288, ffn=49152, layers=2, q=3, g=128),
        # quantising one layer of a model
        dict(name="quantize_4096", kind="quantize", N=4096, K=4096, q=3, g=128, rounds=15),
        # loading one uniformly quantised layer
        dict(name="convert_8192", kind="convert", N=8192, K=8192, q=4, g=128),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["matvec", "batch", "linear", "stack", "quantize", "convert"], [6, 4, 2, 1, 1, 1])[0]
    if kind in ("matvec", "batch", "linear"):
        m = 1 if kind == "matvec" else _log_uniform(rng, 2, 128) if kind == "batch" else _log_uniform(rng, 129, 2048)
        g = rng.choice([64, 128, 128, 256] if m > 4 else [32, 64, 96, 128, 128, 128, 256, 512])
        q = rng.choice([1, 2, 3, 3, 4, 4, 5])
        # output features: mostly multiples of 256, else of 8; small batches also meet multiples of 4 and odd counts
        unit = rng.choices([256, 8, 4, 1], [6, 5, 2, 1] if m <= 4 else [6, 5, 0, 0])[0]
        top = 603_979_776 if kind != "linear" else 67_108_864 * 2048 // m      # weights of the largest listed case
        K = max(1, _log_uniform(rng, 1024, 28672 if kind != "linear" else 12288) // g) * g
        N = max(1, min(_log_uniform(rng, 1024, 49152 if kind != "linear" else 12288), top * 4 // (K * q)) // unit) * unit
        if kind == "linear":
            return dict(kind="linear", N=N, K=K, q=min(q, 4), g=g, m=m, bias=rng.random() < 0.5)
        return dict(kind="matmul", N=N, K=K, q=q, g=g, m=m, bias=rng.random() < 0.4, f32=rng.random() < 0.2)
    if kind == "stack":
        hidden = 1024 * rng.randint(2, 12)
        return dict(kind="stack", hidden=hidden, ffn=4 * hidden, layers=rng.randint(1, 2), q=rng.choice([2, 3]), g=128)
    g = rng.choice([64, 128, 256])
    top = 4096 * 4096 if kind == "quantize" else 8192 * 8192
    K = _log_uniform(rng, 1024, 8192) // g * g
    N = min(_log_uniform(rng, 1024, 8192), top // K) // 8 * 8
    if kind == "quantize":
        return dict(kind="quantize", N=N, K=K, q=rng.choice([2, 3]), g=g, rounds=15)
    return dict(kind="convert", N=N, K=K, q=rng.choice([2, 3, 4]), g=g)


def _gen(seed, salt=0):
    return torch.Generator(device="cuda").manual_seed(1_000_003 * int(seed) + salt)


def _planes(gen, N, K, q):
    return torch.randint(-2**31, 2**31, (K // 32, q, N), dtype=torch.int32, device="cuda", generator=gen)


def _scales(gen, shape, std):
    return (torch.randn(shape, device="cuda", generator=gen).abs_() * std).half()


def _uniform_scale_zero(gen, N, G, q):
    scale = (torch.randn((N, G), device="cuda", generator=gen).abs_() * 0.01).half().float().clamp_(min=2.0**-14)
    zero = torch.randint(0, 2**q, (N, G), device="cuda", generator=gen).float()
    return scale, zero


def _layer(gen, N, K, q, g, bias):
    """Container tensors (bW, alpha, q_bias) of one layer; with an offset they are those of a uniformly quantised one
    (codes of q fair bits are q fair planes; alpha_b = scale / 2 * 2^b, q_bias = sum_b alpha_b - scale * zero)."""
    bW, G = _planes(gen, N, K, q), K // g
    if not bias:
        return bW, _scales(gen, (G, q, N), 0.02), None
    scale, zero = _uniform_scale_zero(gen, N, G, q)
    scale, zero = scale.t(), zero.t()
    alpha = torch.stack([scale * (0.5 * 2**b) for b in range(q)], dim=1).half().contiguous()
    q_bias = (scale * (0.5 * (2**q - 1) - zero)).half().contiguous()
    return bW, alpha, q_bias


def prepare(case, seed):
    kind, gen = case["kind"], _gen(seed)
    if kind in ("matmul", "linear"):
        N, K, q, g, m = (case[k] for k in ("N", "K", "q", "g", "m"))
        bW, alpha, q_bias = _layer(gen, N, K, q, g, case["bias"])
        x = torch.randn((m, K), device="cuda", generator=gen).half()
        if kind == "linear":
            return dict(kind=kind, module=BCQLinear(bW, alpha, q_bias, max_batch=m).reserve(), x=x.view(1, m, K))
        w = L.nQWeight_fp16.from_device(bW, alpha, q_bias, K, N, q, False, K // g)
        w.reserve_batch(m)
        f32 = bool(case["f32"])
        y = torch.empty((m, N), dtype=torch.float32 if f32 else torch.float16, device="cuda")
        return dict(kind=kind, w=w, x=x, y=y, m=m, f32=f32)
    if kind == "stack":
        h, f, q, g = case["hidden"], case["ffn"], case["q"], case["g"]
        x = torch.randn(h, device="cuda", generator=gen).half()
        y = torch.empty(h, dtype=torch.float16, device="cuda")
        buffers, ops = stack_program(h, f, case["layers"], 0, 1)
        for o in ops:
            if o["idx"] is not None:
                N, K = ((3 * h, h), (h, h), (f, h), (h, f))[o["idx"]]
                # scales that keep the activations' size through the layers
                o["w"] = L.nQWeight_fp16.from_device(_planes(gen, N, K, q), _scales(gen, (K // g, q, N), 1.0 / math.sqrt(K * q)),
                                                     None, K, N, q, False, K // g)
            if o["in_kind"] == 0:
                o["x_ext"] = x
            if o["out_kind"] == 0:
                o["y_ext"] = y
        return dict(kind=kind, seq=L.MatvecSequence(ops, buffers), x=x, y=y)
    N, K, q, g = case["N"], case["K"], case["q"], case["g"]
    if kind == "quantize":
        w = torch.randn((N, K), device="cuda", generator=gen) * 0.02
        return dict(kind=kind, w=w, q=q, g=g, rounds=case["rounds"])
    scale, zero = _uniform_scale_zero(gen, N, K // g, q)
    code = torch.randint(0, 2**q, (N, K // g, g), dtype=torch.int32, device="cuda", generator=gen)
    return dict(kind=kind, scale=scale, zero=zero, code=code, q=q)


def run(state):
    kind = state["kind"]
    if kind == "matmul":
        if state["f32"]:
            return L.matmul_f32(state["y"], state["x"], state["w"], state["m"])
        return L.matmul(state["y"], state["x"], state["w"], state["m"])
    if kind == "linear":
        return state["module"](state["x"])
    if kind == "stack":
        state["seq"].run()
        return state["y"]
    if kind == "quantize":
        return L.bcq_quantize_device(state["w"], state["q"], rounds=state["rounds"], group_size=state["g"])
    return L.uniform_to_bcq_device(state["scale"], state["zero"], state["code"], state["q"])


def work(case):
    kind, q, g = case["kind"], case["q"], case["g"]

    def weight_bytes(N, K, bias=False):
        return N * K * q // 8 + 2 * (K // g) * N * (q + (1 if bias else 0))

    if kind in ("matmul", "linear"):
        N, K, m = case["N"], case["K"], case["m"]
        out = 4 if case.get("f32") else 2
        return {"bytes": weight_bytes(N, K, case["bias"]) + 2 * m * K + out * m * N, "flops": 2 * m * N * K}
    if kind == "stack":
        h, f = case["hidden"], case["ffn"]
        shapes = ((3 * h, h), (h, h), (f, h), (h, f))
        return {"bytes": case["layers"] * sum(weight_bytes(N, K) for N, K in shapes) + 4 * h,
                "flops": case["layers"] * sum(2 * N * K for N, K in shapes)}
    N, K = case["N"], case["K"]
    if kind == "quantize":
        # per weight and round: B^T w, the Gram matrix' upper triangle (a multiply-add each) and q comparisons
        return {"bytes": 4 * N * K + weight_bytes(N, K), "flops": case["rounds"] * N * K * (2 * q + q * (q + 1) + q)}
    return {"bytes": 4 * N * K + 8 * N * (K // g) + weight_bytes(N, K, True), "flops": 0}


def tolerance(case):
    kind = case["kind"]
    if kind == "convert":
        return "exact"
    if kind == "quantize":
        # Measured with the weights of every group in another order (other summation orders): scales differ by 2.5e-5,
        # where fp32 sums fall on the other side of an fp16 rounding; 1.9e-6 of the packed words hold a weight that
        # changed level.
        return {"rel": 1e-4, "differ": 1e-5}
    if kind == "stack":
        # Every matvec hands its result on in fp16, and the layers amplify it: two runs of the same inputs, whose fp32
        # sums are added in an order that is not fixed, differ by 6.2e-4.
        return {"rel": 2.5e-3}
    if case.get("f32"):
        # against 64-bit sums: 2.1e-6
        return {"rel": 1e-5}
    # against 64-bit sums: 2.1e-4, the rounding to fp16
    return {"rel": 8e-4}


def _dense_columns(bW, alpha, q_bias, n0, n1):
    """Columns n0..n1 of the dense weight in 64 bits, [K, n1 - n0]: bit k % 32 of word k / 32 is the sign of weight k."""
    kw, q, _ = bW.shape
    G = alpha.shape[0]
    shift = torch.arange(32, device=bW.device, dtype=torch.int32).view(1, 32, 1)
    w = 0.0
    for b in range(q):
        sign = ((bW[:, b, None, n0:n1] >> shift) & 1).double().mul_(2).sub_(1).view(G, kw * 32 // G, n1 - n0)
        w = w + sign * alpha[:, b, None, n0:n1].double()
    if q_bias is not None:
        w = w + q_bias[:, None, n0:n1].double()
    return w.view(kw * 32, n1 - n0)


def _product(x, bW, alpha, q_bias):
    """x [m, K] times the weight in 64 bits, a few thousand columns at a time."""
    N = bW.shape[2]
    step = max(1, (1 << 26) // (bW.shape[0] * 32))
    return torch.cat([x.double() @ _dense_columns(bW, alpha, q_bias, n, min(N, n + step)) for n in range(0, N, step)], dim=1)


def _exact_scales(w, q, g, rounds):
    """The quantiser's scales in 64 bits, [G, q, N]: greedy start, then per round the scales from the normal equations
    by q steps of conjugate gradient (1e-6 in both denominators) and every weight to the nearest level."""
    N, K = w.shape
    w = w.double().view(-1, g)
    c, i = torch.arange(2**q, device=w.device)[:, None], torch.arange(q, device=w.device)[None, :]
    signs = torch.where(((c >> (q - 1 - i)) & 1) == 1, -1.0, 1.0).double()
    r, B, alpha = w.clone(), [], []
    for _ in range(q):
        B.append(torch.sign(r))
        alpha.append(r.abs().mean(dim=1))
        r = r - B[-1] * alpha[-1][:, None]
    B, alpha = torch.stack(B, dim=2), torch.stack(alpha, dim=1)
    for _ in range(rounds if q > 1 else 0):
        A = B.transpose(1, 2) @ B
        r = (B.transpose(1, 2) @ w[:, :, None] - A @ alpha[:, :, None])[:, :, 0]
        p, new = r, (r * r).sum(1)
        for _ in range(q):
            old, Ap = new, (A @ p[:, :, None])[:, :, 0]
            a = (old / ((p * Ap).sum(1) + 1e-6))[:, None]
            alpha, r = alpha + a * p, r - a * Ap
            new = (r * r).sum(1)
            p = r + (new / (old + 1e-6))[:, None] * p
        alpha = alpha.abs().sort(dim=1, descending=True).values
        level, order = (alpha @ signs.T).sort(dim=1, stable=True)
        at = torch.searchsorted((level[:, 1:] + level[:, :-1]) / 2, w, right=True)
        B = signs[torch.gather(order, 1, at)]
    return alpha.view(N, K // g, q).permute(1, 2, 0)


def exact(case, seed):
    """The outputs of run in 64 bits.  The converter's are whole numbers and roundings that are compared bit for bit, the
    quantiser's packed words are choices between levels: both have no such value."""
    kind, gen = case["kind"], _gen(seed)
    if kind in ("matmul", "linear"):
        N, K, q, g, m = (case[k] for k in ("N", "K", "q", "g", "m"))
        container = _layer(gen, N, K, q, g, case["bias"])
        x = torch.randn((m, K), device="cuda", generator=gen).half()
        y = _product(x, *container)
        return y.view(1, m, N) if kind == "linear" else y
    if kind == "stack":
        h, f, q, g = case["hidden"], case["ffn"], case["q"], case["g"]
        x = torch.randn(h, device="cuda", generator=gen).half()[None]
        for _ in range(case["layers"]):
            # the first `hidden` values of the first product stand in for the attention result
            for N, K in ((3 * h, h), (h, h), (f, h), (h, f)):
                bW, scales = _planes(gen, N, K, q), _scales(gen, (K // g, q, N), 1.0 / math.sqrt(K * q))
                x = _product(x[:, :K], bW, scales, None)
        return x[0]
    if kind == "quantize":
        w = torch.randn((case["N"], case["K"]), device="cuda", generator=gen) * 0.02
        return None, _exact_scales(w, case["q"], case["g"], case["rounds"])
    return None
