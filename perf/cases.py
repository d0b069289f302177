"""Performance cases of the framework: what its users have it do, through its public entry points.

A case is a dict of plain values; its "path" says which entry point it goes through:

    decode         one mini-batch of 1..15 tokens against the resident TTT-Linear state (token-by-token generation of
                   the inner model, the tail of a sequence), state advanced in place
    decode_layer   one generated token through the whole outer layer, as CUDA graphs replay it
    linear         whole-sequence TTT-Linear inner loop: forward (inference), or forward + backward through autograd
    mlp            the same for the 2-layer TTT-MLP inner model
    prefill        the whole outer layer on a prompt (projections, inner loop, norm, output projection), no gradients
    train          the whole outer layer, forward + backward, gradients of its input and of every parameter

Inputs follow the distributions of ttt_rs_b200.synthetic (rows N(0, 1) / sqrt(head_dim), states N(0, 0.02), learning
rates sigmoid(N(0, 1)) / head_dim, token_eta = 1 / (position in the mini-batch + 1), output gradients N(0, 1e-2)), with
LayerNorm parameters and biases a little off their initial 1 / 0, as they are once training has begun.
"""

import math

import torch

import ttt_rs_b200 as tb

DTYPES = {"bf16": torch.bfloat16, "f32": torch.float32}
BASE = {"dtype": "bf16", "F": 64, "mb": 16, "K": 16, "grad": False, "gate": False, "share_qk": False, "pos": "rope"}


def _case(name, path, B, H, T, **more):
    c = dict(BASE, path=path, B=B, H=H, T=T, **more)
    if name is not None:
        c["name"] = name
    return c


def listed():
    return [
        # generation with a small batch: one token per sequence through the inner model (latency and host cost)
        _case("decode-b8", "decode", 8, 12, 1),
        # the same through one whole layer, the step a serving loop repeats for each layer and token
        _case("decode-layer-b8", "decode_layer", 8, 12, 1),
        # the smallest whole-sequence call: the float32 parity configuration, forward only
        _case("linear-fwd-f32-small", "linear", 2, 4, 256, dtype="f32", K=1),
        # training of the inner loop at the 125M layer shape: the headline workload
        _case("linear-train-b32", "linear", 32, 12, 2048, grad=True),
        # the same hidden width split into 24 heads of 32 features, small batch with an odd number of mini-batches
        _case("linear-train-d32-b3", "linear", 3, 24, 1040, F=32, grad=True),
        # training in float32 (parity and debugging runs)
        _case("linear-train-f32-b8", "linear", 8, 12, 2048, dtype="f32", grad=True),
        # long context at the 1.3B layer shape
        _case("linear-train-8k", "linear", 8, 32, 8192, grad=True),
        # TTT-MLP training
        _case("mlp-train-b16", "mlp", 16, 12, 2048, grad=True),
        # TTT-MLP inference on a few shorter sequences
        _case("mlp-fwd-b4", "mlp", 4, 12, 496),
        # one prompt of ragged length (tail mini-batch of its own), small batch: time to first token
        _case("prefill-b1-ragged", "prefill", 1, 12, 1001, K=1),
        # a large prefill at the 1.3B layer shape: the largest case
        _case("prefill-b8-8k", "prefill", 8, 32, 8192, K=1),
        # training of a whole layer at the 125M shape
        _case("train-layer-b32", "train", 32, 12, 2048),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """Another case of the same ranges, no larger than the listed ones of its kind."""
    while True:
        c = _draw(rng)
        most = max((_cost(x) for x in listed() if (x["path"], x["dtype"]) == (c["path"], c["dtype"])), default=None)
        if c["path"] in ("decode", "decode_layer") or _cost(c) <= most:
            return c


def _cost(case):
    w = work(case)
    return max(w["bytes"], w["flops"] / 50)


def _draw(rng):
    path = rng.choice(("decode", "decode_layer", "linear", "linear", "linear", "mlp", "mlp", "prefill", "prefill", "train", "train"))
    if path == "decode":
        # mostly single tokens; tails of up to 15
        return _case(None, path, _log_int(rng, 1, 256), rng.choice((4, 12, 16, 32)), rng.choice((1, 1, 1, rng.randint(2, 15))),
                     F=rng.choice((64, 64, 32)), dtype=rng.choice(("bf16", "bf16", "f32")))
    if path == "decode_layer":
        return _case(None, path, _log_int(rng, 1, 128), rng.choice((12, 16, 32)), 1, gate=rng.random() < 0.5)
    H = rng.choice((4, 12, 16, 24, 32))
    if path == "linear":
        mb = rng.choice((16, 16, 16, 8))
        return _case(None, path, _log_int(rng, 1, 32), H, mb * _log_int(rng, 4, 1024), F=rng.choice((64, 64, 32)), mb=mb,
                     dtype=rng.choice(("bf16", "bf16", "f32")), K=rng.choice((1, 4, 16, 16)), grad=rng.random() < 0.6)
    if path == "mlp":
        return _case(None, path, _log_int(rng, 1, 32), H, 16 * _log_int(rng, 4, 512), grad=rng.random() < 0.6)
    H = max(H, 12)
    if path == "prefill":
        return _case(None, path, _log_int(rng, 1, 32), H, _log_int(rng, 17, 8192), K=1, gate=rng.random() < 0.4,
                     share_qk=rng.random() < 0.25, pos=rng.choice(("rope", "rope", "rope_global", "none")))
    return _case(None, path, _log_int(rng, 1, 32), H, 16 * _log_int(rng, 4, 256), gate=rng.random() < 0.4,
                 share_qk=rng.random() < 0.25)


# ---- what a user's program has in hand ---------------------------------------------------------------------------

def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _randn(g, *shape, scale=1.0, at=0.0, dtype=torch.float32):
    return (torch.randn(*shape, generator=g, device="cuda") * scale + at).to(dtype)


def _layer(case, seed, partial):
    """An outer layer and its inner model, parameters a little off their initial values."""
    dt = DTYPES[case["dtype"]]
    cfg = tb.TTTLayerConfig(hidden_size=case["H"] * case["F"], num_heads=case["H"], mini_batch_size=case["mb"],
                            pos_encoding=case["pos"], use_gate=case["gate"], share_qk=case["share_qk"])
    torch.manual_seed(seed)
    layer = tb.TTT(cfg, device="cuda", dtype=dt)
    inner = tb.new_inner(cfg, checkpoint_interval=case["K"], device="cuda", dtype=dt, allow_partial=partial,
                         partial_in_place=partial)
    g = _gen(seed)
    with torch.no_grad():
        for p in list(layer.parameters()) + list(inner.parameters()):
            p.add_(_randn(g, *p.shape, scale=0.01, dtype=dt))
    return layer, inner, g


def prepare(case, seed):
    path, B, H, T, F = case["path"], case["B"], case["H"], case["T"], case["F"]
    dt = DTYPES[case["dtype"]]
    if path in ("prefill", "train", "decode_layer"):
        layer, inner, g = _layer(case, seed, partial=path != "train")
        C = H * F
        if path == "decode_layer":
            with torch.no_grad():
                state = inner.init_state(B)
                layer(_randn(g, B, 64, C, scale=0.5, dtype=dt), inner, state, 0)  # the prompt
            return {"path": path, "dec": tb.DecodeGraphs(layer, inner, state, B), "state": state, "pos": 64,
                    "x": _randn(g, B, 64, C, scale=0.5, dtype=dt)}
        s = {"path": path, "layer": layer, "inner": inner, "B": B, "x": _randn(g, B, T, C, scale=0.5, dtype=dt)}
        if path == "train":
            s["x"].requires_grad_(True)
            s["gy"] = _randn(g, B, T, C, scale=1e-2, dtype=dt)
        return s
    g = _gen(seed)
    d = {k: _randn(g, B, H, T, F, scale=F ** -0.5, dtype=dt) for k in ("xq", "xk", "xv")}
    pos = torch.arange(T, device="cuda") % case["mb"]
    d["token_eta"] = (1.0 / (pos + 1)).to(dt)
    d["ttt_lr_eta"] = (torch.sigmoid(_randn(g, B, H, T)) / F).to(dt)
    d["ln_weight"], d["ln_bias"] = _randn(g, H, F, scale=0.05, at=1.0, dtype=dt), _randn(g, H, F, scale=0.05, dtype=dt)

    def state(*shape, scale):  # one initial state per head, the same for every sequence of the batch
        return _randn(g, H, *shape, scale=scale, dtype=dt).unsqueeze(0).repeat(B, *([1] * (len(shape) + 1)))

    if path == "mlp":
        d.update(w1=state(F, 4 * F, scale=0.02), b1=state(4 * F, scale=0.01), w2=state(4 * F, F, scale=0.02),
                 b2=state(F, scale=0.01))
        order = ("xq", "xk", "xv", "w1", "b1", "w2", "b2", "token_eta", "ttt_lr_eta", "ln_weight", "ln_bias")
    else:
        d.update(weight=state(F, F, scale=0.02), bias=state(F, scale=0.01))
        order = ("xq", "xk", "xv", "weight", "bias", "token_eta", "ttt_lr_eta", "ln_weight", "ln_bias")
    ts = [d[k].contiguous() for k in order]
    s = {"path": path, "cfg": tb.FusedTttConfig.new(case["mb"], F, 1e-6, 128, case["K"]), "grad": case["grad"]}
    if path == "decode":
        s["ins"] = tb.TttInputs(*ts)
        return s
    if case["grad"]:
        for t in ts:
            t.requires_grad_(True)
        s["go"] = _randn(g, B, H, T, F, scale=1e-2, dtype=dt)
    s["ts"] = ts
    return s


# ---- one pass ----------------------------------------------------------------------------------------------------

def _inner_loop(s):
    ts, cfg = s["ts"], s["cfg"]
    if s["path"] == "linear":
        return tb.fused_ttt_tile_forward_multi(*ts, cfg)
    st = tb.TTTMLPState(*ts[3:7])
    f = tb.fused_ttt_mlp if s["grad"] else tb.fused_ttt_mlp_forward
    out, new = f(*ts[:3], st, *ts[7:], cfg)
    return out, new.w1, new.b1, new.w2, new.b2


def run(s):
    path = s["path"]
    if path == "decode":
        o = tb.TttTileMultiKernel.forward_partial(s["ins"], s["cfg"], in_place=True)
        return o.output, o.weight, o.bias
    if path == "decode_layer":
        i = s["pos"] % 64
        y = s["dec"].step(s["x"][:, i:i + 1], s["pos"])
        s["pos"] += 1
        return y, s["state"].weight, s["state"].bias
    if path == "prefill":
        with torch.no_grad():
            st = s["inner"].init_state(s["B"])
            y = s["layer"](s["x"], s["inner"], st)
        return y, st.weight, st.bias
    if path == "train":
        params = list(s["layer"].parameters()) + list(s["inner"].inner.parameters())
        for t in params + [s["x"]]:
            t.grad = None
        y = s["layer"](s["x"], s["inner"], s["inner"].init_state(s["B"]))
        y.backward(s["gy"])
        return [y.detach(), s["x"].grad] + [p.grad for p in params]
    if not s["grad"]:
        with torch.no_grad():
            return _inner_loop(s)
    for t in s["ts"]:
        t.grad = None
    res = _inner_loop(s)
    res[0].backward(s["go"])
    return [r.detach() for r in res] + [t.grad for t in s["ts"]]


# ---- what a pass cannot do without -------------------------------------------------------------------------------

def work(case):
    path, B, H, T, F, mb = (case[k] for k in ("path", "B", "H", "T", "F", "mb"))
    e = 2 if case["dtype"] == "bf16" else 4
    rows, C = B * H * T, H * F
    m = min(mb, T)  # tokens of a mini-batch
    E = 4 * F
    if path == "mlp":
        state = 2 * F * E + E + F
        # per token: K W1, Q W1, X2 W2, Xb2 W2, G2 W2^T, two updates; four m-wide products; the backward twice that
        fwd = rows * 2 * (7 * F * E + m * (2 * F + 2 * E))
        bwd = rows * 2 * (14 * F * E + m * (4 * F + 4 * E))
    else:
        state = F * F + F
        fwd = rows * 2 * (3 * F * F + m * 2 * F)  # K W, Q W, the update; Q K^T, M G
        bwd = rows * 2 * (6 * F * F + m * 4 * F)  # dZb W^T, dZ1 W^T, G dW^T, K dW, two updates; dZb G^T, dA K, dA^T Q, M^T dZb
    if path in ("decode", "linear", "mlp"):
        # q, k, v and learning rates in, output out, the state in and out, LayerNorm parameters, token_eta
        nbytes = (rows * (4 * F + 1) + 2 * B * H * state + 2 * C + T) * e
        if case["grad"]:  # output gradient in, the other inputs' gradients out
            nbytes += (rows * (4 * F + 1) + B * H * state + 2 * C + T) * e
        return {"bytes": nbytes, "flops": fwd + (bwd if case["grad"] else 0)}
    nproj = (2 if case["share_qk"] else 3) + (1 if case["gate"] else 0)
    weights = (nproj + 1) * C * C + H * C + H * state
    gemm = 2 * B * T * C * ((nproj + 1) * C + H)
    if path == "train":  # input and output gradient in, output and input gradient out; weights in, their gradients out
        return {"bytes": (4 * B * T * C + 2 * weights) * e, "flops": fwd + bwd + 3 * gemm}
    own = 2 * B * H * state if path == "decode_layer" else B * H * state  # a prefill's state starts from the parameters
    return {"bytes": (2 * B * T * C + weights + own) * e, "flops": fwd + gemm}


def tolerance(case):
    # bf16 operands and float32 sums chained over up to 1024 mini-batches: gradients of two correct implementations
    # differ by about 5e-3 (2-norm); float32 ones by a few 1e-6, the sums over all tokens by more
    if case["dtype"] == "f32":
        return {"rel": 3e-5, "max": 2e-3}
    return {"rel": 1e-2, "max": 0.4}
