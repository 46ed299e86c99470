"""What the performance of this package is measured on: the calls its users make, over the sizes they make them at.

`listed()` names one case per way of using the package; `draw(rng)` gives more of the same ranges.  Every case is a dict of
plain values, `prepare` makes what the caller has in hand (bounds, weights, a verifier), `run` is one call or the short
chain of calls that belongs together, `work` the bytes and operations that call cannot do without, `tolerance` what another
correct fp32 implementation may differ by.

Kinds of case:
  dense_relu    Bounds.dense + relu: one layer of the op-by-op interface, latency at the small end
  tanh_dense    Bounds.tanh + dense: relaxation with bisections, then a wide layer, several perturbed words
  attention     Bounds.dot_product, multiply, softmax, context: the attention core of one or a few sentences
  hand_relu     c_bound.c_relu_verification: the drop-in entry point, transposed layout, caller-owned outputs
  hand_qk       c_bound.c_dot_product_verification_QK, likewise
  block         one encoder block operator by operator on Bounds, as the reference's verifier drives it
  encoder       EncoderVerifier.forward: the whole pass for a batch of sentences of one length
  instances     EncoderVerifier.forward_instances: one round of the radius search, a position and a radius per instance
  cnn           CnnVerifier.forward: an image with every pixel perturbed
  conv          ops.conv2d on dense dim_in rows (a shard of an image's pixels behind a first layer)
"""
import math
import types

import torch

import faith_b200
from faith_b200 import c_bound, ops
from faith_b200.sharded import CnnVerifier

DEV = "cuda:0"
INF = float("inf")
NORMS = {"1": 1.0, "2": 2.0, "inf": INF}
# Radius of a whole pass per norm: where a search for the certified radius starts.  (Much smaller ones say little about an
# implementation: the chord slopes of intervals a few ulps wide are rounding noise in any fp32 evaluation.)
RADIUS = {"1": 0.3, "2": 0.05, "inf": 0.005}


def listed():
    return [
        # A single layer of one short sentence: what an interactive user of the op-by-op interface waits for.
        {"name": "linear_relu_small", "kind": "dense_relu", "B": 1, "L": 16, "E": 64, "words": 1, "Do": 64, "Dy": 128,
         "p": "inf", "eps": 0.01},
        # A wide layer of a batch, four perturbed words, L1 ball (bandwidth of the relaxation, then a square product).
        {"name": "tanh_linear_wide", "kind": "tanh_dense", "B": 8, "L": 64, "E": 64, "words": 4, "Do": 256, "Dy": 256,
         "p": "1", "eps": 0.1},
        # Attention core of one sentence: 4 heads of 32 features, two perturbed words of 64 features, L2 ball.
        {"name": "attention_one", "kind": "attention", "S": 1, "H": 4, "L": 32, "E": 64, "words": 2, "d": 32, "p": "2",
         "eps": 0.05},
        # The reference's hand-tuned entry points at the upper and the middle part of its own sweep (L x dim_in x dim_out).
        {"name": "hand_relu_large", "kind": "hand_relu", "L": 128, "Di": 512, "Do": 256, "eps": 0.5},
        {"name": "hand_qk_mid", "kind": "hand_qk", "B": 4, "L": 32, "Di": 128, "K": 64, "eps": 0.5},
        # One encoder block of one sentence through Bounds, standard layer norm: a user who swapped the Bounds class in.
        {"name": "block_standard_norm", "kind": "block", "S": 1, "L": 32, "D": 128, "H": 4, "F": 512, "norm": "standard",
         "p": "inf", "eps": 0.001},
        # The whole model: one sentence (latency), sentences of an odd length with two perturbed words, the full batch.
        {"name": "encoder_one", "kind": "encoder", "S": 1, "L": 32, "words": 1, "p": "inf", "eps": 0.01, "first_only": False},
        {"name": "encoder_ragged", "kind": "encoder", "S": 24, "L": 21, "words": 2, "p": "2", "eps": 0.025, "first_only": False},
        {"name": "encoder_batch", "kind": "encoder", "S": 256, "L": 32, "words": 1, "p": "inf", "eps": 0.01,
         "first_only": False},
        # One round of the radius search over two sentences: every perturbable position with a radius of its own.
        {"name": "search_round", "kind": "instances", "S": 60, "L": 32, "words": 1, "p": "inf", "eps": 0.006},
        # One 3 x 32 x 32 image, every pixel perturbed.
        {"name": "cnn_image", "kind": "cnn", "C": 3, "HW": 32, "C1": 16, "C2": 32, "out": 10, "p": "inf", "eps": 2.0 / 255},
        # Second convolution of that network on dense rows, an eighth of dim_in.
        {"name": "conv_shard", "kind": "conv", "Di": 384, "C": 16, "HW": 32, "Co": 32, "k": 3, "stride": 2, "pad": 1},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["dense_relu", "tanh_dense", "attention", "hand_relu", "hand_qk", "block", "encoder", "encoder",
                       "encoder", "instances", "cnn", "conv"])
    p = rng.choice(["1", "2", "inf"])
    if kind in ("dense_relu", "tanh_dense"):
        while True:
            c = {"kind": kind, "B": _log(rng, 1, 16), "L": _log(rng, 4, 128), "E": rng.choice([32, 64, 128]),
                 "words": rng.choice([1, 1, 2, 4]), "Do": _log(rng, 32, 512), "Dy": _log(rng, 32, 512), "p": p, "eps": 0.05}
            rows = c["B"] * c["L"] * c["E"] * c["words"]
            if rows * max(c["Do"], c["Dy"]) <= 1 << 27:
                return c
    if kind == "attention":
        return {"kind": kind, "S": _log(rng, 1, 16), "H": rng.choice([2, 4]), "L": _log(rng, 6, 64), "E": 64,
                "words": rng.choice([1, 2]), "d": rng.choice([16, 32, 64]), "p": p, "eps": 0.02}
    if kind == "hand_relu":
        return {"kind": kind, "L": _log(rng, 2, 128), "Di": 32 * _log(rng, 2, 16), "Do": _log(rng, 64, 512), "eps": 0.5}
    if kind == "hand_qk":
        return {"kind": kind, "B": rng.choice([1, 2, 4]), "L": _log(rng, 2, 64), "Di": 32 * _log(rng, 2, 16),
                "K": _log(rng, 16, 256), "eps": 0.5}
    if kind == "block":
        return {"kind": kind, "S": 1, "L": _log(rng, 6, 48), "D": 128, "H": 4, "F": 512,
                "norm": rng.choice(["no_var", "standard"]), "p": p, "eps": 0.001}
    if kind == "encoder":
        words, L = rng.choice([1, 1, 2]), _log(rng, 8, 40)
        most = max(1, min(256, 4096 // (L * words)))
        return {"kind": kind, "S": _log(rng, 1, most), "L": L, "words": words, "p": p, "eps": RADIUS[p] / words,
                "first_only": rng.random() < 0.2}
    if kind == "instances":
        L = _log(rng, 8, 40)
        words = rng.choice([1, 1, 2])
        return {"kind": kind, "S": _log(rng, 4, max(8, 4096 // (L * words))), "L": L, "words": words, "p": p,
                "eps": RADIUS[p] / words}
    if kind == "cnn":
        return {"kind": kind, "C": rng.choice([1, 3]), "HW": rng.randint(16, 40), "C1": rng.choice([8, 16, 24]),
                "C2": rng.choice([16, 32, 48]), "out": rng.choice([2, 10, 16]), "p": p, "eps": 2.0 / 255}
    return {"kind": "conv", "Di": _log(rng, 16, 512), "C": rng.choice([3, 8, 16]), "HW": rng.randint(12, 40),
            "Co": rng.choice([8, 16, 32, 40]), "k": rng.choice([3, 3, 5]), "stride": rng.choice([1, 2]), "pad": 1}


# ------------------------------------------------------------------------------------------------ inputs
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _randn(g, *shape):
    return torch.randn(*shape, generator=g, device=DEV)


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device=DEV)


def _bounds(g, B, L, Di, Do, scale, gap):
    """A bound in the middle of a network: lines of slope ~ scale with a tenth of that between them, bias terms ~ N(0, 1)
    `gap` apart.  Returns lw, uw, lb, ub."""
    lw = _randn(g, B, L, Di, Do).mul_(scale)
    uw = lw + _rand(g, B, L, Di, Do).mul_(0.1 * scale)
    lb = _randn(g, B, L, Do)
    ub = lb + _rand(g, B, L, Do).mul_(gap)
    return lw, uw, lb, ub


def _sweep_bounds(g, B, L, Do, Di):
    """The distribution of the reference's kernel test, in the transposed layout of the drop-in module."""
    lb = _rand(g, B, L, Do) - 0.7
    ub = lb + _rand(g, B, L, Do)
    return lb, ub, (_rand(g, B, L, Do, Di) - 0.5).mul_(0.1), (_rand(g, B, L, Do, Di) - 0.5).mul_(0.1)


def _linear(g, out, inp, std):
    return types.SimpleNamespace(weight=_randn(g, out, inp) * std, bias=_randn(g, out) * std)


def _norm(g, D):
    return types.SimpleNamespace(weight=1.0 + 0.1 * _randn(g, D), bias=0.02 * _randn(g, D))


def _as_bounds(c, p, t, words=1):
    args = types.SimpleNamespace(method="forward", perturbed_words=words, current_flag=1)
    return faith_b200.Bounds(args, p, c["eps"], lw=t[0], uw=t[1], lb=t[2], ub=t[3])


def _model(g, layers=3, D=128, H=4, F=512, std=0.02):
    m = {"heads": H, "layer_norm": "no_var", "layers": []}

    def put(d, name, out, inp):
        lin = _linear(g, out, inp, std)
        d[name + "_w"], d[name + "_b"] = lin.weight, lin.bias

    def put_norm(d, name):
        n = _norm(g, D)
        d[name + "_g"], d[name + "_b"] = n.weight, n.bias
    put_norm(m, "emb_ln")
    for _ in range(layers):
        ly = {}
        for name, o, i in (("q", D, D), ("k", D, D), ("v", D, D), ("ao", D, D), ("f1", F, D), ("f2", D, F)):
            put(ly, name, o, i)
        put_norm(ly, "ln1")
        put_norm(ly, "ln2")
        m["layers"].append(ly)
    put(m, "pool", D, D)
    put(m, "cls", 2, D)
    return m


def prepare(case, seed):
    c, g, k = case, _gen(seed), case["kind"]
    s = types.SimpleNamespace(kind=k, case=c, p=NORMS[c.get("p", "2")])
    if k in ("dense_relu", "tanh_dense"):
        Di = c["E"] * c["words"]
        t = _bounds(g, c["B"], c["L"], Di, c["Do"], 1.0 / math.sqrt(Di), 0.05)
        s.x, s.lin = _as_bounds(c, s.p, t, c["words"]), _linear(g, c["Dy"], c["Do"], 1.0 / math.sqrt(c["Do"]))
    elif k == "attention":
        B, Di = c["S"] * c["H"], c["E"] * c["words"]
        s.q, s.k, s.v = (_as_bounds(c, s.p, _bounds(g, B, c["L"], Di, c["d"], 0.3 / Di, 0.01), c["words"]) for _ in range(3))
    elif k == "hand_relu":
        s.x = _sweep_bounds(g, 1, c["L"], c["Do"], c["Di"])
        s.out = tuple(torch.empty_like(t) for t in s.x)
    elif k == "hand_qk":
        B, L, K, Di = c["B"], c["L"], c["K"], c["Di"]
        s.x, s.y = _sweep_bounds(g, B, L, K, Di), _sweep_bounds(g, B, L, K, Di)
        s.ranges = tuple(torch.empty(B, L, K, device=DEV) for _ in range(4))
        s.out = (torch.empty(B, L, L, device=DEV), torch.empty(B, L, L, device=DEV), torch.empty(B, L, L, Di, device=DEV),
                 torch.empty(B, L, L, Di, device=DEV))
    elif k == "block":
        D, F = c["D"], c["F"]
        t = _bounds(g, c["S"], c["L"], D, D, 0.1 / D, 0.001)
        s.x = _as_bounds(c, s.p, t)
        s.wq, s.wk, s.wv, s.wo = (_linear(g, D, D, 0.02) for _ in range(4))
        s.f1, s.f2, s.ln1, s.ln2 = _linear(g, F, D, 0.02), _linear(g, D, F, 0.02), _norm(g, D), _norm(g, D)
    elif k in ("encoder", "instances"):
        s.ver = faith_b200.EncoderVerifier(_model(g), DEV, first_token_only=c.get("first_only", False))
        if k == "encoder":
            s.emb = _randn(g, c["S"], c["L"], 128)
            s.positions = [1 + 2 * w for w in range(c["words"])]
        else:
            # every instance is one (sentence, position) pair: the sentences repeat, positions run over 1 .. L - 2
            n = c["L"] - 2
            s.emb = _randn(g, -(-c["S"] // n), c["L"], 128).repeat_interleave(n, 0)[:c["S"]].contiguous()
            first = torch.arange(c["S"], device=DEV) % n
            s.positions = torch.stack([1 + (first + w) % n for w in range(c["words"])], 1).to(torch.int32).contiguous()
            s.eps = (_rand(g, c["S"]) * 0.5 + 0.5) * c["eps"]
    elif k == "cnn":
        ho = (c["HW"] + 2 - 3) // 2 + 1

        def kaiming(*shape):
            return _randn(g, *shape) * math.sqrt(2.0 / math.prod(shape[1:]))
        s.ver = CnnVerifier([("conv", kaiming(c["C1"], c["C"], 3, 3), 0.02 * _randn(g, c["C1"]), 1, 1), ("relu",),
                             ("conv", kaiming(c["C2"], c["C1"], 3, 3), 0.02 * _randn(g, c["C2"]), 2, 1), ("relu",),
                             ("linear", kaiming(c["out"], c["C2"] * ho * ho), 0.02 * _randn(g, c["out"]))], DEV)
        s.image = _rand(g, c["C"], c["HW"], c["HW"])
    else:
        shape = (1, c["Di"], c["C"], c["HW"], c["HW"])
        lw = _randn(g, *shape).mul_(0.1)
        lb = _randn(g, 1, *shape[2:])
        s.x = (lw, lw + _rand(g, *shape).mul_(0.01), lb, lb + _rand(g, 1, *shape[2:]).mul_(0.05))
        s.weight = _randn(g, c["Co"], c["C"], c["k"], c["k"]) * math.sqrt(2.0 / (c["C"] * c["k"] ** 2))
        s.bias = 0.02 * _randn(g, c["Co"])
    return s


# ------------------------------------------------------------------------------------------------ the calls
def _four(b):
    return b.lw, b.uw, b.lb, b.ub


def _split(x, heads):
    """The reference's head split (transpose_for_scores) of a bound [S, L, Di, H * d] -> [S * H, L, Di, d]."""
    z = ops.split_heads(_four(x), heads)
    return x._new(z[0], z[1], z[2], z[3])


def _merge(x, heads):
    z = ops.merge_heads(_four(x), heads)
    return x._new(z[0], z[1], z[2], z[3])


def run(s):
    c, k = s.case, s.kind
    if k == "dense_relu":
        return _four(s.x.dense(s.lin).relu())
    if k == "tanh_dense":
        return _four(s.x.tanh().dense(s.lin))
    if k == "attention":
        probs = s.q.dot_product(s.k).multiply(1.0 / math.sqrt(c["d"])).softmax()
        return _four(probs) + _four(probs.context(s.v))
    if k == "hand_relu":
        c_bound.c_relu_verification(*s.x, *s.out, c["L"], c["Di"], c["Do"], c["eps"])
        return s.out
    if k == "hand_qk":
        x_l, y_l, x_u, y_u = s.ranges
        x_lb, x_ub, x_lw, x_uw = s.x
        y_lb, y_ub, y_lw, y_uw = s.y
        c_bound.c_dot_product_verification_QK(x_l, y_l, x_u, y_u, x_lb, x_ub, y_lb, y_ub, x_lw, x_uw, y_lw, y_uw, *s.out,
                                              c["B"], c["L"], c["K"], c["Di"], c["eps"])
        return s.out + s.ranges
    if k == "block":
        q, key, v = (_split(s.x.dense(w), c["H"]) for w in (s.wq, s.wk, s.wv))
        probs = q.dot_product(key).multiply(1.0 / math.sqrt(c["D"] // c["H"])).softmax()
        h = _merge(probs.context(v), c["H"]).dense(s.wo).add(s.x).layer_norm(s.ln1, c["norm"])
        return _four(h.dense(s.f1).relu().dense(s.f2).add(h).layer_norm(s.ln2, c["norm"]))
    if k == "encoder":
        return s.ver.forward(s.emb, s.positions, s.p, c["eps"])
    if k == "instances":
        return s.ver.forward_instances(s.emb, s.positions, s.p, s.eps)
    if k == "cnn":
        return s.ver.forward(s.image, s.p, c["eps"])
    return ops.conv2d(s.x, s.weight, s.bias, c["stride"], c["pad"])


# ------------------------------------------------------------------------------------------------ what a call needs
def _gemm_flops(rows, K, N):
    """Split-sign product of `rows` bound rows: one product for the centres and one for the radii."""
    return 4.0 * rows * K * N


def _dot_flops(B, Lx, Ly, Di, K):
    """Bound times bound: six multiply-adds per term (centre and radius of x against the lower and the upper range of y,
    centre and radius of y against the range of x)."""
    return 12.0 * B * Lx * Ly * (Di + 1) * K


def _encoder_flops(S, L, Di, D, H, F, layers, first_only):
    f = 0.0
    for i in range(layers):
        rows = S * L * (Di + 1)
        q = rows / L if first_only and i == layers - 1 else rows    # rows behind the query side
        lq = 1 if first_only and i == layers - 1 else L
        # before the first relaxation the two lines coincide: one product, and only the perturbed positions' rows
        if i == 0:
            f += 3 * 2.0 * (S * (Di * (Di // D) + L)) * D * D
        else:
            f += _gemm_flops(q, D, D) + 2 * _gemm_flops(rows, D, D)
        f += _dot_flops(S * H, lq, L, Di, D // H) + _dot_flops(S * H, lq, D // H, Di, L)
        f += _gemm_flops(q, D, D) + 2 * _gemm_flops(q, D, F)
    return f + _gemm_flops(S * (Di + 1), D, D)


def _encoder_weight_bytes(D=128, F=512, layers=3):
    return 4.0 * (layers * (4 * D * D + 2 * D * F + F + 9 * D) + D * D + 6 * D)


def work(case):
    c, k = case, case["kind"]
    if k in ("dense_relu", "tanh_dense"):
        rows = c["B"] * c["L"] * (c["E"] * c["words"] + 1)
        return {"bytes": 4.0 * (2 * rows * (c["Do"] + c["Dy"]) + c["Do"] * c["Dy"] + c["Dy"]),
                "flops": _gemm_flops(rows, c["Do"], c["Dy"])}
    if k == "attention":
        B, Di, L, d = c["S"] * c["H"], c["E"] * c["words"], c["L"], c["d"]
        return {"bytes": 8.0 * B * L * (Di + 1) * (4 * d + L),
                "flops": _dot_flops(B, L, L, Di, d) + _dot_flops(B, L, d, Di, L)}
    if k == "hand_relu":
        rows = c["L"] * c["Do"] * (c["Di"] + 1)
        return {"bytes": 16.0 * rows, "flops": 4.0 * rows}
    if k == "hand_qk":
        B, L, K, Di = c["B"], c["L"], c["K"], c["Di"]
        return {"bytes": 4.0 * B * (4 * L * K * (Di + 1) + 2 * L * L * (Di + 1) + 4 * L * K), "flops": _dot_flops(B, L, L, Di, K)}
    if k == "block":
        S, L, D, H, F = c["S"], c["L"], c["D"], c["H"], c["F"]
        rows = S * L * (D + 1)
        return {"bytes": 4.0 * (4 * rows * D + 4 * D * D + 2 * D * F + F + 9 * D),
                "flops": 4 * _gemm_flops(rows, D, D) + 2 * _gemm_flops(rows, D, F) + _dot_flops(S * H, L, L, D, D // H)
                + _dot_flops(S * H, L, D // H, D, L)}
    if k in ("encoder", "instances"):
        return {"bytes": 4.0 * c["S"] * (c["L"] * 128 + 2) + _encoder_weight_bytes(),
                "flops": _encoder_flops(c["S"], c["L"], 128 * c["words"], 128, 4, 512, 3, c.get("first_only", False))}
    if k == "cnn":
        hw, ho = c["HW"], (c["HW"] + 2 - 3) // 2 + 1
        pix = c["C"] * hw * hw
        # a pixel reaches 3 x 3 outputs of the first convolution, each of those 9 / 4 outputs of the second, of which at
        # most 3 x 3 are distinct and go through the head
        conv1, conv2 = 9 * c["C1"], 9 * c["C1"] * c["C2"] * 2.25
        head = 4 * c["C2"] * c["out"]
        weights = 9 * c["C1"] * c["C"] + 9 * c["C1"] * c["C2"] + c["out"] * c["C2"] * ho * ho
        return {"bytes": 4.0 * (pix + weights + 2 * c["out"]), "flops": 4.0 * pix * (conv1 + conv2 + head)}
    ho = (c["HW"] + 2 * c["pad"] - c["k"]) // c["stride"] + 1
    rows = c["Di"] + 1
    return {"bytes": 4.0 * (2 * rows * (c["C"] * c["HW"] ** 2 + c["Co"] * ho * ho) + c["Co"] * c["C"] * c["k"] ** 2),
            "flops": 4.0 * rows * c["Co"] * ho * ho * c["C"] * c["k"] ** 2}


def tolerance(case):
    k = case["kind"]
    if k in ("encoder", "instances"):
        # rounding is amplified by every layer (chord slopes of narrow intervals): two fp32 evaluations of this pass with other
        # summation orders were seen 2e-4 apart in norm and 1e-3 in a single logit bound
        return {"rel": 1e-3, "max": 1e-2}
    if k == "tanh_dense":
        # a last-bit difference of a range moves a bisected tangent point by one step for a few columns
        return {"rel": 1e-4, "max": 1e-2}
    if k in ("block", "attention", "cnn"):
        return {"rel": 5e-5, "max": 2e-3}     # a chain of relaxations and products
    return {"rel": 1e-5, "max": 1e-3}
