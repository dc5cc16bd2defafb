"""Workloads that a user of this framework runs, for timing and for comparing two builds of it.

Four kinds of call, each through the public entry points:

* ``ortho``      one orthogonalization driver on a matrix or a batch (``dion_b200.ops.newton_schulz``);
* ``optimizer``  ``optimizer.step()`` on the parameters of a GPT with gradients in place;
* ``train``      a whole training step of the GPT model: forward, backward, optimizer step;
* ``logits``     the model without gradients: scores of given text, or the next-token logits that
                 ``GPT.generate`` computes for every token it appends.

``listed()`` are the cases to report, ``draw(rng)`` gives others of the same ranges, ``prepare`` /
``run`` execute one, ``work`` and ``tolerance`` say what a pass has to do and how closely two
correct implementations agree.
"""
import math

import torch

import dion_b200
from dion_b200.models.gpt import GPT, GPTConfig
from dion_b200.ops import newton_schulz as NS

DTYPES = {"bf16": torch.bfloat16, "fp32": torch.float32}
DRIVERS = {
    "quintic": NS.newton_schulz_quintic,
    "polar_express": NS.polar_express,
    "aol": NS.newton_schulz_aol,
    "gram": NS.gram_newton_schulz,
}
LR, SCALAR_LR, MU, WD = 0.02, 0.002, 0.95, 0.01


def listed():
    return [
        # One attention weight of GPT-160M orthogonalized on its own: launches and latency.
        {"name": "ortho_1x768x768", "op": "ortho", "driver": "polar_express", "batch": 1,
         "rows": 768, "cols": 768, "dtype": "bf16"},
        # A few fp32 gradients whose sides fit no tile or vector width.
        {"name": "ortho_6x997x1531", "op": "ortho", "driver": "polar_express", "batch": 6,
         "rows": 997, "cols": 1531, "dtype": "fp32"},
        # The MLP matrices of several GPT-160M models' worth of layers, wide, tuned quintic.
        {"name": "ortho_64x768x3072", "op": "ortho", "driver": "quintic", "batch": 64,
         "rows": 768, "cols": 3072, "dtype": "bf16"},
        # Tall MLP matrices of GPT-1B through the Gram-matrix driver.
        {"name": "ortho_gram_8x8192x2048", "op": "ortho", "driver": "gram", "batch": 8,
         "rows": 8192, "cols": 2048, "dtype": "bf16"},
        # A large square batch: throughput of the symmetric products.
        {"name": "ortho_16x4096x4096", "op": "ortho", "driver": "quintic", "batch": 16,
         "rows": 4096, "cols": 4096, "dtype": "bf16"},
        # Optimizer steps.  GPT-160M under Muon with fp32 master weights, AdamW for the rest.
        {"name": "muon_160m", "op": "optimizer", "algorithm": "muon", "width": 768, "layers": 12,
         "vocab": 50304, "dtype": "fp32", "scalar": "adamw", "fraction": 1.0},
        # GPT-1B under Dion2: a quarter of the rows, fp32 master weights.
        {"name": "dion2_1b", "op": "optimizer", "algorithm": "dion2", "width": 2048, "layers": 24,
         "vocab": 50304, "dtype": "fp32", "scalar": "adamw", "fraction": 0.25},
        # GPT-1B under NorMuon with bf16 parameters and state: the largest case.
        {"name": "normuon_1b", "op": "optimizer", "algorithm": "normuon", "width": 2048,
         "layers": 24, "vocab": 50304, "dtype": "bf16", "scalar": "adamw", "fraction": 1.0},
        # Four layers of GPT-1B under legacy Dion (rank 1/4), Lion for the rest.
        {"name": "dion_1b_4layers", "op": "optimizer", "algorithm": "dion", "width": 2048,
         "layers": 4, "vocab": 50304, "dtype": "fp32", "scalar": "lion", "fraction": 0.25},
        # A small model's training step: hundreds of short kernels.
        {"name": "train_small", "op": "train", "algorithm": "muon", "width": 256, "layers": 4,
         "heads": 4, "vocab": 50304, "batch": 8, "tokens": 256, "scalar": "adamw",
         "fraction": 1.0},
        # The headline training step: GPT-160M, Dion2, 32 sequences of 1024 tokens.
        {"name": "train_160m", "op": "train", "algorithm": "dion2", "width": 768, "layers": 12,
         "heads": 12, "vocab": 50304, "batch": 32, "tokens": 1024, "scalar": "adamw",
         "fraction": 0.25},
        # One step of sampling from GPT-160M: next-token logits of a short prompt.
        {"name": "sample_160m", "op": "logits", "width": 768, "layers": 12, "heads": 12,
         "vocab": 50304, "batch": 1, "tokens": 128, "all_positions": False},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _width(rng, lo, hi, step=64):
    """Model width: a multiple of 64 mostly, of 8 sometimes."""
    w = _log_int(rng, lo, hi)
    unit = step if rng.random() < 0.7 else 8
    return max(lo, w // unit * unit)


def draw(rng):
    op = rng.choices(["ortho", "optimizer", "train", "logits"], [5, 4, 2, 2])[0]
    if op == "ortho":
        rows, cols = _log_int(rng, 128, 6144), _log_int(rng, 128, 8192)
        if rng.random() < 0.6:           # weight shapes are mostly multiples of 64
            rows, cols = max(64, rows // 64 * 64), max(64, cols // 64 * 64)
        m, n = min(rows, cols), max(rows, cols)
        cap = max(1, int(1.2e13 / (5 * (3.0 * m * m * n + 1.0 * m ** 3))))
        return {"op": op, "driver": rng.choice(["quintic", "polar_express", "polar_express",
                                                "aol", "gram"]),
                "batch": min(_log_int(rng, 1, 64), cap), "rows": rows, "cols": cols,
                "dtype": rng.choice(["bf16", "fp32"])}
    if op == "optimizer":
        algorithm = rng.choice(["muon", "dion2", "normuon", "nordion2", "dion"])
        width = _width(rng, 256, 2048)
        most = 4 if algorithm == "dion" else 24
        return {"op": op, "algorithm": algorithm, "width": width,
                "layers": rng.randint(1, most), "vocab": rng.choice([50304, 50257, 32000, 8192]),
                "dtype": rng.choice(["fp32", "fp32", "bf16"]),
                "scalar": rng.choice(["adamw", "lion"]),
                "fraction": 1.0 if algorithm in ("muon", "normuon") else rng.choice([0.25, 0.5])}
    head_dim = rng.choice([64, 128])
    heads = _log_int(rng, 256, 1024) // head_dim
    case = {"op": op, "width": heads * head_dim, "layers": rng.randint(2, 12), "heads": heads,
            "vocab": rng.choice([50304, 50304, 32000, 8192])}
    tokens = _log_int(rng, 32, 1024)
    if op == "train":
        batch = min(_log_int(rng, 1, 32), max(1, 16384 // tokens))
        case.update(algorithm=rng.choice(["muon", "dion2", "normuon"]), batch=batch,
                    tokens=tokens, scalar=rng.choice(["adamw", "lion"]))
        case["fraction"] = 0.25 if case["algorithm"] == "dion2" else 1.0
    else:
        whole = rng.random() < 0.4
        batch = min(_log_int(rng, 1, 16), max(1, 4096 // tokens))
        case.update(batch=batch, tokens=tokens, all_positions=whole)
    return case


# ------------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------------
def _gradient(gen, shape, dtype, scale=1e-3):
    """Gradients have rows of different size: normal entries times a log-normal row factor."""
    g = torch.randn(shape, device="cuda", generator=gen)
    rows = torch.randn(tuple(shape[:-1]) + (1,), device="cuda", generator=gen)
    return g.mul_(rows.mul_(0.5).exp_().mul_(scale)).to(dtype)


def _shapes(case):
    d = case["width"]
    per_layer = [(d, d)] * 4 + [(4 * d, d), (d, 4 * d)]
    return per_layer * case["layers"], [(case["vocab"], d), (case["vocab"], d)]


def _flat_views(shapes, dtype):
    """One zeroed buffer and a view of it for every shape, each on a 256-byte boundary (weights
    and optimizer state kept in one allocation, as a program does that checkpoints them whole)."""
    sizes = [math.prod(s) for s in shapes]
    padded = [-(-n // 128) * 128 for n in sizes]
    flat = torch.zeros(sum(padded), dtype=dtype, device="cuda")
    views, at = [], 0
    for s, n, p in zip(shapes, sizes, padded):
        views.append(flat[at:at + n].view(s))
        at += p
    return flat, views


def _make_optimizer(case, matrices, scalars):
    head = dict(lr=SCALAR_LR / math.sqrt(case["width"]) if case["scalar"] == "lion" else SCALAR_LR)
    groups = [dict(params=matrices),
              dict(params=scalars[:1], algorithm=case["scalar"], lr=SCALAR_LR, weight_decay=0.0),
              dict(params=scalars[1:], algorithm=case["scalar"], weight_decay=0.0, **head)]
    name = case["algorithm"]
    if name == "dion":
        return dion_b200.Dion(groups, lr=LR, mu=MU, weight_decay=WD,
                              rank_fraction=case["fraction"])
    if name == "dion2":
        return dion_b200.Dion2(groups, lr=LR, ef_decay=MU, weight_decay=WD,
                               fraction=case["fraction"])
    if name == "nordion2":
        return dion_b200.NorDion2(groups, lr=LR, mu=MU, weight_decay=WD,
                                  fraction=case["fraction"])
    cls = dion_b200.Muon if name == "muon" else dion_b200.NorMuon
    return cls(groups, lr=LR, mu=MU, weight_decay=WD, nesterov=True)


def _resume(opt, matrices, scalars, gen=None):
    """Load optimizer state the way a resumed run does, from flat buffers (zeros, or values of a
    running training when ``gen`` is given).  -> {output name: flat buffer}"""
    sd = opt.state_dict()
    out = {}
    for kind, params, first in (("matrix", matrices, 0), ("scalar", scalars, len(matrices))):
        for key in sorted(k for k, v in sd["state"][first].items() if v.ndim >= 1):
            flat, views = _flat_views([sd["state"][first + i][key].shape
                                       for i in range(len(params))], params[0].dtype)
            if gen is not None:
                for i, (p, v) in enumerate(zip(params, views)):
                    if key == "momentum":
                        v.copy_(_gradient(gen, v.shape, v.dtype, 3e-3))
                    elif key == "variance":
                        v.copy_(_gradient(gen, v.shape, torch.float32, 1e-3).square_())
                    else:   # NorMuon's per-row second moment of an orthonormal update
                        v.copy_(torch.rand(v.shape, device="cuda", generator=gen).add_(0.5)
                                .div_(max(p.shape)))
            for i, v in enumerate(views):
                sd["state"][first + i][key] = v
            out[f"{key}_{kind}"] = flat
        if gen is not None:
            for i in range(len(params)):
                if "step_dev" in sd["state"][first + i]:
                    sd["state"][first + i]["step_dev"] = torch.full((), 100.0, device="cuda")
    opt.load_state_dict(sd)
    return out


def _prepare_optimizer(case, gen):
    dtype = DTYPES[case["dtype"]]
    mats, scals = _shapes(case)
    w_mat, mv = _flat_views(mats, dtype)
    w_sca, sv = _flat_views(scals, dtype)
    for v in mv:
        v.copy_(torch.randn(v.shape, device="cuda", generator=gen)
                .mul_(min(1.0, math.sqrt(v.shape[0] / v.shape[1])) / math.sqrt(v.shape[1])))
    for i, v in enumerate(sv):
        v.copy_(torch.randn(v.shape, device="cuda", generator=gen)
                .mul_(1.0 if i == 0 else 1.0 / math.sqrt(v.shape[1])))
    matrices = [torch.nn.Parameter(v) for v in mv]
    scalars = [torch.nn.Parameter(v) for v in sv]
    opt = _make_optimizer(case, matrices, scalars)
    grads = lambda: [_gradient(gen, p.shape, dtype) for p in matrices + scalars]  # noqa: E731
    outputs = {"weights_matrix": w_mat, "weights_scalar": w_sca}
    if case["algorithm"] == "dion":
        # This optimizer allocates its state in its first step and keeps it itself.
        for p, g in zip(matrices + scalars, grads()):
            p.grad = g
        opt.step()
    else:
        outputs.update(_resume(opt, matrices, scalars, gen))
    for p, g in zip(matrices + scalars, grads()):
        p.grad = g
    return {"case": case, "opt": opt, "params": matrices + scalars, "outputs": outputs}


def _make_model(case):
    model = GPT(GPTConfig(sequence_len=case["tokens"], vocab_size=case["vocab"],
                          n_layer=case["layers"], n_head=case["heads"], n_embd=case["width"]))
    return model


def _tokens(gen, case, extra):
    """Token ids with the skew of text: frequency falls off as one over the rank."""
    u = torch.rand((case["batch"], case["tokens"] + extra), device="cuda", generator=gen,
                   dtype=torch.float64)
    return (case["vocab"] ** u).long().sub_(1).clamp_(0, case["vocab"] - 1)


def _prepare_model(case, gen, seed):
    torch.manual_seed(seed)
    with torch.device("cuda"):
        model = _make_model(case)
    model.init_weights()
    matrices = list(model.transformer.h.parameters())
    scalars = list(model.transformer.wte.parameters()) + list(model.lm_head.parameters())
    if case["op"] == "logits":
        model.eval()
        extra = 1 if case["all_positions"] else 0
        ids = _tokens(gen, case, extra)
        state = {"case": case, "model": model, "x": ids[:, :case["tokens"]].contiguous()}
        if extra:
            state["y"] = ids[:, 1:].contiguous()
        return state
    outputs = {}
    for kind, params in (("matrix", matrices), ("scalar", scalars)):
        flat, views = _flat_views([p.shape for p in params], torch.float32)
        for p, v in zip(params, views):
            v.copy_(p.detach())
            p.data = v
        outputs[f"weights_{kind}"] = flat
    opt = _make_optimizer(case, matrices, scalars)
    outputs.update(_resume(opt, matrices, scalars))
    ids = _tokens(gen, case, 1)
    return {"case": case, "model": model, "opt": opt, "outputs": outputs,
            "x": ids[:, :-1].contiguous(), "y": ids[:, 1:].contiguous()}


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    torch.manual_seed(seed)
    if case["op"] == "ortho":
        shape = (case["rows"], case["cols"])
        if case["batch"] > 1:
            shape = (case["batch"],) + shape
        return {"case": case, "G": _gradient(gen, shape, DTYPES[case["dtype"]])}
    if case["op"] == "optimizer":
        return _prepare_optimizer(case, gen)
    return _prepare_model(case, gen, seed)


# ------------------------------------------------------------------------------------------------
# one pass
# ------------------------------------------------------------------------------------------------
def run(state):
    case = state["case"]
    op = case["op"]
    if op == "ortho":
        return DRIVERS[case["driver"]](state["G"])
    if op == "optimizer":
        state["opt"].step()
        if case["algorithm"] != "dion":
            return state["outputs"]
        # The low-rank factors themselves are defined up to the sign of each column (it depends
        # on rounding); their product is what weights and momentum receive.
        return {**state["outputs"],
                "momentum": [state["opt"].state[p]["momentum"] for p in state["params"]]}
    model = state["model"]
    if op == "train":
        with torch.autocast("cuda", dtype=torch.bfloat16):
            loss = model(state["x"], state["y"])
        loss.backward()
        state["opt"].step()
        model.zero_grad(set_to_none=True)
        return {"loss": loss.detach(), **state["outputs"]}
    with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
        return model(state["x"], state.get("y"), return_logits=True)


# ------------------------------------------------------------------------------------------------
# what a pass has to do, and how closely two correct implementations agree
# ------------------------------------------------------------------------------------------------
def _ortho_flops(rows, cols, iters=5, gram=False):
    """The two symmetric products of an iteration are needed as a half only.  The Gram driver
    iterates on the small matrix (four symmetric products a step) and touches the full one for
    two Gram matrices and two products."""
    m, n = float(min(rows, cols)), float(max(rows, cols))
    if gram:
        return 6 * m * m * n + 4 * iters * m ** 3
    return iters * (3 * m * m * n + m ** 3)


def _optimizer_work(case, element):
    mats, scals = _shapes(case)
    elems = float(sum(math.prod(s) for s in mats))
    scalar = float(sum(math.prod(s) for s in scals))
    # weights and momentum read and written, gradients read (AdamW: a second moment too)
    nbytes = element * (5 * elems + (7 if case["scalar"] == "adamw" else 5) * scalar)
    flops = 0.0
    for r, c in mats:
        m, n = min(r, c), max(r, c)
        if case["algorithm"] == "dion":
            k = math.ceil(case["fraction"] * m)
            flops += 8.0 * r * c * k + 8.5 * n * k * k
        else:
            k = math.ceil(case["fraction"] * m)
            flops += _ortho_flops(k, n)
    return nbytes, flops


def _model_flops(case, positions):
    """Forward pass: every token through the blocks, causal attention, the head on ``positions``
    rows."""
    d, t, rows = case["width"], case["tokens"], case["batch"] * case["tokens"]
    return (2.0 * 12 * d * d * case["layers"] * rows + 2.0 * t * d * case["layers"] * rows
            + 2.0 * d * case["vocab"] * positions)


def work(case):
    op = case["op"]
    if op == "ortho":
        numel = float(case["batch"] * case["rows"] * case["cols"])
        iters = 4 if case["driver"] == "aol" else 5
        return {"bytes": numel * ((2 if case["dtype"] == "bf16" else 4) + 2),
                "flops": case["batch"] * _ortho_flops(case["rows"], case["cols"], iters,
                                                      case["driver"] == "gram")}
    if op == "optimizer":
        nbytes, flops = _optimizer_work(case, 2 if case["dtype"] == "bf16" else 4)
        return {"bytes": nbytes, "flops": flops}
    rows = case["batch"] * case["tokens"]
    if op == "train":
        nbytes, flops = _optimizer_work(case, 4)
        return {"bytes": nbytes + 16.0 * rows, "flops": flops + 3 * _model_flops(case, rows)}
    positions = rows if case["all_positions"] else case["batch"]
    weights = 4.0 * (12 * case["width"] ** 2 * case["layers"] + case["vocab"] * case["width"])
    return {"bytes": weights + 4.0 * positions * case["vocab"] + 4.0 * rows * case["width"],
            "flops": _model_flops(case, positions)}


def tolerance(case):
    """Measured: five bf16 iterations are 0.5-1.4 % (2-norm) from the same iteration in fp64, so two
    correct ones may be 2-3 % apart; in weights and state that shrinks by the learning rate (0.2 %
    in bf16 weights at most, 0.05 % in fp32).  A training step started from zero state holds the
    bf16 gradients and the statistics of one update (1.1 %); bf16 logits are 0.7 % from fp32."""
    op = case["op"]
    if op == "ortho":
        return {"rel": 0.03, "max": 0.4}
    if op == "optimizer":
        return {"rel": 0.006, "max": 0.1}
    if op == "train":
        return {"rel": 0.02, "max": 0.4}
    return {"rel": 0.02, "max": 0.2}


# ------------------------------------------------------------------------------------------------
# the same outputs in 64 bits, in plain torch
# ------------------------------------------------------------------------------------------------
_QUINTIC = ((4.0848, -6.8946, 2.9270), (3.9505, -6.3029, 2.6377), (3.7418, -5.5913, 2.3037),
            (2.8769, -3.1427, 1.2046), (2.8366, -3.0525, 1.2012))
_POLAR = ((8.156554524902461, -22.48329292557795, 15.878769915207462),
          (4.042929935166739, -2.808917465908714, 0.5000178451051316),
          (3.8916678022926607, -2.772484153217685, 0.5060648178503393),
          (3.285753657755655, -2.3681294933425376, 0.46449024233003106),
          (2.3465413258596377, -1.7097828382687081, 0.42323551169305323))
_AOL = ((4.6051, -9.6552, 5.6769), (4.7505, -6.0861, 2.1790), (2.7763, -2.3190, 0.5523),
        (2.4231, -2.2861, 0.8193))


def _ortho64(G, driver, eps):
    """Newton-Schulz iteration of one matrix; the Gram driver is the same iteration reordered."""
    X = G.double()
    tall = X.size(0) > X.size(1)
    X = X.mT if tall else X
    coeffs, mult = (_QUINTIC, 1.0) if driver == "quintic" else (_POLAR, 1.02)
    if driver == "aol":
        coeffs = _AOL
        X = X * (X @ X.mT).abs().sum(dim=-1, keepdim=True).clamp_min(eps).rsqrt()
    else:
        X = X / (X.norm() * mult + eps)
    for a, b, c in coeffs:
        A = X @ X.mT
        X = a * X + (b * A + c * (A @ A)) @ X
    return X.mT if tall else X


def _split(flat, shapes):
    views, at = [], 0
    for s in shapes:
        n = math.prod(s)
        views.append(flat[at:at + n].view(s))
        at += -(-n // 128) * 128
    return views


def _update64(case, out, shapes, grads, steps):
    """One optimizer step on the flat fp64 buffers ``out`` (weights and state), in place."""
    mats, scals = shapes
    w, m = _split(out["weights_matrix"], mats), _split(out["momentum_matrix"], mats)
    v = None
    if case["algorithm"] == "normuon":
        key = next(k for k in out if k.startswith("variance") and k.endswith("_matrix"))
        v = _split(out[key], [(r, 1) for r, _ in mats])
    for i, (rows, cols) in enumerate(mats):
        W, M, G = w[i], m[i], grads[i].double()
        ratio = math.sqrt(rows / cols)
        if case["algorithm"] == "dion2":
            dim = 0 if rows <= cols else 1
            M.add_(G)
            k = math.ceil(case["fraction"] * M.size(dim))
            sel = M.abs().sum(dim=1 - dim).topk(k).indices.sort().values
            U = _ortho64(M.index_select(dim, sel), "polar", 1e-8)
            full = torch.zeros_like(M).index_copy_(dim, sel, U)
            M.index_copy_(dim, sel, M.index_select(dim, sel) * MU)
        else:
            M.mul_(MU).add_(G)
            full = _ortho64(MU * M + G, "polar", 1e-8)
            if v is not None:
                before = full.norm()
                v[i].lerp_(full.square().mean(dim=1, keepdim=True), 0.05)
                full = full / (v[i].sqrt() + 1e-8)
                full = full * (before / full.norm())
        W.mul_(1 - LR * WD).sub_(full, alpha=LR * ratio)
    w, m = _split(out["weights_scalar"], scals), _split(out["momentum_scalar"], scals)
    for i in range(len(scals)):
        W, M, G = w[i], m[i], grads[len(mats) + i].double()
        if case["scalar"] == "lion":
            lr = SCALAR_LR if i == 0 else SCALAR_LR / math.sqrt(case["width"])
            W.sub_(torch.lerp(M, G, 0.1).sign_(), alpha=lr)
            M.lerp_(G, 0.05)
        else:
            V = _split(out["variance_scalar"], scals)[i]
            M.lerp_(G, 0.1)
            V.lerp_(G.square(), 0.05)
            W.sub_(SCALAR_LR * (M / (1 - 0.9 ** steps))
                   / ((V / (1 - 0.95 ** steps)).sqrt_() + 1e-8))
    return out


def _norm64(x, eps):
    return x * (x.square().mean(dim=-1, keepdim=True) + eps).rsqrt()


def _hidden64(weights, embedding, ids, heads):
    """Residual stream of the GPT after its last norm; norms use the epsilon of their input's
    data type (fp32 residual stream, bf16 queries and keys)."""
    x = embedding[ids]
    B, T, C = x.shape
    D = C // heads
    inv = 10000.0 ** (-torch.arange(0, D, 2, device="cuda", dtype=torch.float64) / D)
    ang = torch.outer(torch.arange(T, device="cuda", dtype=torch.float64), inv)
    cos, sin = ang.cos(), ang.sin()

    def rope(t):
        a, b = t[..., :D // 2], t[..., D // 2:]
        return _norm64(torch.cat([a * cos + b * sin, b * cos - a * sin], dim=-1), 2.0 ** -7)

    mask = torch.ones(T, T, dtype=torch.bool, device="cuda").triu(1)
    for q, k, v, o, fc, proj in weights:
        h = _norm64(x, 2.0 ** -23)
        q, k, v = ((h @ W.mT).view(B, T, heads, D).transpose(1, 2) for W in (q, k, v))
        s = (rope(q) @ rope(k).mT / math.sqrt(D)).masked_fill(mask, -math.inf)
        y = (s.softmax(dim=-1) @ v).transpose(1, 2).reshape(B, T, C)
        x = x + y @ o.mT
        x = x + (_norm64(x, 2.0 ** -23) @ fc.mT).relu().square() @ proj.mT
    return _norm64(x, 2.0 ** -23)


def _weights64(model, grad):
    mats = [p.detach().double().requires_grad_(grad) for p in model.transformer.h.parameters()]
    scals = [p.detach().double().requires_grad_(grad)
             for p in (model.transformer.wte.weight, model.lm_head.weight)]
    return mats, scals, [mats[i:i + 6] for i in range(0, len(mats), 6)]


def exact(case, seed):
    op = case["op"]
    if case.get("algorithm") in ("dion", "nordion2"):
        return None   # a sketch drawn on the device; rows selected and normalized together
    state = prepare(case, seed)
    if op == "ortho":
        G = state["G"]
        one = lambda g: _ortho64(g, case["driver"],  # noqa: E731
                                 1e-7 if case["driver"] in ("quintic", "aol") else 1e-6)
        return one(G) if G.ndim == 2 else torch.stack([one(g) for g in G])
    if op == "optimizer":
        grads = [p.grad for p in state["params"]]
        out = {k: t.double() for k, t in state["outputs"].items()}
        return _update64(case, out, _shapes(case), grads, 101)
    mats, scals, blocks = _weights64(state["model"], op == "train")
    if op == "logits":
        h = _hidden64(blocks, scals[0], state["x"], case["heads"])
        return (h if "y" in state else h[:, -1:]) @ scals[1].mT
    total, rows = 0.0, max(1, 4096 // case["tokens"])
    count = state["y"].numel()
    for x, y in zip(state["x"].split(rows), state["y"].split(rows)):
        h = _hidden64(blocks, scals[0], x, case["heads"])
        loss = torch.nn.functional.cross_entropy((h @ scals[1].mT).flatten(0, 1), y.flatten(),
                                                 reduction="sum") / count
        loss.backward()
        total = total + loss.detach()
    out = {k: t.double() for k, t in state["outputs"].items()}
    shapes = [tuple(p.shape) for p in mats], [tuple(p.shape) for p in scals]
    grads = [p.grad for p in mats + scals]
    return {"loss": total, **_update64(case, out, shapes, grads, 1)}
