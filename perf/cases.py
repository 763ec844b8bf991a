"""The work that a user of this framework has it do, as measurable cases.

    matmul   one linear layer over rows that are on the device (DeviceOps.qmatmul), GGUF weights in the three formats, with
             quantised ("q8") or fp32 ("f32") activations
    decode   one token for each of `batch` sequences over a filled cache (Decoder.step)
    verify   the drafted tokens of one sequence, every row's logits (Decoder.forward_logits)
    prompt   a prompt in one call (Decoder.forward_last_logits)
    layered  a layered decoder served in bfloat16 (LayeredDecoder): its prompt pass, or short prompts of several sequences
             followed by steps for all of them

Model shapes are the two decoder configurations of `sharpmind_b200.synth` and the layered decoder of benchmark sizes;
weights are random, blocks are made here by a plain block quantiser.
"""
import math
import random

import torch

from sharpmind_b200 import layered, ops, synth
from sharpmind_b200.decoder import Decoder

FMT = {"q8_0": 8, "q4_k": 12, "q6_k": 14}
BYTES = {"q8_0": 34 / 32, "q4_k": 144 / 256, "q6_k": 210 / 256}
NAME = {v: k for k, v in FMT.items()}
MODE = {"q8": ops.Mode.ACT_Q8, "f32": ops.Mode.ACT_F32}
SHAPES = {"0.6b": synth.QWEN3_0_6B, "8b": synth.LLAMA3_8B}
MATRICES = {"q8_0": [(3072, 1024), (6144, 1024), (1024, 3072), (4096, 1024)], "q4_k": [(28672, 4096), (4096, 4096), (6144, 4096), (8192, 28672)],
            "q6_k": [(4096, 14336), (1024, 4096), (8192, 28672)]}
# layered decoder: width, layers, ffn, vocab, heads, window
LAYERED = {"w1024": (1024, 16, 3072, 32000, 8, 1024), "w2048": (2048, 16, 5632, 32000, 16, 1024)}


def listed():
    return [
        # one decoded token through the smallest linear layer: latency and launches
        {"name": "row-q8_0-small", "kind": "matmul", "fmt": "q8_0", "n": 3072, "k": 1024, "rows": 1, "mode": "q8"},
        # one decoded token through a large feed-forward matrix: the weight stream
        {"name": "row-q4_k", "kind": "matmul", "fmt": "q4_k", "n": 28672, "k": 4096, "rows": 1, "mode": "q8"},
        # the same matrix for 32 sequences that decode together
        {"name": "rows32-q4_k", "kind": "matmul", "fmt": "q4_k", "n": 28672, "k": 4096, "rows": 32, "mode": "q8"},
        # a prompt through a down projection with fp32 activations, the default of a linear layer; a ragged number of rows
        {"name": "rows500-q6_k-f32", "kind": "matmul", "fmt": "q6_k", "n": 4096, "k": 14336, "rows": 500, "mode": "f32"},
        # a chat of one sequence with a small and with an ordinary model
        {"name": "decode-0.6b", "kind": "decode", "model": "0.6b", "batch": 1, "ctx": 2048, "kv": "f32", "mode": "q8"},
        {"name": "decode-8b", "kind": "decode", "model": "8b", "batch": 1, "ctx": 2048, "kv": "f32", "mode": "q8"},
        # a server's step for 32 sequences with quantised caches
        {"name": "decode-0.6b-batch32", "kind": "decode", "model": "0.6b", "batch": 32, "ctx": 1501, "kv": "q8_0", "mode": "q8"},
        # five drafted tokens and the last accepted one
        {"name": "verify-8b", "kind": "verify", "model": "8b", "rows": 6, "ctx": 1021, "kv": "f32", "mode": "q8"},
        # long prompt of the small model; ordinary, ragged prompt of the other
        {"name": "prompt-0.6b", "kind": "prompt", "model": "0.6b", "rows": 2048, "kv": "f32", "mode": "q8"},
        {"name": "prompt-8b", "kind": "prompt", "model": "8b", "rows": 777, "kv": "f32", "mode": "q8"},
        # a layered decoder: a long prompt; eight short requests and their first tokens
        {"name": "layered-prompt", "kind": "layered", "model": "w2048", "batch": 1, "rows": 2048, "steps": 0},
        {"name": "layered-serve", "kind": "layered", "model": "w1024", "batch": 8, "rows": 96, "steps": 8},
    ]


def _spread(rng, lo, hi):
    """A whole number of [lo, hi], spread over its logarithm."""
    return min(hi, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))


def draw(rng: random.Random):
    kind = rng.choice(["matmul", "matmul", "decode", "decode", "verify", "prompt", "layered"])
    if kind == "matmul":
        fmt = rng.choice(sorted(FMT))
        n, k = rng.choice(MATRICES[fmt])
        return {"kind": kind, "fmt": fmt, "n": n, "k": k, "rows": _spread(rng, 1, 600), "mode": rng.choice(["q8", "q8", "f32"])}
    model, kv = rng.choice(["0.6b", "8b"]), rng.choice(["f32", "q8_0"])
    mode = rng.choice(["q8", "q8", "q8", "f32"]) if model == "0.6b" else "q8"
    if kind == "decode":
        return {"kind": kind, "model": model, "batch": _spread(rng, 1, 32), "ctx": _spread(rng, 16, 2200), "kv": kv, "mode": mode}
    if kind == "verify":
        return {"kind": kind, "model": model, "rows": _spread(rng, 2, 16), "ctx": _spread(rng, 16, 2200), "kv": kv, "mode": mode}
    if kind == "prompt":
        return {"kind": kind, "model": model, "rows": _spread(rng, 17, 2048 if model == "0.6b" else 777), "kv": kv, "mode": mode}
    if rng.random() < 0.5:
        return {"kind": kind, "model": rng.choice(sorted(LAYERED)), "batch": 1, "rows": _spread(rng, 32, 2048), "steps": 0}
    return {"kind": kind, "model": "w1024", "batch": _spread(rng, 1, 16), "rows": _spread(rng, 8, 128), "steps": rng.randint(2, 8)}


# ------------------------------------------------------------------------------------------------ inputs from the seed
def _gen(seed, *tag):
    key = seed
    for t in tag:
        key = (key * 1000003 + t + 1) % (1 << 62)
    return torch.Generator(device="cuda").manual_seed(key)


def _randn(shape, seed, *tag):
    return torch.randn(shape, generator=_gen(seed, *tag), device="cuda")


def _div(a, b):
    """a / b with 0 where b is 0."""
    return torch.where(b > 0, a / torch.where(b > 0, b, torch.ones_like(b)), torch.zeros_like(a))


def _blocks(fmt, v, values):
    """fp32 matrix -> its GGUF blocks as bytes, or (values) the numbers that the blocks stand for, in 64 bits."""
    u8 = torch.uint8
    if fmt == "q8_0":
        v = v.reshape(-1, 32)
        d = (v.abs().amax(-1, keepdim=True) / 127).half()
        q = _div(v, d.float()).round_().clamp_(-127, 127).to(torch.int8)
        return d.double() * q.double() if values else torch.cat([d.view(u8), q.view(u8)], 1).reshape(-1)
    if fmt == "q4_k":
        v = v.reshape(-1, 8, 32)
        low = v.amin(-1).clamp_(max=0)
        sc, mn = (v.amax(-1) - low) / 15, -low
        d, dm = (sc.amax(-1, keepdim=True) / 63).half(), (mn.amax(-1, keepdim=True) / 63).half()
        s6, m6 = _div(sc, d.float()).round_().clamp_(0, 63), _div(mn, dm.float()).round_().clamp_(0, 63)
        q = _div(v + (dm.float() * m6)[..., None], (d.float() * s6)[..., None]).round_().clamp_(0, 15)
        if values:
            return (d.double() * s6.double())[..., None] * q.double() - (dm.double() * m6.double())[..., None]
        s, m, q = s6.to(u8), m6.to(u8), q.to(u8).reshape(-1, 4, 2, 32)
        head = torch.cat([s[:, :4] | (s[:, 4:] >> 4) << 6, m[:, :4] | (m[:, 4:] >> 4) << 6, (s[:, 4:] & 15) | (m[:, 4:] & 15) << 4], 1)
        return torch.cat([d.view(u8), dm.view(u8), head, (q[:, :, 0] | q[:, :, 1] << 4).reshape(-1, 128)], 1).reshape(-1)
    v = v.reshape(-1, 16, 16)
    sc = v.abs().amax(-1) / 31
    d = (sc.amax(-1, keepdim=True) / 127).half()
    s8 = _div(sc, d.float()).round_().clamp_(0, 127)
    q = _div(v, (d.float() * s8)[..., None]).round_().clamp_(-32, 31)
    if values:
        return (d.double() * s8.double())[..., None] * q.double()
    q = (q + 32).to(u8).reshape(-1, 2, 4, 32)
    lo, hi = q & 15, q >> 4
    ql = torch.stack([lo[:, :, 0] | lo[:, :, 2] << 4, lo[:, :, 1] | lo[:, :, 3] << 4], 2).reshape(-1, 128)
    qh = (hi[:, :, 0] | hi[:, :, 1] << 2 | hi[:, :, 2] << 4 | hi[:, :, 3] << 6).reshape(-1, 64)
    return torch.cat([ql, qh, s8.to(torch.int8).view(u8), d.view(u8)], 1).reshape(-1)


def _matrix(fmt, n, k, values, seed, *tag):
    b = _blocks(fmt, _randn((n, k), seed, *tag).mul_(0.02), values)
    return b.reshape(n, k) if values else b


def _vector(n, seed, *tag):
    return 1.0 + 0.1 * _randn((n,), seed, *tag)


def _tokens(vocab, n, seed, *tag):
    return torch.randint(0, vocab, (n,), generator=_gen(seed, *tag), device="cuda", dtype=torch.int32)


def _decoder_config(case):
    cfg = dict(SHAPES[case["model"]], kv_dtype=8 if case["kv"] == "q8_0" else 0)
    return cfg


def _decoder_shapes(cfg):
    H, hd, F, dt = cfg["hidden"], cfg["head_dim"], cfg["ffn"], NAME[cfg["dtype"]]
    q, kv = cfg["n_heads"] * hd, cfg["n_kv_heads"] * hd
    return {"wq": (dt, q, H), "wk": (dt, kv, H), "wv": (dt, kv, H), "wo": (dt, H, q), "wgu": (dt, 2 * F, H),
            "wdown": (NAME[cfg.get("down_dtype") or cfg["dtype"]], H, F)}


def _decoder_weights(cfg, layer, values, seed):
    """One layer's matrices (bytes or values) and norm vectors."""
    w = {name: _matrix(fmt, n, k, values, seed, layer, i) for i, (name, (fmt, n, k)) in enumerate(_decoder_shapes(cfg).items())}
    for i, name in enumerate(("norm1", "norm2", "qnorm", "knorm")):
        w[name] = _vector(cfg["hidden"] if i < 2 else cfg["head_dim"], seed, layer, 10 + i)
    return w


def _cache(cfg, case, layer, seed):
    shape = (case.get("batch", 1), cfg["n_kv_heads"], case["ctx"], cfg["head_dim"])
    return _randn(shape, seed, layer, 20), _randn(shape, seed, layer, 21)


def _layered_config(case):
    H, L, F, V, heads, window = LAYERED[case["model"]]

    def decays(n):
        return [1.0 - 2.0 ** (-3.0 - 6.0 * i / n) for i in range(n)]

    light = {"heads": heads, "dim": 128, "vdim": 128, "decay": decays(heads)}
    both = {"left": {"heads": heads, "kv_heads": heads // 4, "dim": 128, "vdim": 128, "mask": {"size": window}, "scale": 128 ** -0.5, "bias_max": window},
            "right": {"heads": heads // 2, "dim": 128, "vdim": 128, "rot": {"base": 10000.0, "dims": 128}, "decay": decays(heads // 2)},
            "left_scale": 0.7, "right_scale": 0.7}
    layers = [{"type": ("lightning", "parallel")[i & 1], "mixer": (light, both)[i & 1], "mlp": {"kind": "dense", "ff": F}} for i in range(L)]
    return layered.read_config({"architecture": "Molopel", "vocab": V, "width": H, "norm": {"eps": 1e-5}, "embedding": {"scale": 1.0},
                                "logit_softcap": 30.0, "layers": layers})


class _LayeredTensors:
    """Random tensors of a layered configuration by name, matrices in bfloat16."""

    def __init__(self, cfg, seed):
        self.shapes = {k: tuple(32 if n is None else n for n in v) for k, v in layered.tensor_shapes(cfg).items()}
        self.index, self.seed = {k: i for i, k in enumerate(self.shapes)}, seed

    def __getitem__(self, name):
        shape = self.shapes[name]
        x = _randn(shape, self.seed, self.index[name])
        if len(shape) == 1:
            x = (0.0 if name.endswith(".b") else 1.0) + 0.1 * x
        else:
            x = x * shape[1] ** -0.5
        return x.to(torch.bfloat16)


class _State:
    """What a user's program holds; gives the device memory back when it goes."""

    def __init__(self, case):
        self.case, self.ctx, self.model, self.weights = case, ops.CudaContext(0), None, []

    def __del__(self):
        torch.cuda.synchronize()
        if self.model is not None:
            self.model.close()
        for w in self.weights:
            self.ctx.release(w)
        self.ctx.close()


def prepare(case, seed):
    st = _State(case)
    ctx, kind = st.ctx, case["kind"]
    if kind == "matmul":
        st.ops = ops.DeviceOps(ctx)
        raw = _matrix(case["fmt"], case["n"], case["k"], False, seed, 0)
        st.w = ctx.register_dev(raw, FMT[case["fmt"]], case["n"], case["k"])
        st.weights.append(st.w)
        st.x = _randn((case["rows"], case["k"]), seed, 1)
    elif kind == "layered":
        cfg = _layered_config(case)
        st.model = layered.LayeredDecoder(ctx, cfg, _LayeredTensors(cfg, seed), max_batch=case["batch"],
                                          max_seq=case["rows"] + case["steps"] + 16, max_chunk=case["rows"])
        st.tokens = _tokens(cfg["vocab"], case["batch"] * (case["rows"] + case["steps"]), seed, 999).reshape(-1, case["batch"])
        st.prompts = st.tokens[:case["rows"]].t().contiguous()
        st.last = torch.tensor([case["rows"] - 1], dtype=torch.int32, device="cuda")
    else:
        cfg = _decoder_config(case)
        keys, w = list(_decoder_shapes(cfg)), {}
        for i in range(cfg["n_layers"]):
            for name, t in _decoder_weights(cfg, i, False, seed).items():
                if name in keys:  # registered one by one: the bytes need not wait for the whole model
                    fmt, n, k = _decoder_shapes(cfg)[name]
                    t = ctx.register_dev(t, FMT[fmt], n, k)
                    st.weights.append(t)
                w.setdefault(name, []).append(t)
        head = NAME[cfg.get("head_dtype") or cfg["dtype"]]
        w["embedding"] = ctx.register_dev(_matrix(head, cfg["vocab"], cfg["hidden"], False, seed, 500), FMT[head], cfg["vocab"], cfg["hidden"])
        st.weights.append(w["embedding"])
        w["final_norm"] = _vector(cfg["hidden"], seed, 501)
        st.model = Decoder(ctx, cfg, w, max_batch=case.get("batch", 1))
        if kind != "prompt":
            layers = [_cache(cfg, case, i, seed) for i in range(cfg["n_layers"])]
            st.model.load_kv(torch.stack([k for k, _ in layers]), torch.stack([v for _, v in layers]))
        st.tokens = _tokens(cfg["vocab"], case["batch"] if kind == "decode" else case["rows"], seed, 502)
    torch.cuda.synchronize()
    return st


def run(state):
    case, m = state.case, state.model
    if case["kind"] == "matmul":
        return state.ops.qmatmul(state.x, state.w, MODE[case["mode"]])
    if case["kind"] == "decode":
        return m.step(state.tokens, case["ctx"], MODE[case["mode"]])[0]
    if case["kind"] == "verify":
        return m.forward_logits(state.tokens, case["ctx"], 0, MODE[case["mode"]])[0]
    if case["kind"] == "prompt":
        return m.forward_last_logits(state.tokens, 0, 0, MODE[case["mode"]])[0]
    first = []
    for i in range(case["batch"]):
        m.reset_sequence(i)
        first.append(m.forward_rows(state.prompts[i], 0, i, state.last))
    steps = [m.step(state.tokens[case["rows"] + s], layered.POS_NEXT)[0] for s in range(case["steps"])]
    return first + steps


# ----------------------------------------------------------------------------------------------------------- work
def _decoder_work(cfg, case, rows, head_rows):
    params = {name: n * k for name, (_, n, k) in _decoder_shapes(cfg).items()}
    nbytes = cfg["n_layers"] * sum(n * k * BYTES[fmt] for fmt, n, k in _decoder_shapes(cfg).values())
    nbytes += cfg["vocab"] * cfg["hidden"] * BYTES[NAME[cfg.get("head_dtype") or cfg["dtype"]]]
    per_pos = 2 * cfg["n_kv_heads"] * cfg["head_dim"] * (34 / 32 if case["kv"] == "q8_0" else 4)
    kind, ctx = case["kind"], case.get("ctx", 0)
    read = rows * ctx if kind == "decode" else ctx
    nbytes += cfg["n_layers"] * per_pos * (read + rows) + 4 * head_rows * cfg["vocab"]
    pairs = rows * (ctx + 1) if kind == "decode" else rows * ctx + rows * (rows + 1) / 2
    flops = 2 * rows * cfg["n_layers"] * sum(params.values()) + 2 * head_rows * cfg["vocab"] * cfg["hidden"]
    flops += cfg["n_layers"] * 4 * pairs * cfg["n_heads"] * cfg["head_dim"]
    return {"bytes": int(nbytes), "flops": int(flops)}


def work(case):
    kind = case["kind"]
    if kind == "matmul":
        M, N, K = case["rows"], case["n"], case["k"]
        return {"bytes": int(N * K * BYTES[case["fmt"]]) + 4 * M * (N + K), "flops": 2 * M * N * K}
    if kind != "layered":
        rows = case["batch"] if kind == "decode" else case["rows"]
        return _decoder_work(_decoder_config(case), case, rows, 1 if kind == "prompt" else rows)
    H, L, F, V, heads, window = LAYERED[case["model"]]
    n, B, T, S = heads * 128, case["batch"], case["rows"], case["steps"]
    light, both = 5 * H * n, H * (n + n // 2 + 4 * (n // 2)) + H * (n + n // 2)
    params = L * 3 * H * F + L // 2 * (light + both)
    state = L // 2 * (n * 128 * 4 + n // 2 * 128 * 4)  # fp32 states of one sequence, read and written by every step
    ring = L // 2 * 2 * (n // 4) * 2 * min(window, T)
    passes = B + S  # every prompt and every step reads the weights
    span = sum(min(i + 1, window) for i in range(T))
    flops = B * (T + S) * 2 * params + B * (1 + S) * 2 * V * H + B * L // 2 * (4 * n * span + 1.5 * 4 * n * 128 * T)
    return {"bytes": int(passes * 2 * (params + V * H) + B * S * (2 * state + ring) + 4 * B * (1 + S) * V), "flops": int(flops)}


# ---------------------------------------------------------------------------------------- tolerances and 64-bit results
def tolerance(case):
    """About four times what is measured against `exact`.  Single matmuls: fp32 sums of exact products.  Models with quantised
    activations: where another order of fp32 sums moves an activation across the border between two codes, the step of 1/127
    of its block's largest value travels on through the layers.  fp32 models over a quantised cache: the new rows' codes
    alone.  Layered models: bfloat16 operands."""
    if case["kind"] == "matmul":
        return {"rel": 5e-6}
    if case["kind"] == "layered":
        return {"rel": 1e-1}
    if case["mode"] == "f32":
        return {"rel": 1e-5 if case["kv"] == "f32" else 3e-2}
    return {"rel": 4e-1}


def _q8_rows(x):
    """Rows as the quantised activations stand for them: 32-element blocks, scale amax / 127 kept in fp16, codes from the
    unrounded scale."""
    b = x.float().reshape(-1, 32)
    top = b.abs().amax(-1, keepdim=True)
    d = torch.where(top > 0, top / torch.full_like(top, 127.0), torch.ones_like(top))  # a tensor: torch divides by a number through its reciprocal
    return ((b / d).round().clamp(-128, 127).double() * d.half().double()).reshape(x.shape)


def _unit(x, eps):
    return x / (x.square().mean(-1, keepdim=True) + eps).sqrt()


def _rope(x, pos, theta, neox):
    """x [rows, heads, dim]; angles in fp32, as the tables define them."""
    h = x.shape[-1] // 2
    f = 1.0 / torch.tensor(theta, device="cuda") ** (2.0 * torch.arange(h, device="cuda").float() / x.shape[-1])
    a = (pos.float()[:, None] * f[None]).double()[:, None]
    u, v = (x[..., :h], x[..., h:]) if neox else (x[..., 0::2], x[..., 1::2])
    u, v = u * a.cos() - v * a.sin(), v * a.cos() + u * a.sin()
    return torch.cat([u, v], -1) if neox else torch.stack([u, v], -1).flatten(-2)


def _embedding_rows(cfg, tokens, seed):
    """The chosen rows of the table, and the table in 64 bits (which is also the head)."""
    head = NAME[cfg.get("head_dtype") or cfg["dtype"]]
    table = _matrix(head, cfg["vocab"], cfg["hidden"], True, seed, 500)
    return table[tokens.long()], table


def _exact_decoder(case, seed):
    """The model's function; in a quantised mode every matmul's input is rounded as the mode says, and cache rows as they are
    kept."""
    cfg, kind = _decoder_config(case), case["kind"]
    rows = case["batch"] if kind == "decode" else case["rows"]
    nh, kvh, hd, eps, F = cfg["n_heads"], cfg["n_kv_heads"], cfg["head_dim"], cfg["eps"], cfg["ffn"]
    x, table = _embedding_rows(cfg, _tokens(cfg["vocab"], rows, seed, 502), seed)
    ctx = case.get("ctx", 0)
    pos = torch.full((rows,), ctx, device="cuda") if kind == "decode" else ctx + torch.arange(rows, device="cuda")
    keep = _q8_rows if case["kv"] == "q8_0" else (lambda t: t)
    act = _q8_rows if case["mode"] == "q8" else (lambda t: t)
    for i in range(cfg["n_layers"]):
        w = _decoder_weights(cfg, i, True, seed)
        h = act(_unit(x, eps) * w["norm1"])
        q, k, v = (h @ w[n].T for n in ("wq", "wk", "wv"))
        q, k, v = q.reshape(rows, nh, hd), k.reshape(rows, kvh, hd), v.reshape(rows, kvh, hd)
        if cfg["qk_norm"]:
            q, k = _unit(q, eps) * w["qnorm"], _unit(k, eps) * w["knorm"]
        q, k = _rope(q, pos, cfg["rope_theta"], cfg["neox"]), _rope(k, pos, cfg["rope_theta"], cfg["neox"])
        k, v = keep(k), keep(v)
        q = q.reshape(rows, kvh, nh // kvh, hd)
        if kind == "decode":
            ck, cv = (keep(t) for t in _cache(cfg, case, i, seed))
            att = []
            for b in range(rows):  # one sequence at a time: the cache in 64 bits is large
                kk, vv = torch.cat([ck[b].double(), k[b][:, None]], 1), torch.cat([cv[b].double(), v[b][:, None]], 1)
                att.append(torch.softmax(q[b] @ kk.transpose(1, 2) * hd ** -0.5, -1) @ vv)
            att = torch.stack(att)
        else:
            kk, vv = k.transpose(0, 1), v.transpose(0, 1)
            if ctx:
                ck, cv = (keep(t)[0].double() for t in _cache(cfg, case, i, seed))
                kk, vv = torch.cat([ck, kk], 1), torch.cat([cv, vv], 1)
            hidden = torch.arange(ctx + rows, device="cuda")[None] > pos[:, None]
            att = torch.empty_like(q)
            for g in range(kvh):
                s = (q[:, g].transpose(0, 1) @ kk[g].T * hd ** -0.5).masked_fill(hidden, -math.inf)
                att[:, g] = (torch.softmax(s, -1) @ vv[g]).transpose(0, 1)
        x = x + act(att.reshape(rows, -1)) @ w["wo"].T
        g = act(_unit(x, eps) * w["norm2"]) @ w["wgu"].T
        x = x + act(torch.nn.functional.silu(g[:, :F]) * g[:, F:]) @ w["wdown"].T
    x = act(_unit(x, eps) * _vector(cfg["hidden"], seed, 501))
    return x[-1] @ table.T if kind == "prompt" else x @ table.T


def _decayed(q, k, v, decay):
    """q, k, v [T, heads, .]: o_t = sum over s <= t of decay^(t - s) (q_t . k_s) v_s."""
    t = torch.arange(q.shape[0], device="cuda")
    out = []
    for h, a in enumerate(decay):
        gap = (t[:, None] - t[None]).double()
        m = torch.where(gap >= 0, torch.tensor(a, dtype=torch.float64, device="cuda") ** gap.clamp(min=0), torch.zeros_like(gap))
        out.append((q[:, h] @ k[:, h].T * m) @ v[:, h])
    return torch.stack(out, 1)


def _exact_layered(case, seed):
    cfg = _layered_config(case)
    names, T = _LayeredTensors(cfg, seed), case["rows"] + case["steps"]
    cache = {}

    def w(name):
        if name not in cache:
            cache[name] = names[name].double()
        return cache[name]

    silu, eps = torch.nn.functional.silu, cfg["eps"]

    def norm(x, name):
        d = x - x.mean(-1, keepdim=True)
        return d / (d.square().mean(-1, keepdim=True) + eps).sqrt() * w(name)

    def light(h, p, m):
        q, k = (silu(h @ w(p + n).T).reshape(-1, m["heads"], m["dim"]) for n in "qk")
        v = silu(h @ w(p + "v").T).reshape(-1, m["heads"], m["vdim"])
        o = _decayed(q, k, v, m["decay"]).reshape(h.shape[0], -1)
        return (_unit(o, eps) * w(p + "norm") * torch.sigmoid(h @ w(p + "g").T)) @ w(p + "o").T

    def window(h, p, m):
        n, H, G, t = h.shape[0], m["heads"], m["kv_heads"], torch.arange(h.shape[0], device="cuda")
        q, k, v = ((h @ w(p + s).T + w(p + s + ".b")).reshape(n, -1, 128) for s in "qkv")
        q, k = _unit(q, eps) * w(p + "q.norm"), _unit(k, eps) * w(p + "k.norm")
        rel = w(p + "rel")
        half, rows = rel.shape[0] // 2, rel.shape[0]
        bucket = [d if d < half else min(rows - 1, half + math.floor(math.log(d / half) / math.log(m["bias_max"] / half) * (rows - half)))
                  for d in range(n)]
        gap = t[:, None] - t[None]
        which = torch.tensor(bucket, device="cuda")[gap.clamp(min=0)]
        out = []
        for i in range(H):
            s = q[:, i] @ k[:, i // (H // G)].T * m["scale"] + rel[:, i][which]
            s = s.masked_fill((gap < 0) | (gap >= m["mask"]["size"]), -math.inf)
            out.append(torch.softmax(s, -1) @ v[:, i // (H // G)])
        return torch.cat(out, 1) @ w(p + "o").T

    def retention(h, p, m):
        n, D, t = h.shape[0], m["dim"], torch.arange(h.shape[0], device="cuda").double()
        f = m["rot"]["base"] ** (-2.0 * torch.arange(D // 2, device="cuda").double() / D)
        c, s = (t[:, None] * f).cos()[:, None], (t[:, None] * f).sin()[:, None]

        def turn(x):
            u, v = x.reshape(n, -1, D).chunk(2, -1)
            return torch.cat([u * c - v * s, v * c + u * s], -1)

        q, k = turn(h @ w(p + "q").T), turn(h @ w(p + "k").T) * D ** -0.5
        o = _unit(_decayed(q, k, (h @ w(p + "v").T).reshape(n, -1, m["vdim"]), m["decay"]), eps).reshape(n, -1)
        return (o * silu(h @ w(p + "g").T)) @ w(p + "o").T

    tokens = _tokens(cfg["vocab"], case["batch"] * T, seed, 999).reshape(-1, case["batch"]).long()
    every = []
    for b in range(case["batch"]):
        x = w("embed")[tokens[:, b]]
        for i, layer in enumerate(cfg["layers"]):
            p, m = f"l{i}.", layer["mixer"]
            h = norm(x, p + "norm1")
            if layer["type"] == "lightning":
                x = x + light(h, p + "mix.", m)
            else:
                x = x + m["left_scale"] * window(h, p + "mix.left.", m["left"]) + m["right_scale"] * retention(h, p + "mix.right.", m["right"])
            h = norm(x, p + "norm2")
            x = x + (torch.nn.functional.gelu(h @ w(p + "mlp.gate").T, approximate="tanh") * (h @ w(p + "mlp.up").T)) @ w(p + "mlp.down").T
        every.append(30.0 * torch.tanh(norm(x[case["rows"] - 1:], "final.norm") @ w("embed").T / 30.0))
    every = torch.stack(every, 1)
    return [every[:1, b] for b in range(case["batch"])] + [every[1 + s] for s in range(case["steps"])]


def exact(case, seed):
    if case["kind"] == "matmul":
        x = _randn((case["rows"], case["k"]), seed, 1)
        x = _q8_rows(x) if case["mode"] == "q8" else x.double()
        return x @ _matrix(case["fmt"], case["n"], case["k"], True, seed, 0).T
    return _exact_layered(case, seed) if case["kind"] == "layered" else _exact_decoder(case, seed)
