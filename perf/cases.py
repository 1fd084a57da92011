"""The work that this framework is used for, as cases that can be timed and compared: the Llama decode path (linears, paged
attention, a whole step) and the blocks of the models described layer by layer (routed experts, latent and windowed attention,
recurrences), through the C ABI and the runner.

Sizes are those of Llama-3.1-8B and of the 2048-wide layer-list configurations of bench.py.  listed() names the cases, draw() gives
others of the same ranges, prepare() makes inputs and workspaces, run() is one pass, exact() the same result in 64 bits."""
import importlib
import math
import random

import torch

_abi = importlib.import_module("enterprise-inference_b200._abi")
BF16, F32, F64 = torch.bfloat16, torch.float32, torch.float64
BLOCK = 128   # tokens of a cache block
_streams = {}


def listed():
    return [
        # one sequence of an 8B model: the fused q|k|v projection of one token row (the smallest call)
        {"name": "linear_qkv_1", "kind": "linear", "rows": 1, "n_out": 6144, "k": 4096},
        # the down projection of an ordinary prefill chunk, not a multiple of any tile (the largest call)
        {"name": "linear_down_2000", "kind": "linear", "rows": 2000, "n_out": 4096, "k": 14336},
        # decode attention of 64 running sequences of different lengths
        {"name": "attn_decode_64", "kind": "attn_decode", "rows": 64, "ctx": 1000, "heads": 32, "kv": 8},
        # a 2048-row prefill chunk of one sequence behind 1000 cached tokens
        {"name": "attn_prefill_2048", "kind": "attn_prefill", "rows": 2048, "ctx": 1000, "heads": 32, "kv": 8},
        # a whole decode step of 64 sequences through the runner: four layers of 8B's width, its vocabulary, logits out
        {"name": "llama_step_64", "kind": "step", "rows": 64, "ctx": 600, "layers": 4},
        # routed experts, decode step: 64 rows over 32 gated experts, 4 chosen
        {"name": "moe_64", "kind": "moe", "rows": 64, "width": 2048, "ff": 1024, "experts": 32, "top": 4, "gated": True},
        # the same experts under a prefill chunk
        {"name": "moe_2048", "kind": "moe", "rows": 2048, "width": 2048, "ff": 1024, "experts": 32, "top": 4, "gated": True},
        # latent attention (16 heads over rows of 512 + 64) of a prefill chunk
        {"name": "latent_2048", "kind": "latent", "rows": 2048, "seqs": 1, "ctx": 0, "heads": 16, "rank": 512, "rot": 64},
        # latent attention of 64 decoding sequences
        {"name": "latent_64", "kind": "latent", "rows": 64, "seqs": 64, "ctx": 1000, "heads": 16, "rank": 512, "rot": 64},
        # windowed attention with capped, distance-biased scores and a gate per head: a chunk of three sequences
        {"name": "window_1900", "kind": "window", "rows": 1900, "seqs": 3, "ctx": 700, "heads": 16, "kv": 4, "dim": 128, "window": 1024},
        # matrix-memory recurrence of a prefill chunk
        {"name": "mlstm_2048", "kind": "mlstm", "rows": 2048, "seqs": 1, "heads": 8, "dim": 128, "vdim": 256},
        # delta-rule recurrence with channel decays: a chunk of three sequences
        {"name": "delta_1900", "kind": "delta", "rows": 1900, "seqs": 3, "heads": 16, "kv": 16, "dim": 128, "vdim": 128, "rule": "channel"},
    ]


def _log(rng, lo, hi):
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    kind = rng.choice(["linear", "attn_decode", "attn_prefill", "step", "moe", "latent", "window", "mlstm", "delta"])
    if kind == "linear":
        n_out, k = rng.choice([(6144, 4096), (4096, 4096), (28672, 4096), (4096, 14336), (7168, 5120), (5120, 5120), (2048, 2048), (8192, 2048)])
        rows = _log(rng, 1, 2048)
        return {"kind": kind, "rows": max(1, min(rows, int(2000 * 4096 * 14336 / (n_out * k)))), "n_out": n_out, "k": k}
    if kind == "attn_decode":
        rows = _log(rng, 1, 128)
        return {"kind": kind, "rows": rows, "ctx": _log(rng, 100, min(16384, 200000 // rows)), "heads": 32, "kv": 8}
    if kind == "attn_prefill":
        return {"kind": kind, "rows": _log(rng, 40, 2048), "ctx": rng.choice([0, rng.randint(1, 2048)]), "heads": 32, "kv": 8}
    if kind == "step":
        return {"kind": kind, "rows": _log(rng, 1, 64), "ctx": _log(rng, 100, 600), "layers": rng.randint(2, 4)}
    if kind == "moe":
        width, ff, experts, top = rng.choice([(2048, 1024, 32, 4), (4096, 512, 64, 8), (1024, 1024, 16, 2)])
        return {"kind": kind, "rows": _log(rng, 1, 2048), "width": width, "ff": ff, "experts": experts, "top": top, "gated": rng.random() < 0.5}
    if kind == "latent":
        rank, rot = rng.choice([(512, 64), (256, 32), (512, 0)])
        rows, decode = _log(rng, 1, 2048), rng.random() < 0.4
        if decode:
            rows = min(rows, 128)
        return {"kind": kind, "rows": rows, "seqs": rows if decode else rng.randint(1, min(rows, 4)), "ctx": rng.choice([0, rng.randint(1, 3000)]),
                "heads": 16, "rank": rank, "rot": rot}
    if kind == "window":
        rows, decode = _log(rng, 1, 2048), rng.random() < 0.3
        if decode:
            rows = min(rows, 128)
        return {"kind": kind, "rows": rows, "seqs": rows if decode else rng.randint(1, min(rows, 4)), "ctx": rng.choice([0, rng.randint(1, 2000)]),
                "heads": 16, "kv": 4, "dim": rng.choice([64, 128]), "window": rng.choice([0, 512, 1024, 4096])}
    if kind == "mlstm":
        heads, dim, vdim = rng.choice([(8, 128, 256), (4, 128, 256), (8, 64, 128)])
        rows = _log(rng, 1, 2048)
        return {"kind": kind, "rows": rows, "seqs": rng.randint(1, min(rows, 4)), "heads": heads, "dim": dim, "vdim": vdim}
    rule = rng.choice(["channel", "head", "plain"])
    heads, kv, dim, vdim = (64, 2, 128, 64) if rule == "plain" else rng.choice([(16, 16, 128, 128), (8, 8, 128, 128), (16, 4, 64, 128)])
    rows = _log(rng, 1, 2048)
    return {"kind": "delta", "rows": rows, "seqs": rng.randint(1, min(rows, 4)), "heads": heads, "kv": kv, "dim": dim, "vdim": vdim, "rule": rule}


# ---- shapes of a step: rows dealt to sequences, context lengths ------------------------------------------------------------

def _portions(case):
    """Rows of each sequence of the step: whole sequences of uneven length."""
    rows, seqs = case["rows"], case.get("seqs", 1)
    r = random.Random(repr(sorted((k, v) for k, v in case.items() if k != "name")))
    cuts = sorted(r.sample(range(1, rows), seqs - 1)) if seqs < rows else list(range(1, rows))
    return [b - a for a, b in zip([0] + cuts, cuts + [rows])], r


def _contexts(case):
    """(rows per sequence, tokens cached before the step per sequence): half to all of `ctx` where several sequences run."""
    if case["kind"] in ("attn_decode", "step"):
        case = dict(case, seqs=case["rows"])
    parts, r = _portions(case)
    before = [case["ctx"] if len(parts) == 1 else r.randint(case["ctx"] // 2, case["ctx"]) for _ in parts]
    return parts, before


class _Paged:
    """Block tables in random order and the per-row arrays of one step."""

    def __init__(self, case, g):
        parts, before = _contexts(case)
        need = [(b + n + BLOCK - 1) // BLOCK for n, b in zip(parts, before)]
        self.n_blocks, self.stride = sum(need) + 1, max(need)
        order = (torch.randperm(self.n_blocks - 1, generator=g, device="cuda") + 1).to(torch.int32)
        self.bt = torch.zeros(len(parts), self.stride, dtype=torch.int32, device="cuda")
        at = 0
        for s, n in enumerate(need):
            self.bt[s, :n] = order[at:at + n]
            at += n
        pos = [b + i for n, b in zip(parts, before) for i in range(n)]
        seq = [s for s, n in enumerate(parts) for _ in range(n)]
        self.rows, self.parts, self.before, self.max_ctx = len(pos), parts, before, max(pos) + 1
        self.positions = torch.tensor(pos, dtype=torch.int32, device="cuda")
        self.ctx = self.positions + 1
        self.seq = torch.tensor(seq, dtype=torch.int32, device="cuda")
        own = self.bt[self.seq.long(), (self.positions // BLOCK).long()]
        self.slots = (own * BLOCK + self.positions % BLOCK).to(torch.int32)


def _pairs(case):
    """(row, key) pairs that the attention of one head sees, and the keys that have to be read."""
    parts, before = _contexts(case)
    w = case.get("window", 0)
    seen = sum(min(b + i + 1, w) if w else b + i + 1 for n, b in zip(parts, before) for i in range(n))
    keys = sum(min(b + n, n + w - 1) if w else b + n for n, b in zip(parts, before))
    return seen, keys


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _randn(g, *shape, dtype=BF16, std=1.0):
    return torch.empty(shape, dtype=dtype, device="cuda").normal_(0.0, std, generator=g)


def _splits(rows, heads, max_ctx):
    """Context splits as the framework's own steps choose them."""
    ctas = (rows * heads + 15) // 16
    if ctas >= 148 or max_ctx <= (4 if ctas < 16 else 16) * 64:
        return 1
    return max(1, min(((max_ctx + 63) // 64 + 1) // 2, (296 + ctas - 1) // ctas, 16))


# ---- inputs ----------------------------------------------------------------------------------------------------------------

def prepare(case, seed):
    g, kind, lib = _gen(seed), case["kind"], _abi.lib()
    s = {"case": case, "lib": lib}
    T = case["rows"]
    if kind == "linear":
        n, k = case["n_out"], case["k"]
        wsb = int(lib.b200_linear_workspace_bytes(T, n, k))
        s.update(x=_randn(g, T, k), w=_randn(g, n, k, std=0.02), y=torch.empty(T, n, dtype=BF16, device="cuda"),
                 ws=torch.zeros(max(wsb, 16), dtype=torch.uint8, device="cuda"), wsb=wsb)
    elif kind in ("attn_decode", "attn_prefill"):
        p, H, kv = _Paged(case, g), case["heads"], case["kv"]
        wsb = int(lib.b200_paged_attn_workspace_bytes(T, H, p.max_ctx, BLOCK))
        s.update(p=p, q=_randn(g, T, H * 128), kc=_randn(g, p.n_blocks, kv, BLOCK, 128), vc=_randn(g, p.n_blocks, kv, BLOCK, 128),
                 y=torch.empty(T, H * 128, dtype=BF16, device="cuda"), ws=torch.zeros(max(wsb, 16), dtype=torch.uint8, device="cuda"), wsb=wsb)
    elif kind == "step":
        R = importlib.import_module("enterprise-inference_b200.runner")
        C = importlib.import_module("enterprise-inference_b200.config")
        p = _Paged(case, g)
        cfg = C.ModelConfig(name="8b-width", hidden=4096, n_layers=case["layers"], n_q_heads=32, n_kv_heads=8, intermediate=14336, vocab=128256,
                            max_pos=8192)
        r = R.ModelRunner(cfg, max_tokens=max(T, 16), max_model_len=1024, n_blocks=p.n_blocks)
        r.init_random_weights(seed=seed)
        r.k_cache.normal_(0.0, 1.0, generator=g)
        r.v_cache.normal_(0.0, 1.0, generator=g)
        if "step" not in _streams:
            _streams["step"] = torch.cuda.Stream()   # one stream for all runners (a step cannot be captured on the default one)
        s.update(p=p, r=r, stream=_streams["step"], ids=torch.randint(0, cfg.vocab, (T,), generator=g, device="cuda", dtype=torch.int32),
                 tokens=torch.empty(T, dtype=torch.int32, device="cuda"), logits=torch.empty(T, cfg.vocab, dtype=BF16, device="cuda"))
    elif kind == "moe":
        W, ff, E, top = case["width"], case["ff"], case["experts"], case["top"]
        wsb = int(lib.b200_moe_workspace_bytes(T, top, E, W, ff))
        s.update(x=_randn(g, T, W), wr=_randn(g, E, W, std=0.02), wu=_randn(g, E, (2 if case["gated"] else 1) * ff, W, std=0.02),
                 wd=_randn(g, E, W, ff, std=0.02), ids=torch.empty(T, top, dtype=torch.int32, device="cuda"),
                 wts=torch.empty(T, top, dtype=F32, device="cuda"), logits=torch.empty(T, E, dtype=F32, device="cuda"),
                 parts=torch.empty(T, top, W, dtype=F32, device="cuda"), ws=torch.zeros(wsb, dtype=torch.uint8, device="cuda"))
    elif kind in ("latent", "window"):
        p, H = _Paged(case, g), case["heads"]
        if kind == "latent":
            krow, vd = case["rank"] + case["rot"], case["rank"]
            s.update(kc=_randn(g, p.n_blocks, 1, BLOCK, krow), sink=_randn(g, H, dtype=F32))
            scale, seen = 1.0 / math.sqrt(192.0), p.max_ctx
            q = _randn(g, T, H, krow, dtype=F32, std=0.6)
        else:
            krow = vd = case["dim"]
            s.update(kc=_randn(g, p.n_blocks, case["kv"], BLOCK, krow), vc=_randn(g, p.n_blocks, case["kv"], BLOCK, vd),
                     bias=_randn(g, H, 256, dtype=F32, std=0.5), gate=_randn(g, T, H))
            scale, seen = 1.0 / math.sqrt(krow), min(p.max_ctx, case["window"] + T) if case["window"] else p.max_ctx
            q = _randn(g, T, H, krow, dtype=F32)
        ns = _splits(T, H, seen)
        s.update(p=p, q=q, scale=scale, ns=ns, y=torch.empty(T, H, vd, dtype=BF16, device="cuda"),
                 part=torch.empty(T * H * ns * (vd + 2), dtype=F32, device="cuda"),
                 ws=torch.zeros(int(lib.b200_paged_attn_anydim_workspace_bytes(T)), dtype=torch.uint8, device="cuda"))
    else:
        parts, _ = _portions(case)
        H, d, vd, S = case["heads"], case["dim"], case["vdim"], len(parts)
        start = [0]
        for n in parts:
            start.append(start[-1] + n)
        slots = torch.randperm(S + 2, generator=g, device="cuda")[:S].to(torch.int32)
        floats = int(lib.b200_mlstm_state_floats(H, d, vd)) if kind == "mlstm" else H * d * vd
        s.update(positions=torch.tensor([i for n in parts for i in range(n)], dtype=torch.int32, device="cuda"),
                 start=torch.tensor(start, dtype=torch.int32, device="cuda"), slots=slots, S=S, parts=parts,
                 state=torch.zeros(S + 2, floats, dtype=F32, device="cuda"), floats=floats, y=torch.empty(T, H * vd, dtype=F32, device="cuda"))
        if kind == "mlstm":
            gates = _randn(g, T, 2 * H, dtype=F32, std=1.5)
            gates[:, H:] = torch.nn.functional.logsigmoid(gates[:, H:] + 3.0)
            s.update(qkv=_randn(g, T, 2 * H * d + 2 * H * vd), gates=gates)
        else:
            kv = case["kv"]
            unit = lambda x: x / x.norm(dim=-1, keepdim=True)   # noqa: E731
            s.update(q=(unit(_randn(g, T, kv, d, dtype=F32)) * d ** -0.5).reshape(T, kv * d), k=unit(_randn(g, T, kv, d, dtype=F32)).reshape(T, kv * d),
                     v=torch.nn.functional.silu(_randn(g, T, H * vd, dtype=F32)), beta=torch.sigmoid(_randn(g, T, H, dtype=F32)))
            wide = d if case["rule"] == "channel" else 1
            a = torch.empty(H, dtype=F32, device="cuda").uniform_(1.0, 16.0, generator=g)
            dt = torch.exp(torch.empty(T, H, wide, dtype=F32, device="cuda").uniform_(math.log(1e-3), math.log(1e-1), generator=g))
            s["decay"] = torch.exp(-a[None, :, None] * dt).reshape(T, H * wide).contiguous()
    return s


# ---- one pass --------------------------------------------------------------------------------------------------------------

def run(s):
    c, lib, kind = s["case"], s["lib"], s["case"]["kind"]
    T, st = c["rows"], torch.cuda.current_stream().cuda_stream
    P = _abi.ptr
    if kind == "linear":
        _abi.check(lib.b200_linear_bf16(P(s["x"]), c["k"], P(s["w"]), None, P(s["y"]), c["n_out"], T, c["n_out"], c["k"], 0, P(s["ws"]), s["wsb"], st))
        return s["y"]
    if kind in ("attn_decode", "attn_prefill"):
        p, H = s["p"], c["heads"]
        f = lib.b200_paged_attn_decode if kind == "attn_decode" else lib.b200_paged_attn_prefill
        _abi.check(f(P(s["q"]), H * 128, P(s["kc"]), P(s["vc"]), P(p.bt), p.stride, P(p.seq), P(p.ctx), P(s["y"]), H * 128, T, H, c["kv"], BLOCK,
                     p.max_ctx, 128 ** -0.5, P(s["ws"]), s["wsb"], st))
        return s["y"]
    if kind == "step":
        p = s["p"]
        s["r"].step_device(s["ids"], p.positions, p.slots, p.bt, p.ctx, p.max_ctx, out_tokens=s["tokens"], out_logits=s["logits"], stream=s["stream"])
        return s["logits"]
    if kind == "moe":
        W, ff, E, top = c["width"], c["ff"], c["experts"], c["top"]
        _abi.check(lib.b200_moe_route_linear(P(s["x"]), P(s["wr"]), None, T, W, E, top, 1, 1, P(s["ids"]), P(s["wts"]), P(s["logits"]), st))
        if c["gated"]:
            _abi.check(lib.b200_moe_experts(0, P(s["x"]), P(s["wu"]), P(s["wd"]), P(s["ids"]), P(s["wts"]), T, W, ff, E, top, P(s["parts"]), P(s["ws"]), st))
        else:
            _abi.check(lib.b200_moe_experts_form(0, P(s["x"]), P(s["wu"]), P(s["wd"]), P(s["ids"]), P(s["wts"]), T, W, ff, E, top, P(s["parts"]),
                                                 P(s["ws"]), 0, _abi.ACT_RELU2, 0, st))
        return {"logits": s["logits"], "parts": s["parts"]}
    if kind == "latent":
        p, krow = s["p"], c["rank"] + c["rot"]
        _abi.check(lib.b200_latent_attn(P(s["q"]), P(s["kc"]), P(p.bt), p.stride, P(p.seq), P(p.ctx), P(s["y"]), T, c["heads"], krow, c["rank"], BLOCK,
                                        s["scale"], P(s["sink"]), P(s["ws"]), s["ns"], P(s["part"]), st))
        return s["y"]
    if kind == "window":
        p = s["p"]
        _abi.check(lib.b200_paged_attn_biased(0, 2, P(s["q"]), P(s["kc"]), P(s["vc"]), P(p.bt), p.stride, P(p.seq), P(p.ctx), P(p.positions), P(s["y"]),
                                              T, c["heads"], c["kv"], c["dim"], c["dim"], BLOCK, s["scale"], c["window"], 30.0, P(s["bias"]), 256,
                                              P(s["gate"]), c["heads"], P(s["ws"]), s["ns"], P(s["part"]), st))
        return s["y"]
    H, d, vd = c["heads"], c["dim"], c["vdim"]
    if kind == "mlstm":
        _abi.check(lib.b200_mlstm_scan(0, P(s["qkv"]), s["qkv"].shape[1], 0, H * d, 2 * H * d, P(s["gates"]), P(s["positions"]), P(s["start"]),
                                       P(s["slots"]), P(s["state"]), s["floats"], P(s["y"]), s["S"], H, d, vd, st))
    elif c["rule"] == "channel":
        _abi.check(lib.b200_delta_scan(P(s["q"]), P(s["k"]), P(s["v"]), P(s["beta"]), P(s["decay"]), P(s["positions"]), P(s["start"]), P(s["slots"]),
                                       P(s["state"]), s["floats"], P(s["y"]), s["S"], H, c["kv"], d, vd, st))
    else:
        _abi.check(lib.b200_linear_scan(int(c["rule"] == "head"), P(s["q"]), P(s["k"]), P(s["v"]), P(s["beta"]), P(s["decay"]), H, 1, 0,
                                        P(s["positions"]), P(s["start"]), P(s["slots"]), P(s["state"]), s["floats"], P(s["y"]), s["S"], H, c["kv"], d,
                                        vd, st))
    return {"y": s["y"], "state": s["state"]}


# ---- what a pass cannot do without -----------------------------------------------------------------------------------------

def work(case):
    kind, T = case["kind"], case["rows"]
    if kind == "linear":
        n, k = case["n_out"], case["k"]
        return {"bytes": 2 * (n * k + T * k + T * n), "flops": 2 * T * n * k}
    if kind in ("attn_decode", "attn_prefill"):
        seen, keys = _pairs(case)
        return {"bytes": 4 * T * case["heads"] * 128 + keys * case["kv"] * 512, "flops": 4 * seen * case["heads"] * 128}
    if kind == "step":
        seen, keys = _pairs(case)
        L, h, I, V = case["layers"], 4096, 14336, 128256
        weights = L * (6144 * h + h * h + 3 * I * h) + V * h
        return {"bytes": 2 * weights + L * keys * 8 * 512 + 2 * T * (V + h), "flops": 2 * T * weights + L * 4 * seen * 32 * 128}
    if kind == "moe":
        W, ff, E, top, m = case["width"], case["ff"], case["experts"], case["top"], 3 if case["gated"] else 2
        used = E * (1.0 - (1.0 - top / E) ** T)
        return {"bytes": 2 * used * m * ff * W + 2 * E * W + 2 * T * W + 4 * T * (E + top * W), "flops": 2 * T * (top * m * ff * W + E * W)}
    if kind == "latent":
        seen, keys = _pairs(case)
        H, r, kr = case["heads"], case["rank"], case["rank"] + case["rot"]
        return {"bytes": 4 * T * H * kr + 2 * keys * kr + 2 * T * H * r, "flops": 2 * seen * H * (kr + r)}
    if kind == "window":
        seen, keys = _pairs(case)
        H, d = case["heads"], case["dim"]
        return {"bytes": T * H * (6 * d + 2) + keys * case["kv"] * 4 * d + 1024 * H, "flops": 4 * seen * H * d}
    H, d, vd, S = case["heads"], case["dim"], case["vdim"], case["seqs"]
    if kind == "mlstm":
        return {"bytes": 2 * T * H * (2 * d + vd) + 8 * T * H + 4 * T * H * vd + 4 * S * H * vd * d, "flops": 6 * T * H * d * vd}
    wide = d if case["rule"] == "channel" else 1
    return {"bytes": 4 * T * (2 * case["kv"] * d + 2 * H * vd + H + H * wide) + 4 * S * H * vd * d,
            "flops": (8 if case["rule"] != "plain" else 6) * T * H * d * vd}


def tolerance(case):
    """About four times what the framework's results differ from those in 64 bits (a step's: one layer's rounding travels through the others)."""
    return {"linear": {"rel": 7e-3, "max": 1.6e-2}, "attn_decode": {"rel": 7e-3, "max": 1.6e-2}, "attn_prefill": {"rel": 7e-3, "max": 1.6e-2},
            "step": {"rel": 3e-2, "max": 0.4}, "moe": {"rel": 1.4e-2, "max": 0.28}, "latent": {"rel": 1.1e-2, "max": 0.18},
            "window": {"rel": 1.1e-2, "max": 0.1}, "mlstm": {"rel": 5e-6, "max": 1e-4}, "delta": {"rel": 2e-6, "max": 2e-5}}[case["kind"]]


# ---- the same results in 64 bits -------------------------------------------------------------------------------------------

def _rows_of(cache, p, s, n):
    """The first n cached rows of sequence s, 64 bits: [kv][n][dim]."""
    b = cache[p.bt[s, :(n + BLOCK - 1) // BLOCK].long()]          # [blocks][kv][BLOCK][dim]
    return b.transpose(0, 1).reshape(b.shape[1], -1, b.shape[3])[:, :n].to(F64)


def _attend(q, kc, vc, p, kv, vdim, scale, window=0, shape=None, sink=None):
    """Causal paged attention of q [T][heads][dim]; shape(scores, distance) is applied to the scaled scores [kv][G][rows][keys]."""
    T, H, d = q.shape
    G, out, at = H // kv, torch.empty(q.shape[0], H, vdim, dtype=F64, device="cuda"), 0
    for s, (n, b) in enumerate(zip(p.parts, p.before)):
        K, V = _rows_of(kc, p, s, b + n), _rows_of(vc, p, s, b + n)[..., :vdim]
        for lo in range(0, n, 256):
            hi = min(n, lo + 256)
            Q = q[at + lo:at + hi].to(F64).reshape(hi - lo, kv, G, d).permute(1, 2, 0, 3)
            x = torch.matmul(Q, K[:, None].transpose(-1, -2)) * scale
            dist = torch.arange(b + lo, b + hi, device="cuda")[:, None] - torch.arange(b + n, device="cuda")[None, :]
            if shape:
                x = shape(x, dist.clamp(min=0))
            x = x.masked_fill((dist < 0) | ((dist >= window) if window else (dist < 0)), -math.inf)
            if sink is not None:
                x = torch.cat([x, sink.to(F64).reshape(kv, G, 1, 1).expand(kv, G, hi - lo, 1)], -1)
            w = torch.softmax(x, -1)[..., :b + n]
            out[at + lo:at + hi] = torch.matmul(w, V[:, None]).permute(2, 0, 1, 3).reshape(hi - lo, H, vdim)
        at += n
    return out


def _exact_step(s, case):
    p, r, T, H, kv = s["p"], s["r"], case["rows"], 32, 8
    w = [t.to(F64) if t.dim() == 1 else t for t in r._weights]   # embedding, then six per layer, then final norm and head
    mm = lambda x, m: torch.cat([x @ c.to(F64).T for c in m.split(8192)], 1)   # noqa: E731
    rms = lambda x, g: x / torch.sqrt((x * x).mean(-1, keepdim=True) + r.cfg.rms_eps) * g   # noqa: E731
    cs = r.cos_sin[p.positions.long()].to(F64)
    cos, sin = cs[:, None, :64], cs[:, None, 64:]
    rope = lambda x: torch.cat([x[..., :64] * cos - x[..., 64:] * sin, x[..., 64:] * cos + x[..., :64] * sin], -1)   # noqa: E731
    x = w[0][s["ids"].long()].to(F64)
    for l in range(case["layers"]):
        ln1, qkv, o, ln2, gu, down = w[1 + 6 * l:7 + 6 * l]
        z = mm(rms(x, ln1), qkv).reshape(T, H + 2 * kv, 128)
        q, k, v = rope(z[:, :H]), rope(z[:, H:H + kv]), z[:, H + kv:]
        K, V = r.k_cache[l].to(F64), r.v_cache[l].to(F64)
        blk, off = (p.slots // BLOCK).long(), (p.slots % BLOCK).long()
        K[blk, :, off], V[blk, :, off] = k, v
        x = x + mm(_attend(q, K, V, p, kv, 128, 128 ** -0.5).reshape(T, H * 128), o)
        z = mm(rms(x, ln2), gu).reshape(T, -1, 2, 64)   # slabs of 64 gate and 64 up rows
        x = x + mm((torch.nn.functional.silu(z[:, :, 0]) * z[:, :, 1]).reshape(T, -1), down)
    return mm(rms(x, w[-2]), w[-1])


def exact(case, seed):
    s, kind, T = prepare(case, seed), case["kind"], case["rows"]
    if kind == "linear":
        return torch.cat([s["x"].to(F64) @ c.to(F64).T for c in s["w"].split(4096)], 1)
    if kind in ("attn_decode", "attn_prefill"):
        H = case["heads"]
        return _attend(s["q"].reshape(T, H, 128), s["kc"], s["vc"], s["p"], case["kv"], 128, 128 ** -0.5).reshape(T, H * 128)
    if kind == "step":
        return _exact_step(s, case)
    if kind == "moe":
        x = s["x"].to(F64)
        logits = x @ s["wr"].to(F64).T
        wts, ids = torch.topk(torch.softmax(logits, -1), case["top"], -1)
        parts = torch.zeros(T, case["top"], case["width"], dtype=F64, device="cuda")
        for e in range(case["experts"]):
            t, j = (ids == e).nonzero(as_tuple=True)
            u = x[t] @ s["wu"][e].to(F64).T
            if case["gated"]:
                u = torch.nn.functional.silu(u[:, :case["ff"]]) * u[:, case["ff"]:]
            else:
                u = torch.relu(u) ** 2
            parts[t, j] = (u @ s["wd"][e].to(F64).T) * wts[t, j, None]
        return {"logits": logits, "parts": parts}
    if kind == "latent":
        return _attend(s["q"], s["kc"], s["kc"], s["p"], 1, case["rank"], s["scale"], sink=s["sink"])
    if kind == "window":
        H, kv = case["heads"], case["kv"]
        bias = s["bias"].to(F64).reshape(kv, H // kv, 256)
        shape = lambda x, dist: 30.0 * torch.tanh(x / 30.0) + bias[:, :, dist.clamp(max=255)]   # noqa: E731
        y = _attend(s["q"], s["kc"], s["vc"], s["p"], kv, case["dim"], s["scale"], case["window"], shape)
        return y * torch.sigmoid(s["gate"].to(F64))[..., None]
    H, d, vd = case["heads"], case["dim"], case["vdim"]
    y, at = torch.empty(T, H, vd, dtype=F64, device="cuda"), 0
    state = torch.zeros(s["state"].shape, dtype=F64, device="cuda")
    for i, n in enumerate(s["parts"]):
        S = torch.zeros(H, vd, d, dtype=F64, device="cuda")
        if kind == "mlstm":
            x = s["qkv"][at:at + n].to(F64)
            q, k = x[:, :H * d].reshape(n, H, d) * d ** -0.5, x[:, H * d:2 * H * d].reshape(n, H, d)
            v, gt = x[:, 2 * H * d:2 * H * d + H * vd].reshape(n, H, vd), s["gates"][at:at + n].to(F64)
            nn, m = torch.zeros(H, d, dtype=F64, device="cuda"), torch.zeros(H, dtype=F64, device="cuda")
            for t in range(n):
                ig, fg = gt[t, :H], gt[t, H:]
                mn = torch.maximum(fg + m, ig)
                a, b, m = torch.exp(fg + m - mn), torch.exp(ig - mn), mn
                bk = b[:, None] * k[t]
                S = a[:, None, None] * S + v[t][:, :, None] * bk[:, None, :]
                nn = a[:, None] * nn + bk
                den = torch.maximum((nn * q[t]).sum(-1).abs(), torch.exp(-m)) + 1e-6
                y[at + t] = torch.matmul(S, q[t][:, :, None])[..., 0] / den[:, None]
            nz = (vd + 31) // 32
            state[s["slots"][i].long()] = torch.cat([S.reshape(-1), nn[:, None].expand(H, nz, d).reshape(-1), m[:, None].expand(H, nz).reshape(-1)])
        else:
            kv, rule = case["kv"], case["rule"]
            wide = lambda z, w: z[at:at + n].to(F64).reshape(n, -1, w)   # noqa: E731
            q, k = (wide(s[z], d).repeat_interleave(H // kv, 1) for z in "qk")
            v, beta, g = wide(s["v"], vd), s["beta"][at:at + n].to(F64), wide(s["decay"], d if rule == "channel" else 1)
            for t in range(n):
                S = S * g[t][:, None, :]
                u = v[t] if rule == "plain" else v[t] - torch.matmul(S, k[t][:, :, None])[..., 0]
                S = S + (beta[t][:, None] * u)[:, :, None] * k[t][:, None, :]
                y[at + t] = torch.matmul(S, q[t][:, :, None])[..., 0]
            state[s["slots"][i].long()] = S.reshape(-1)
        at += n
    return {"y": y.reshape(T, H * vd), "state": state}
