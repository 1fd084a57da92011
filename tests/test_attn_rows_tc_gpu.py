"""Attention of runs of rows on tcgen05 (heads of at most 128, cache blocks of whole 64-key tiles) against the same attention in float64."""
import pytest
import torch

from conftest import pkg

pytestmark = pytest.mark.gpu
DEV = "cuda"
CTXS = [1, 2, 63, 64, 65, 127, 128, 129, 500] + list(range(1, 71)) + list(range(300, 431)) + list(range(490, 500))
SEQ = list(range(9)) + [9] * 70 + [10] * 131 + [11] * 10      # decode rows at tile and block edges, then runs of odd lengths that start inside tiles


def _case(heads, kv, dim, vdim, bs, seed):
    g = torch.Generator().manual_seed(seed)
    n_tok, T = 500, len(CTXS)
    nb = (n_tok + bs - 1) // bs
    perm = torch.randperm(nb + 3, generator=g)[:nb]
    rows = [torch.randn(n_tok, kv, d, generator=g).to(torch.bfloat16) for d in (dim, vdim)]
    caches = []
    for r in rows:   # poison behind the contexts, where nobody may look
        c = torch.full((nb + 3, kv, bs, r.shape[2]), float("nan"), dtype=torch.bfloat16)
        for j in range(n_tok):
            c[perm[j // bs], :, j % bs] = r[j]
        caches.append(c.to(DEV))
    q = (torch.randn(T, heads, dim, generator=g) * 3).to(torch.bfloat16)   # the running maximum jumps
    bt = perm.to(torch.int32)[None, :].repeat(12, 1).to(DEV)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)   # noqa: E731
    return g, q, rows, caches, bt, i32(SEQ), i32(CTXS), T


def _oracle(q, rows, scale, window=0, keep=0, cap=0.0, bias=None, sink=None, gate=None):
    T, heads, _ = q.shape
    K, V = (r.double() for r in rows)
    kv, out = K.shape[1], []
    for t in range(T):
        c = CTXS[t]
        k, v = (x[:c].repeat_interleave(heads // kv, 1) for x in (K, V))
        s = torch.einsum("hd,chd->hc", q[t].double(), k) * scale
        if cap:
            s = cap * torch.tanh(s / cap)
        dist = c - 1 - torch.arange(c)
        if bias is not None:
            s = s + bias.double()[:, dist.clamp(max=bias.shape[1] - 1)]
        if window:
            s = s.masked_fill((dist >= window) & (torch.arange(c) >= keep), float("-inf"))
        m = s.max(-1, keepdim=True).values
        m = torch.maximum(m, sink.double()[:, None]) if sink is not None else m
        e = torch.exp(s - m)
        o = torch.einsum("hc,chd->hd", e, v) / (e.sum(-1, keepdim=True) + (torch.exp(sink.double()[:, None] - m) if sink is not None else 0.0))
        out.append(o * torch.sigmoid(gate[t].double())[:, None] if gate is not None else o)
    return torch.stack(out)


def _close(out, want):
    got = out.double().cpu()
    assert torch.isfinite(got).all()
    # queries are exact in bf16 and weights carry 16 bits, so a result is rounded once: 2^-9 of itself at most, beside fp32 noise of the sums
    # (a capped score's exponential and reciprocal: a few 2^-22 of the cap)
    assert ((got - want).abs() <= 2.0 ** -8 * want.abs() + 2e-4).all(), float((got - want).abs().max())


# pairs per row: 4, 1 (128 rows a tile), 16, 5 (idle pairs); heads with a partial second chunk of columns; values narrower than keys
@pytest.mark.parametrize("heads,kv,dim,vdim,bs", [(8, 2, 128, 128, 128), (2, 2, 64, 64, 64), (16, 1, 80, 48, 128), (10, 2, 96, 128, 192)])
@pytest.mark.parametrize("form", ["plain", "capped, biased, gated", "window", "kept keys, biased, sink", "long bias", "split"])
def test_runs_of_rows_tile_edges(heads, kv, dim, vdim, bs, form):
    lib, check = pkg("_abi").lib(), pkg("_abi").check
    g, q, rows, (kc, vc), bt, seq, ctx, T = _case(heads, kv, dim, vdim, bs, heads * 100 + dim)
    scale, ns = dim ** -0.5, 3 if form == "split" else 1
    ws = torch.zeros(int(lib.b200_paged_attn_anydim_workspace_bytes(T)), dtype=torch.uint8, device=DEV)
    out = torch.full((T, heads, vdim), float("nan"), dtype=torch.bfloat16, device=DEV)
    part = torch.full((T * heads * ns * (vdim + 2),), float("nan"), device=DEV)
    qd, pos = q.float().to(DEV), (ctx - 1).contiguous()
    lead = [qd.data_ptr(), kc.data_ptr(), vc.data_ptr(), bt.data_ptr(), bt.shape[1], seq.data_ptr(), ctx.data_ptr()]
    if form in ("plain", "split"):
        sink = torch.randn(heads, generator=g).to(DEV)
        check(lib.b200_paged_attn_mma(*lead, out.data_ptr(), T, heads, kv, dim, vdim, bs, scale, sink.data_ptr(), ws.data_ptr(), 0, ns,
                                      part.data_ptr() if ns > 1 else None, None))
        want = _oracle(q, rows, scale, sink=sink.cpu())
    elif form in ("capped, biased, gated", "long bias", "window"):
        nd = 3000 if form == "long bias" else 40      # 3000: longer than the on-chip table
        cap, window = (20.0, 0) if form == "capped, biased, gated" else (0.0, 100 if form == "window" else 0)
        bias = (torch.randn(heads, nd, generator=g) if form != "window" else None)
        gate = torch.randn(T, heads, generator=g).to(torch.bfloat16)
        bd, gd = bias.to(DEV) if bias is not None else None, gate.to(DEV)
        check(lib.b200_paged_attn_biased(0, 2, *lead, pos.data_ptr(), out.data_ptr(), T, heads, kv, dim, vdim, bs, scale, window, cap,
                                         bd.data_ptr() if bd is not None else None, nd if bd is not None else 0, gd.data_ptr(), heads, ws.data_ptr(), 1,
                                         None, None))
        want = _oracle(q, rows, scale, window, 0, cap, bias, gate=gate)
    else:
        bias, sink = torch.randn(heads, 200, generator=g), torch.randn(heads, generator=g)
        bd, sd = bias.to(DEV), sink.to(DEV)
        check(lib.b200_paged_attn_kept(0, 2, *lead, pos.data_ptr(), out.data_ptr(), T, heads, kv, dim, vdim, bs, scale, 90, 70, sd.data_ptr(),
                                       bd.data_ptr(), 200, ws.data_ptr(), 1, None, None))
        want = _oracle(q, rows, scale, 90, 70, 0.0, bias, sink=sink)
    torch.cuda.synchronize()
    _close(out, want)


@pytest.mark.parametrize("heads,kv", [(8, 2), (4, 4), (8, 1), (10, 2), (64, 8), (32, 32)])
def test_prefill_rows_of_the_decoder_stack(heads, kv):
    lib, check = pkg("_abi").lib(), pkg("_abi").check
    g, q, rows, (kc, vc), bt, seq, ctx, T = _case(heads, kv, 128, 128, 128, heads * 7 + kv)
    wsb = int(lib.b200_paged_attn_workspace_bytes(T, heads, 500, 128))
    ws = torch.zeros(wsb, dtype=torch.uint8, device=DEV)
    out = torch.full((T, heads, 128), float("nan"), dtype=torch.bfloat16, device=DEV)
    qd = q.to(DEV)
    check(lib.b200_paged_attn_prefill(qd.data_ptr(), heads * 128, kc.data_ptr(), vc.data_ptr(), bt.data_ptr(), bt.shape[1], seq.data_ptr(), ctx.data_ptr(),
                                      out.data_ptr(), heads * 128, T, heads, kv, 128, 500, 128 ** -0.5, ws.data_ptr(), wsb, None))
    torch.cuda.synchronize()
    _close(out, _oracle(q, rows, 128 ** -0.5))


@pytest.mark.parametrize("ns", [1, 2])
def test_long_steps_of_decode_rows_go_to_the_other_kernel(ns):
    """More than 128 rows, almost all of them runs of one: which kernel works is decided on the device, the other leaves."""
    lib, check = pkg("_abi").lib(), pkg("_abi").check
    heads, kv, dim, bs, T = 8, 2, 64, 64, 150
    g = torch.Generator().manual_seed(3)
    K, V = (torch.randn(500, kv, dim, generator=g).to(torch.bfloat16) for _ in range(2))
    kc, vc = (torch.cat([x, torch.zeros(12, kv, dim, dtype=torch.bfloat16)]).reshape(8, bs, kv, dim).transpose(1, 2).contiguous().to(DEV) for x in (K, V))
    ctxs = [(37 * i) % 500 + 1 for i in range(T)]
    q = torch.randn(T, heads, dim, generator=g).to(torch.bfloat16)
    bt = torch.arange(8, dtype=torch.int32, device=DEV)[None, :].repeat(T, 1).contiguous()
    seq, ctx = torch.arange(T, dtype=torch.int32, device=DEV), torch.tensor(ctxs, dtype=torch.int32, device=DEV)
    ws = torch.zeros(int(lib.b200_paged_attn_anydim_workspace_bytes(T)), dtype=torch.uint8, device=DEV)
    out = torch.full((T, heads, dim), float("nan"), dtype=torch.bfloat16, device=DEV)
    part = torch.full((T * heads * ns * (dim + 2),), float("nan"), device=DEV)
    qd = q.float().to(DEV)
    check(lib.b200_paged_attn_mma(qd.data_ptr(), kc.data_ptr(), vc.data_ptr(), bt.data_ptr(), 8, seq.data_ptr(), ctx.data_ptr(), out.data_ptr(), T, heads,
                                  kv, dim, dim, bs, dim ** -0.5, None, ws.data_ptr(), 0, ns, part.data_ptr() if ns > 1 else None, None))
    torch.cuda.synchronize()
    got = out.double().cpu()
    for t in range(T):
        k, v = (x[:ctxs[t]].double().repeat_interleave(heads // kv, 1) for x in (K, V))
        w = torch.softmax(torch.einsum("hd,chd->hc", q[t].double(), k) * dim ** -0.5, -1)
        want = torch.einsum("hc,chd->hd", w, v)
        # weights and results rounded to bf16 once each: 2^-9 of the largest value, 2^-9 of the result
        assert ((got[t] - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -9 * v.abs().max()).all(), t


# The bias of a distance is that distance's alone: what the table holds for the farthest keys, a mask or a sentinel, leaves near keys as they are.
@pytest.mark.parametrize("last", [float("-inf"), -1e9, -1e4, "lowest everywhere"])
@pytest.mark.parametrize("nd", [40, 3000])       # on chip and not
@pytest.mark.parametrize("cap", [0.0, 20.0])
def test_masks_and_sentinels_in_the_distance_bias(last, nd, cap):
    lib, check = pkg("_abi").lib(), pkg("_abi").check
    heads, kv, dim, bs = 8, 2, 64, 64
    g, q, rows, (kc, vc), bt, seq, ctx, T = _case(heads, kv, dim, dim, bs, 17)
    bias = torch.randn(heads, nd, generator=g)
    if last == "lowest everywhere":
        bias[:] = torch.finfo(torch.float32).min      # nothing but sentinels: all keys weigh the same
    else:
        bias[:, 39:] = last
    ws = torch.zeros(int(lib.b200_paged_attn_anydim_workspace_bytes(T)), dtype=torch.uint8, device=DEV)
    out = torch.full((T, heads, dim), float("nan"), dtype=torch.bfloat16, device=DEV)
    qd, bd, pos = q.float().to(DEV), bias.to(DEV), (ctx - 1).contiguous()
    check(lib.b200_paged_attn_biased(0, 2, qd.data_ptr(), kc.data_ptr(), vc.data_ptr(), bt.data_ptr(), bt.shape[1], seq.data_ptr(), ctx.data_ptr(),
                                     pos.data_ptr(), out.data_ptr(), T, heads, kv, dim, dim, bs, dim ** -0.5, 0, cap, bd.data_ptr(), nd, None, 0,
                                     ws.data_ptr(), 1, None, None))
    torch.cuda.synchronize()
    _close(out, _oracle(q, rows, dim ** -0.5, cap=cap, bias=bias))


@pytest.mark.parametrize("scale", [0.0, -0.1])
@pytest.mark.parametrize("cap", [0.0, 20.0])
def test_scales_that_are_not_positive(scale, cap):
    lib, check = pkg("_abi").lib(), pkg("_abi").check
    heads, kv, dim, bs = 8, 2, 64, 64
    g, q, rows, (kc, vc), bt, seq, ctx, T = _case(heads, kv, dim, dim, bs, 23)
    ws = torch.zeros(int(lib.b200_paged_attn_anydim_workspace_bytes(T)), dtype=torch.uint8, device=DEV)
    out = torch.full((T, heads, dim), float("nan"), dtype=torch.bfloat16, device=DEV)
    qd, pos = q.float().to(DEV), (ctx - 1).contiguous()
    lead = [qd.data_ptr(), kc.data_ptr(), vc.data_ptr(), bt.data_ptr(), bt.shape[1], seq.data_ptr(), ctx.data_ptr()]
    if cap:
        check(lib.b200_paged_attn_biased(0, 2, *lead, pos.data_ptr(), out.data_ptr(), T, heads, kv, dim, dim, bs, scale, 0, cap, None, 0, None, 0,
                                         ws.data_ptr(), 1, None, None))
    else:
        check(lib.b200_paged_attn_mma(*lead, out.data_ptr(), T, heads, kv, dim, dim, bs, scale, None, ws.data_ptr(), 0, 1, None, None))
    torch.cuda.synchronize()
    got, want = out.double().cpu(), _oracle(q, rows, scale, cap=cap)
    # weights and results rounded to bf16 once each: 2^-9 of the largest value, 2^-9 of the result
    assert ((got - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -9 * rows[1].float().abs().max()).all()


def _dense(q, rows, ctxs, scale, window=0):
    """All rows at once over the same cached tokens, float64."""
    K, V = (r.double() for r in rows)
    G, c = q.shape[1] // K.shape[1], torch.tensor(ctxs)[:, None]
    j = torch.arange(K.shape[0])[None, :]
    seen = (j < c) & ((j >= c - window) if window else (j >= 0))
    s = torch.einsum("thd,chd->thc", q.double(), K.repeat_interleave(G, 1)) * scale
    return torch.einsum("thc,chd->thd", torch.softmax(s.masked_fill(~seen[:, None], float("-inf")), -1), V.repeat_interleave(G, 1))


def _steps(runs):
    """(first context, rows) per run of a sequence of its own -> sequence and context of every row."""
    return [s for s, (_, n) in enumerate(runs) for _ in range(n)], [c + i for c, n in runs for i in range(n)]


_MIX = [(7 * i % 180 + 1, 1) for i in range(300)] + [(5, 2), (60, 3), (1, 5), (33, 8), (100, 9), (64, 15), (20, 16), (1, 17), (127, 40), (3, 100)]
_MIX = _MIX[:150] + _MIX[300:] + _MIX[150:300] + [(50 + i, 2) for i in range(8)]      # long runs between decode rows


# Which kernel takes a run, over steps that both share or one has to itself, and walks of several trips in either: a mixed step (300 runs of one
# row, others of 2 to 100) with 16 heads over 4, 32 over 2, splits, a window; decode rows only; runs at the border of 16 pairs an item; few
# rows with many heads a group (items of 8 rows); 5 120 items of 40 rows (more than a CTA describes ahead).
@pytest.mark.parametrize("heads,kv,dim,runs,ns,window", [
    (16, 4, 64, _MIX, 1, 0), (16, 4, 64, _MIX, 2, 0), (32, 2, 48, _MIX, 1, 0), (32, 2, 64, _MIX, 2, 50), (8, 8, 32, _MIX, 1, 0),
    (16, 4, 64, [(i % 190 + 1, 1) for i in range(400)], 1, 0), (16, 4, 64, [(3 * i + 1, 4) for i in range(50)], 1, 0),
    (16, 4, 64, [(3 * i + 1, 5) for i in range(50)], 1, 0), (16, 1, 64, [(9 * i + 1, 12) for i in range(14)], 1, 40), (16, 1, 128, [(30, 150)], 1, 0),
    (2, 2, 64, [(1, 180)], 1, 0), (32, 32, 16, [(i % 120 + 1, 40) for i in range(160)], 1, 0)])
def test_runs_shared_between_the_kernels(heads, kv, dim, runs, ns, window):
    lib, check = pkg("_abi").lib(), pkg("_abi").check
    bs, n_tok = 64, 192
    seq, ctxs = _steps(runs)
    T, g = len(seq), torch.Generator().manual_seed(heads + dim)
    rows = [torch.randn(n_tok, kv, dim, generator=g).to(torch.bfloat16) for _ in range(2)]
    kc, vc = (r.reshape(n_tok // bs, bs, kv, dim).transpose(1, 2).contiguous().to(DEV) for r in rows)
    q = torch.randn(T, heads, dim, generator=g).to(torch.bfloat16)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)   # noqa: E731
    bt, sq, cx = i32([[0, 1, 2]]).repeat(len(runs), 1).contiguous(), i32(seq), i32(ctxs)
    ws = torch.zeros(int(lib.b200_paged_attn_anydim_workspace_bytes(T)), dtype=torch.uint8, device=DEV)
    out = torch.full((T, heads, dim), float("nan"), dtype=torch.bfloat16, device=DEV)
    part = torch.full((T * heads * ns * (dim + 2),), float("nan"), device=DEV)
    qd = q.float().to(DEV)
    check(lib.b200_paged_attn_mma(qd.data_ptr(), kc.data_ptr(), vc.data_ptr(), bt.data_ptr(), 3, sq.data_ptr(), cx.data_ptr(), out.data_ptr(), T, heads, kv,
                                  dim, dim, bs, dim ** -0.5, None, ws.data_ptr(), window, ns, part.data_ptr() if ns > 1 else None, None))
    torch.cuda.synchronize()
    got, want = out.double().cpu(), _dense(q, rows, ctxs, dim ** -0.5, window)
    assert torch.isfinite(got).all()
    # where the mma.sync kernel works, weights and results are rounded to bf16 once each: 2^-9 of the largest value, 2^-9 of the result
    assert ((got - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -9 * rows[1].float().abs().max()).all()
