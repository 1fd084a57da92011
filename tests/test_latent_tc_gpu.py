"""The tcgen05 form of latent attention (cache blocks of whole 64-key tiles) against the same attention in float64."""
import pytest
import torch

from conftest import pkg

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _oracle(q, rows, ctx, rank, scale, sink, window):
    lo = max(ctx - window, 0) if window else 0
    s = (q @ rows[lo:ctx].T) * scale
    m = s.max(-1, keepdim=True).values
    m = torch.maximum(m, sink[:, None]) if sink is not None else m
    e = torch.exp(s - m)
    den = e.sum(-1, keepdim=True) + (torch.exp(sink[:, None] - m) if sink is not None else 0.0)
    return (e / den) @ rows[lo:ctx, :rank]


# heads: one, a count that leaves pairs idle (5 x 16 rows = 80 of 128), the tile's own divisor, more rows than a run (1), all pairs one row (128).
# rank / rotated part: one half with a partial last chunk, two halves, the second half short, everything in TMEM (rank = row), a key row of
# nine chunks
@pytest.mark.parametrize("heads,rank,rd,bs,splits,window,with_sink", [
    (16, 512, 64, 128, 1, 0, True), (16, 512, 64, 64, 3, 0, True), (5, 256, 32, 128, 1, 0, False), (1, 16, 16, 128, 16, 0, False),
    (128, 64, 0, 128, 1, 0, True), (16, 304, 16, 64, 2, 0, False), (16, 256, 0, 128, 1, 100, True), (7, 80, 48, 192, 1, 64, False)])
def test_latent_attention_tile_edges(heads, rank, rd, bs, splits, window, with_sink):
    lib, check = pkg("_abi").lib(), pkg("_abi").check
    g = torch.Generator().manual_seed(heads * 1000 + rank)
    krow, n_tok, scale = rank + rd, 700, 0.6 / (rank + rd) ** 0.5
    nb = (n_tok + bs - 1) // bs
    rows = torch.randn(n_tok, krow, generator=g).to(torch.bfloat16)
    perm = torch.randperm(nb + 3, generator=g)[:nb]
    # decode rows of sequences of their own around tile and block edges, then two runs that start inside a tile
    ctxs = [1, 2, 63, 64, 65, 127, 128, 129, 700] + list(range(1, 39)) + list(range(650, 700))
    seq = list(range(9)) + [9] * 38 + [10] * 50
    T = len(ctxs)
    q = (torch.randn(T, heads, krow, generator=g) * 4).to(torch.bfloat16).float()   # large scores: the running maximum jumps
    sink = torch.randn(heads, generator=g) * 2 if with_sink else None
    want = torch.stack([_oracle(q[t].double(), rows.double(), ctxs[t], rank, scale, sink.double() if with_sink else None, window) for t in range(T)])
    # every sequence reads the same first n_tok rows through its own table; what lies past a context is poison where nobody may look
    kc = torch.full((nb + 3, 1, bs, krow), float("nan"), dtype=torch.bfloat16)
    for j in range(n_tok):
        kc[perm[j // bs], 0, j % bs] = rows[j]
    dev = lambda t: t.to(DEV).contiguous()   # noqa: E731
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)   # noqa: E731
    bt = dev(perm.to(torch.int32)[None, :].repeat(11, 1))
    ws = torch.zeros(int(lib.b200_paged_attn_anydim_workspace_bytes(T)), dtype=torch.uint8, device=DEV)
    out = torch.full((T, heads, rank), float("nan"), dtype=torch.bfloat16, device=DEV)
    part = torch.full((T * heads * splits * (rank + 2),), float("nan"), device=DEV)
    qd, kd, sd, sq, cx = dev(q), dev(kc), dev(sink) if with_sink else None, i32(seq), i32(ctxs)
    sp = sd.data_ptr() if with_sink else None
    if window:
        check(lib.b200_latent_attn_window(qd.data_ptr(), kd.data_ptr(), bt.data_ptr(), nb, sq.data_ptr(), cx.data_ptr(), out.data_ptr(), T, heads, krow,
                                          rank, bs, scale, sp, ws.data_ptr(), window, None))
    else:
        check(lib.b200_latent_attn(qd.data_ptr(), kd.data_ptr(), bt.data_ptr(), nb, sq.data_ptr(), cx.data_ptr(), out.data_ptr(), T, heads, krow, rank,
                                   bs, scale, sp, ws.data_ptr(), splits, part.data_ptr() if splits > 1 else None, None))
    torch.cuda.synchronize()
    got = out.double().cpu()
    assert torch.isfinite(got).all()
    # queries are exact in bf16; weights and results are rounded once each (2^-9 relative, rms 2^-9 / sqrt 3 apiece), the sum over keys only
    # averages the weights' part: below 2^-8 in the 2-norm, and no single result further off than the weights' worst case, 2^-8 of the largest value
    assert (got - want).norm() / want.norm() < 2.0 ** -8
    assert (got - want).abs().max() < 2.0 ** -8 * rows.float().abs().max() + 2.0 ** -9 * want.abs().max()


@pytest.mark.parametrize("scale", [0.0, -0.02])
def test_latent_scales_that_are_not_positive(scale):
    lib, check = pkg("_abi").lib(), pkg("_abi").check
    heads, rank, rd, bs = 4, 64, 16, 64
    g = torch.Generator().manual_seed(9)
    ctxs = [1, 63, 64, 65, 190] + list(range(20, 60))
    seq, T, krow = list(range(5)) + [5] * 40, 45, rank + rd
    rows = torch.randn(192, krow, generator=g).to(torch.bfloat16)
    q = torch.randn(T, heads, krow, generator=g).to(torch.bfloat16).float()
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)   # noqa: E731
    bt, sq, cx, kd, qd = i32([[0, 1, 2]] * 6), i32(seq), i32(ctxs), rows.reshape(3, 1, bs, krow).to(DEV), q.to(DEV)
    ws = torch.zeros(int(lib.b200_paged_attn_anydim_workspace_bytes(T)), dtype=torch.uint8, device=DEV)
    out = torch.full((T, heads, rank), float("nan"), dtype=torch.bfloat16, device=DEV)
    check(lib.b200_latent_attn(qd.data_ptr(), kd.data_ptr(), bt.data_ptr(), 3, sq.data_ptr(), cx.data_ptr(), out.data_ptr(), T, heads, krow, rank, bs,
                               scale, None, ws.data_ptr(), 1, None, None))
    torch.cuda.synchronize()
    want = torch.stack([_oracle(q[t].double(), rows.double(), ctxs[t], rank, scale, None, 0) for t in range(T)])
    # weights and results rounded to bf16 once each: 2^-9 of the largest value, 2^-9 of the result
    assert ((out.double().cpu() - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -9 * rows.float().abs().max()).all()


# Steps of many items: decode rows (the mma.sync kernel's, runs of one), rows in pairs (the tcgen05 kernel's: 32 pairs an item; 4 800 items, more
# than a CTA describes ahead), both in one step, and splits.
@pytest.mark.parametrize("heads,rank,rd,runs,splits", [
    (16, 272, 16, [1] * 400, 1), (16, 272, 16, [2] * 1200, 1), (4, 64, 16, [1] * 300 + [40, 90], 2), (16, 512, 64, [1] * 230, 1), (1, 272, 16, [1] * 64, 5)])
def test_latent_steps_of_many_items(heads, rank, rd, runs, splits):
    lib, check = pkg("_abi").lib(), pkg("_abi").check
    g = torch.Generator().manual_seed(heads + rank)
    krow, bs, scale = rank + rd, 64, 1.0 / (rank + rd) ** 0.5
    seq = [s for s, n in enumerate(runs) for _ in range(n)]
    ctxs = [(11 * s) % 90 + 1 + i for s, n in enumerate(runs) for i in range(n)]
    T, rows = len(seq), torch.randn(192, krow, generator=g).to(torch.bfloat16)
    q = torch.randn(T, heads, krow, generator=g).to(torch.bfloat16)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)   # noqa: E731
    bt, sq, cx, kd, qd = i32([[0, 1, 2]]).repeat(len(runs), 1).contiguous(), i32(seq), i32(ctxs), rows.reshape(3, 1, bs, krow).to(DEV), q.float().to(DEV)
    ws = torch.zeros(int(lib.b200_paged_attn_anydim_workspace_bytes(T)), dtype=torch.uint8, device=DEV)
    out = torch.full((T, heads, rank), float("nan"), dtype=torch.bfloat16, device=DEV)
    part = torch.full((T * heads * splits * (rank + 2),), float("nan"), device=DEV)
    check(lib.b200_latent_attn(qd.data_ptr(), kd.data_ptr(), bt.data_ptr(), 3, sq.data_ptr(), cx.data_ptr(), out.data_ptr(), T, heads, krow, rank, bs,
                               scale, None, ws.data_ptr(), splits, part.data_ptr() if splits > 1 else None, None))
    torch.cuda.synchronize()
    K = rows.double()
    s = torch.einsum("thd,cd->thc", q.double(), K) * scale
    s = s.masked_fill(torch.arange(192)[None, None, :] >= torch.tensor(ctxs)[:, None, None], float("-inf"))
    got, want = out.double().cpu(), torch.einsum("thc,cd->thd", torch.softmax(s, -1), K[:, :rank])
    assert torch.isfinite(got).all()
    # weights and results rounded to bf16 once each: 2^-9 of the largest value, 2^-9 of the result
    assert ((got - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -9 * rows.float().abs().max()).all()


# Rows by themselves (attn_latent_rows.cu): clusters of eight, four, two and one CTA, more CTAs than SMs (rows known to be sequences of their own), heads that
# are no multiple of 16, one to four pairs of value chunks with and without other chunks beside them, contexts around tiles and blocks, windows.
@pytest.mark.parametrize("T,heads,rank,rd,bs,window,with_sink,with_seq", [
    (1, 16, 512, 64, 128, 0, True, True), (15, 16, 512, 64, 64, 0, False, True), (16, 16, 256, 32, 128, 0, True, True), (33, 5, 304, 16, 64, 0, False, True),
    (34, 16, 512, 0, 128, 0, True, True), (74, 16, 128, 64, 128, 300, True, True), (75, 16, 512, 64, 128, 0, False, True), (148, 1, 16, 16, 192, 0, True, True),
    (9, 40, 512, 64, 128, 0, True, True), (3, 128, 64, 128, 64, 65, False, True), (200, 16, 512, 64, 128, 0, True, False),
    (1, 16, 512, 64, 128, -16, True, True), (2, 20, 256, 32, 64, -5, False, True), (7, 16, 80, 48, 128, -2, True, True)])   # (a negative window: so many splits)
def test_latent_rows_by_themselves(T, heads, rank, rd, bs, window, with_sink, with_seq):
    lib, check = pkg("_abi").lib(), pkg("_abi").check
    splits, window = max(-window, 1), max(window, 0)
    g = torch.Generator().manual_seed(T * 1000 + rank + heads)
    krow, n_tok, scale = rank + rd, 1200, 0.6 / (rank + rd) ** 0.5
    nb = (n_tok + bs - 1) // bs
    rows = torch.randn(n_tok, krow, generator=g).to(torch.bfloat16)
    perm = torch.randperm(nb + 3, generator=g)[:nb]
    edges = [1, 2, 15, 16, 17, 63, 64, 65, 127, 128, 129, 143, 255, 257, 640, 1023, 1025, 1200]
    ctxs = [edges[(i * 7 + T) % len(edges)] for i in range(T)]
    q = (torch.randn(T, heads, krow, generator=g) * 4).to(torch.bfloat16).float()   # large scores: the running maximum jumps
    sink = torch.randn(heads, generator=g) * 2 if with_sink else None
    want = torch.stack([_oracle(q[t].double(), rows.double(), ctxs[t], rank, scale, sink.double() if with_sink else None, window) for t in range(T)])
    kc = torch.full((nb + 3, 1, bs, krow), float("nan"), dtype=torch.bfloat16)
    kc[perm] = torch.cat([rows, torch.full((nb * bs - n_tok, krow), float("nan"), dtype=torch.bfloat16)]).reshape(nb, 1, bs, krow)
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)   # noqa: E731
    bt, cx, kd, qd = perm.to(torch.int32)[None, :].repeat(T, 1).to(DEV), i32(ctxs), kc.to(DEV), q.to(DEV)
    for t, c in enumerate(ctxs):   # what lies past a context's last tile of 64 keys is nobody's block
        bt[t, ((c + 63) // 64 * 64 + bs - 1) // bs:] = 1 << 29
    if splits > 1:   # only tables for more than 32 768 tokens have them taken
        nb = 32768 // bs + 1
        bt = torch.nn.functional.pad(bt, (0, nb - bt.shape[1])).contiguous()
    sq = i32(list(range(T))) if with_seq else None
    sd = sink.to(DEV) if with_sink else None
    ws = torch.zeros(int(lib.b200_paged_attn_anydim_workspace_bytes(T)), dtype=torch.uint8, device=DEV)
    out = torch.full((T, heads, rank), float("nan"), dtype=torch.bfloat16, device=DEV)
    args = (qd.data_ptr(), kd.data_ptr(), bt.data_ptr(), nb, sq.data_ptr() if with_seq else None, cx.data_ptr(), out.data_ptr(), T, heads, krow, rank, bs, scale,
            sd.data_ptr() if with_sink else None, ws.data_ptr())
    if splits > 1:
        part = torch.full((T * heads * splits * (rank + 2),), float("nan"), device=DEV)
        check(lib.b200_latent_attn(*args, splits, part.data_ptr(), None))
    else:
        check(lib.b200_latent_attn_window(*args, window, None))
    torch.cuda.synchronize()
    got = out.double().cpu()
    assert torch.isfinite(got).all()
    # (as above)
    assert (got - want).norm() / want.norm() < 2.0 ** -8
    assert (got - want).abs().max() < 2.0 ** -8 * rows.float().abs().max() + 2.0 ** -9 * want.abs().max()


# A window's older blocks may be anybody's: what the table names before the block of the oldest visible key is not read.  Rows by themselves, a row of many heads
# and runs of rows; blocks of one, three and five times 64, windows whose oldest key lies in the first, a middle and the last 64 of one.
@pytest.mark.parametrize("T,heads,rank,rd,bs,window,with_seq", [
    (18, 16, 128, 64, 64, 65, True), (40, 16, 512, 64, 64, 300, True), (100, 16, 256, 32, 192, 130, True), (18, 16, 64, 16, 320, 64, True), (5, 48, 512, 0, 64, 1, True),
    (200, 8, 128, 64, 64, 70, False), (200, 16, 128, 64, 64, 65, True)])
def test_latent_windows_leave_passed_blocks_alone(T, heads, rank, rd, bs, window, with_seq):
    lib, check = pkg("_abi").lib(), pkg("_abi").check
    g = torch.Generator().manual_seed(T + heads + bs)
    krow, n_tok, scale = rank + rd, 1280, 0.6 / (rank + rd) ** 0.5
    nb = (n_tok + bs - 1) // bs
    rows = torch.randn(nb * bs, krow, generator=g).to(torch.bfloat16)
    kc = torch.cat([rows.reshape(nb, 1, bs, krow), torch.full((1, 1, bs, krow), float("nan"), dtype=torch.bfloat16)]).to(DEV)   # block nb: another's
    ctxs = [1 + (i * 61 + window) % n_tok for i in range(T)]
    q = torch.randn(T, heads, krow, generator=g).to(torch.bfloat16).float()
    want = torch.stack([_oracle(q[t].double(), rows.double(), ctxs[t], rank, scale, None, window) for t in range(T)])
    bt = torch.arange(nb, dtype=torch.int32).repeat(T, 1)
    for t, c in enumerate(ctxs):
        bt[t, :max(c - window, 0) // bs] = nb
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)   # noqa: E731
    bt, cx, sq, qd = bt.to(DEV), i32(ctxs), i32(list(range(T))), q.to(DEV)
    ws = torch.zeros(int(lib.b200_paged_attn_anydim_workspace_bytes(T)), dtype=torch.uint8, device=DEV)
    out = torch.full((T, heads, rank), float("nan"), dtype=torch.bfloat16, device=DEV)
    check(lib.b200_latent_attn_window(qd.data_ptr(), kc.data_ptr(), bt.data_ptr(), nb, sq.data_ptr() if with_seq else None, cx.data_ptr(), out.data_ptr(), T, heads,
                                      krow, rank, bs, scale, None, ws.data_ptr(), window, None))
    torch.cuda.synchronize()
    got = out.double().cpu()
    assert torch.isfinite(got).all()
    # (as above)
    assert (got - want).norm() / want.norm() < 2.0 ** -8
    assert (got - want).abs().max() < 2.0 ** -8 * rows.float().abs().max() + 2.0 ** -9 * want.abs().max()


# Runs of rows whose key rows have every count of chunks that are a half's own (1..4) and that are not (0..5), the last one whole or of one to three 16-wide steps;
# then two halves of an odd number of chunks (the middle one is in both), with and without splits.
@pytest.mark.parametrize("rank,rd,splits", [(64 * o - 16 * (r % 3), 64 * r + 16 * (r % 3) - (16 * ((o + r) % 4) if r else 0), 1) for o in range(1, 5) for r in range(6)] + [
    (80, 0, 1), (272, 0, 1), (272, 16, 2), (288, 16, 1), (320, 32, 2), (336, 0, 1), (400, 48, 2), (448, 64, 3), (448, 0, 1), (464, 0, 2)])
def test_latent_runs_of_every_count_of_chunks(rank, rd, splits):
    lib, check = pkg("_abi").lib(), pkg("_abi").check
    heads, bs, seqs, krow = 4, 128, [(150, 1), (33, 300), (17, 64)], rank + rd
    g = torch.Generator(device=DEV).manual_seed(krow * 7 + rank)
    seq, ctx = [s for s, (n, _) in enumerate(seqs) for _ in range(n)], [c + i for n, c in seqs for i in range(n)]
    T, scale = len(seq), 0.6 / krow ** 0.5
    kc = torch.randn(9, 1, bs, krow, generator=g, device=DEV).to(torch.bfloat16)
    bt = torch.randperm(9, generator=g, device=DEV).to(torch.int32).reshape(3, 3).contiguous()
    q = (torch.randn(T, heads, krow, generator=g, device=DEV) * 3).to(torch.bfloat16).float()
    want = torch.stack([_oracle(q[t].double(), kc[bt[seq[t]].long()].reshape(-1, krow).double(), ctx[t], rank, scale, None, 0) for t in range(T)])
    sq, cx = torch.tensor(seq, dtype=torch.int32, device=DEV), torch.tensor(ctx, dtype=torch.int32, device=DEV)
    ws = torch.zeros(int(lib.b200_paged_attn_anydim_workspace_bytes(T)), dtype=torch.uint8, device=DEV)
    part = torch.full((T * heads * splits * (rank + 2),), float("nan"), device=DEV)
    out = torch.full((T, heads, rank), float("nan"), dtype=torch.bfloat16, device=DEV)
    check(lib.b200_latent_attn(q.data_ptr(), kc.data_ptr(), bt.data_ptr(), 3, sq.data_ptr(), cx.data_ptr(), out.data_ptr(), T, heads, krow, rank, bs, scale, None,
                               ws.data_ptr(), splits, part.data_ptr() if splits > 1 else None, None))
    torch.cuda.synchronize()
    got = out.double()
    assert torch.isfinite(got).all()
    # (as above)
    assert (got - want).norm() / want.norm() < 2.0 ** -8
    assert (got - want).abs().max() < 2.0 ** -8 * kc.float().abs().max() + 2.0 ** -9 * want.abs().max()


def test_latent_splits_of_halves_whose_maxima_part():
    """The halves of the value columns add a score's terms in different orders.  Here one of them follows the running maximum (17 units, just over the limit of
    2^8) and the other does not (16, what fp32 leaves of 2^24 + 17 - 2^24): the split's sums have to mean the same in both.  All values are 1."""
    lib, check = pkg("_abi").lib(), pkg("_abi").check
    rank, krow, bs, T, heads, splits = 512, 576, 128, 160, 2, 2
    kc = torch.ones(3, 1, bs, krow)
    kc[..., rank:] = 0.0
    kc[..., 0] = kc[..., 256] = 0.0
    kc[0, 0, 70, 0], kc[0, 0, 70, 256], kc[0, 0, 70, 512] = 4096.0, -4096.0, 17.0
    q = torch.zeros(T, heads, krow)
    q[..., 0] = q[..., 256] = 4096.0
    q[..., 512] = 1.0
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)   # noqa: E731
    kd, qd, bt, sq, cx = kc.to(torch.bfloat16).to(DEV), q.to(DEV), i32([[0, 1, 2]]), i32([0] * T), i32(list(range(200, 200 + T)))
    ws = torch.zeros(int(lib.b200_paged_attn_anydim_workspace_bytes(T)), dtype=torch.uint8, device=DEV)
    part = torch.full((T * heads * splits * (rank + 2),), float("nan"), device=DEV)
    out = torch.full((T, heads, rank), float("nan"), dtype=torch.bfloat16, device=DEV)
    check(lib.b200_latent_attn(qd.data_ptr(), kd.data_ptr(), bt.data_ptr(), 3, sq.data_ptr(), cx.data_ptr(), out.data_ptr(), T, heads, krow, rank, bs, 0.336, None,
                               ws.data_ptr(), splits, part.data_ptr(), None))
    torch.cuda.synchronize()
    got = out.float().cpu()
    got[..., 0] = got[..., 256] = 1.0
    assert (got - 1.0).abs().max() < 2.0 ** -7, got.amax()
