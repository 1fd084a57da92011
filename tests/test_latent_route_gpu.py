"""Steps of latent attention that either kernel may take (block tables for long contexts, splits given): the one that the run plan speaks for takes
them whole, against the same attention in float64."""
import pytest
import torch

from conftest import pkg

pytestmark = pytest.mark.gpu
DEV = "cuda"


# one sequence of many rows and a long row among short ones go over runs in splits; rows of sequences of their own, long or short, by themselves, as long as
# their heads do not fill the other kernel's tile
@pytest.mark.parametrize("heads,rank,rd,seqs,splits,with_seq,over_runs", [
    (16, 512, 64, [(100, 9000)], 3, True, True),
    (16, 512, 64, [(1, 5000)] * 100, 3, True, False),
    (16, 512, 64, [(1, 300 + 7 * i) for i in range(99)] + [(1, 20000)], 3, True, True),
    (16, 512, 64, [(1, 300 + 7 * i) for i in range(99)] + [(1, 20000)], 3, False, True),
    (16, 512, 64, [(1, 1 + 3 * i) for i in range(75)], 4, True, False),
    (40, 256, 32, [(20, 1), (1, 77), (17, 64)], 3, True, False),
    (128, 256, 32, [(1, 12000 - i) for i in range(18)], 3, True, True),
    (4, 128, 64, [(148, 12000)], 8, True, True),
])
def test_steps_that_either_kernel_may_take(heads, rank, rd, seqs, splits, with_seq, over_runs):
    lib, check = pkg("_abi").lib(), pkg("_abi").check
    g = torch.Generator(device=DEV).manual_seed(heads + rank + len(seqs))
    krow, bs, scale, longest = rank + rd, 128, 0.6 / (rank + rd) ** 0.5, 32768
    need = [(ctx + n + bs - 1) // bs for n, ctx in seqs]
    kc = torch.randn(sum(need) + 1, 1, bs, krow, generator=g, device=DEV).to(torch.bfloat16)
    order, at = (torch.randperm(sum(need), generator=g, device=DEV) + 1).to(torch.int32), 0
    bt = torch.zeros(len(seqs), longest // bs, dtype=torch.int32, device=DEV)
    for s, n in enumerate(need):
        bt[s, :n] = order[at:at + n]
        at += n
    seq, ctx = [s for s, (n, _) in enumerate(seqs) for _ in range(n)], [c + i for n, c in seqs for i in range(n)]
    T = len(seq)
    q = torch.randn(T, heads, krow, generator=g, device=DEV).to(torch.bfloat16).float() * 4
    sink = torch.randn(heads, generator=g, device=DEV)
    want = torch.empty(T, heads, rank, dtype=torch.float64, device=DEV)
    for t in range(T):
        if t == 0 or seq[t] != seq[t - 1]:
            rows = kc[bt[seq[t], :need[seq[t]]].long()].reshape(-1, krow).double()
        s = (q[t].double() @ rows[:ctx[t]].T) * scale
        m = torch.maximum(s.max(-1, keepdim=True).values, sink[:, None].double())
        e = torch.exp(s - m)
        want[t] = (e / (e.sum(-1, keepdim=True) + torch.exp(sink[:, None].double() - m))) @ rows[:ctx[t], :rank]
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)   # noqa: E731
    sq, cx, ws = i32(seq), i32(ctx), torch.zeros(int(lib.b200_paged_attn_anydim_workspace_bytes(T)), dtype=torch.uint8, device=DEV)
    for _ in range(2):
        out = torch.full((T, heads, rank), float("nan"), dtype=torch.bfloat16, device=DEV)
        part = torch.full((T * heads * splits * (rank + 2),), float("nan"), device=DEV)
        check(lib.b200_latent_attn(q.data_ptr(), kc.data_ptr(), bt.data_ptr(), longest // bs, sq.data_ptr() if with_seq else None, cx.data_ptr(),
                                   out.data_ptr(), T, heads, krow, rank, bs, scale, sink.data_ptr(), ws.data_ptr(), splits, part.data_ptr(), None))
        torch.cuda.synchronize()
        got = out.double()
        assert torch.isfinite(got).all() and bool(torch.isnan(part).all()) is not over_runs
        # weights of two bf16 terms, results rounded to bf16 once: 2^-9 of a result and of the largest value
        assert (got - want).norm() / want.norm() < 2.0 ** -8
        assert (got - want).abs().max() < 2.0 ** -8 * kc.float().abs().max() + 2.0 ** -9 * want.abs().max()


def test_steps_whose_rows_go_by_themselves_build_no_run_plan():
    """The same step with cache blocks that the kernel of rows by themselves reads, and with blocks that it does not: one launch less, the same logits."""
    import dupolorn_util as D
    import stack_util as U
    cfg = D.make_cfg(width=128, layers=[D.latent(heads=4, dim=16, rot_dim=16, rot_dims=16, vdim=8, kv_rank=32), D.latent(second=True, heads=8, dim=16, rot_dim=16, vdim=8, kv_rank=48)])
    w, ids = D.make_weights(cfg, 3), torch.randint(0, 150, (45,), generator=torch.Generator().manual_seed(5)).tolist()
    launches, logits = [], []
    for bs in (64, 96):
        r = D.make_runner(cfg, w, "bfloat16", block_size=bs, n_blocks=12)
        logits.append(U.replay(U.make_engine(r), [[("p", 45)]], {"p": ids})["p"])
        launches.append(r.last_step_launches())
        r.close()
    assert launches[0] == launches[1] - 1
    e = U.rel_rms(logits[0], logits[1])
    assert (e < 0.15).mean() > 0.9, float(e.max())   # (two kernels in bf16, as between schedules of the model's own tests)
