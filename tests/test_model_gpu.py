"""GPU parity of the whole decode path (C-ABI b200_decode_step / b200_decode_step_host through
the runner and the engine) against the oracle and the frozen golden fixtures.

Bars: per-step logits within bf16 tolerance — max abs error after softmax <= 2e-2,
here held to 2e-3 on the tiny fixtures — and greedy-token agreement, margin-aware: a mismatch is
allowed only where the oracle's own top-1/top-2 logit margin is below MARGIN (random-init logits
are nearly flat)."""
import numpy as np
import pytest
import torch

from conftest import pkg
from oracle import decode_oracle as O

pytestmark = pytest.mark.gpu
MARGIN = 0.08      # ~ 2.5 bf16 ulps at logit magnitude ~4


def make_runner(cfg_o, w, **kw):
    C, R = pkg("config"), pkg("runner")
    cfg = C.ModelConfig(**cfg_o.to_dict())
    kw.setdefault("max_tokens", 256)
    kw.setdefault("max_model_len", 1024)
    kw.setdefault("n_blocks", 64)
    r = R.ModelRunner(cfg, **kw)
    r.load_weights(w)
    return r


def teacher_forced_logits(r, ids, chunk=None, block_ids=None):
    """Run `ids` of one sequence through b200_decode_step in chunks; returns fp32 logits [T,V]."""
    T, bs = len(ids), r.block_size
    nblk = (T + bs - 1) // bs
    block_ids = block_ids or list(range(nblk))[::-1]
    bt = torch.tensor([block_ids], dtype=torch.int32, device="cuda")
    out = []
    chunk = chunk or T
    for s in range(0, T, chunk):
        e = min(T, s + chunk)
        pos = torch.arange(s, e, dtype=torch.int32)
        slots = torch.tensor([block_ids[p // bs] * bs + p % bs for p in range(s, e)], dtype=torch.int32)
        n = e - s
        logits = torch.empty(n, r.cfg.vocab, dtype=torch.bfloat16, device="cuda")
        toks = r.step_device(torch.tensor(ids[s:e], dtype=torch.int32).cuda(), pos.cuda(), slots.cuda(), bt,
                             (pos + 1).cuda(), e, row_to_seq=torch.zeros(n, dtype=torch.int32).cuda(),
                             out_logits=logits)
        torch.cuda.synchronize()
        assert toks.cpu().tolist() == logits.float().argmax(-1).cpu().tolist()
        out.append(logits.float().cpu())
    return torch.cat(out)


def assert_logits_close(got, want, softmax_tol=2e-3):
    err = (torch.softmax(got, -1) - torch.softmax(want, -1)).abs().max().item()
    assert err <= softmax_tol, f"softmax max abs err {err:.3e}"
    assert err <= 2e-2   # the bar
    dis = got.argmax(-1) != want.argmax(-1)
    margins = O.top2_margin(want)
    assert (margins[dis] < MARGIN).all(), f"greedy disagreement at oracle margin {margins[dis].max():.3f}"
    return err, int(dis.sum())


@pytest.mark.parametrize("name", ["tiny", "tiny-qwen", "tiny-g8"])
@pytest.mark.parametrize("graphs", [False, True])
def test_teacher_forced_logits_vs_golden(name, graphs, golden_dir):
    g = np.load(f"{golden_dir}/{name}.npz")
    cfg = O.CONFIGS[name]
    w = O.make_weights(cfg, seed=int(g["seed"]), norm_jitter=float(g["norm_jitter"]))
    assert O.weights_digest(w) == str(g["digest"])
    r = make_runner(cfg, w, graphs=graphs)
    ids = g["prompt"].tolist() + g["tokens"].tolist()[:-1]
    want = torch.from_numpy(g["tf_logits"])
    got = teacher_forced_logits(r, ids)                       # one prefill chunk of T rows
    assert_logits_close(got, want)
    got2 = teacher_forced_logits(r, ids, chunk=5)             # chunked prefill: same cache, same logits
    assert_logits_close(got2, want)
    got3 = teacher_forced_logits(r, ids, chunk=1)             # pure decode steps (GEMV path)
    assert_logits_close(got3, want)
    # and against the frozen HF stand-in
    assert (torch.softmax(got3, -1) - torch.softmax(torch.from_numpy(g["hf_logits"]), -1)).abs().max() <= 2e-2
    r.close()


@pytest.mark.parametrize("name", ["tiny", "tiny-qwen", "tiny-g8"])
def test_folded_norm_step_is_bit_identical_to_the_unfused_step(name, golden_dir, monkeypatch):
    """Steps of <= 64 rows keep the residual stream in fp32 and fold every RMSNorm into the neighbouring linears
    (B200_FUSE_NORM_MAX_T=0 switches that off): same rounding points, same summation order -> the logits of chunked
    prefill steps (5 and 33 rows) and of single-row decode steps are equal bit for bit, with and without CUDA graphs."""
    g = np.load(f"{golden_dir}/{name}.npz")
    cfg = O.CONFIGS[name]
    w = O.make_weights(cfg, seed=int(g["seed"]), norm_jitter=float(g["norm_jitter"]))
    ids = g["prompt"].tolist() + g["tokens"].tolist()[:-1]
    out = {}
    for fold in (0, 64):
        monkeypatch.setenv("B200_FUSE_NORM_MAX_T", str(fold))
        for graphs in (False, True):
            r = make_runner(cfg, w, graphs=graphs)
            out[(fold, graphs)] = [teacher_forced_logits(r, ids, chunk=c) for c in (33, 5, 1)]
            if fold:
                n = r.last_step_launches()
                assert n <= 5 * cfg.n_layers + 4 + 2, f"{n} launches in a folded single-row step"
            r.close()
    for graphs in (False, True):
        for a, b in zip(out[(0, graphs)], out[(64, graphs)]):
            assert torch.equal(a, b)
    assert_logits_close(out[(64, True)][2], torch.from_numpy(g["tf_logits"]))


@pytest.mark.parametrize("name", ["tiny", "tiny-g8"])
def test_overlapped_engine_steps_give_the_synchronous_tokens(name, golden_dir, monkeypatch):
    """LLMEngine enqueues step n+1 before it reads step n (ids of the decode rows are codes -(j+1) that the embedding
    kernel resolves from the tokens step n left on the device; two pinned buffer pairs): the tokens equal those of the
    synchronous engine (B200_ENGINE_ASYNC=0) exactly, through chunked prefill, staggered arrivals and a stop token the
    host cannot foresee.  Also the raw contract: a coded step equals the step with the ids spelled out."""
    g = np.load(f"{golden_dir}/{name}.npz")
    cfg = O.CONFIGS[name]
    w = O.make_weights(cfg, seed=int(g["seed"]), norm_jitter=float(g["norm_jitter"]))
    E, R = pkg("engine"), pkg("runner")
    prompts = [g["prompt"].tolist()] + [O.make_prompt(cfg, i, n) for i, n in ((1, 5), (2, 130), (3, 64), (4, 17))]
    outs = {}
    for mode in ("0", "1"):
        monkeypatch.setenv("B200_ENGINE_ASYNC", mode)
        r = make_runner(cfg, w)
        eng = E.LLMEngine(r, max_num_batched_tokens=64, max_num_seqs=8, max_model_len=1024)
        assert eng.overlap == (mode == "1")
        reqs = [E.Request(f"q{i}", list(p), max_tokens=24 + 3 * i, ignore_eos=True) for i, p in enumerate(prompts)]
        if "0" in outs:     # second pass: stop request 1 at a token it is known to produce
            reqs[1].stop_token_ids = (outs["0"][1][7],)
        for i, q in enumerate(reqs):
            if i < 3:
                eng.add_request(q)
        n = 0
        while eng.has_work() or n < 4:
            if n == 3:
                eng.add_request(reqs[3])
                eng.add_request(reqs[4])
            eng.step()
            n += 1
        outs[mode] = [q.output_ids for q in reqs]
        assert len(eng.blocks.free) == r.n_blocks
        if mode == "1":
            # raw contract on the same runner: step A (ids known), then step B with codes == step B with ids
            bs = r.block_size
            def batch(ids, pos):
                return R.StepBatch(ids=list(ids), positions=[pos, pos], slots=[0 * bs + pos, 1 * bs + pos], ctx_lens=[pos + 1] * 2,
                                   row_to_seq=[0, 1], logit_rows=[0, 1], block_tables=[[0], [1]])
            t0 = r.step_result(r.step_async(batch([5, 9], 0))).tolist()
            hb = r.step_async(batch([-2, -1], 1))            # row 0 <- token of logit row 1, row 1 <- token of row 0
            tb = r.step_result(hb).tolist()
            assert r.step(batch([5, 9], 0)).tolist() == t0
            assert r.step(batch([t0[1], t0[0]], 1)).tolist() == tb
        r.close()
    want = outs["0"]
    cut = want[1].index(want[1][7]) + 1
    assert outs["1"][1] == want[1][:cut]
    for i in (0, 2, 3, 4):
        assert outs["1"][i] == want[i]


@pytest.mark.parametrize("name", ["tiny", "tiny-g8"])
def test_engine_greedy_generation_vs_oracle(name, golden_dir):
    """Free-running greedy through the serving engine (scheduler, block manager, host-buffer step):
    tokens equal the oracle's until the first near-tie; report-and-allow only below MARGIN."""
    g = np.load(f"{golden_dir}/{name}.npz")
    cfg = O.CONFIGS[name]
    w = O.make_weights(cfg, seed=int(g["seed"]), norm_jitter=float(g["norm_jitter"]))
    r = make_runner(cfg, w)
    E = pkg("engine")
    eng = E.LLMEngine(r, max_num_batched_tokens=64, max_num_seqs=8, max_model_len=1024)
    om = O.OracleModel(cfg, w, capacity=512)
    prompts = [g["prompt"].tolist()] + [O.make_prompt(cfg, i, n) for i, n in ((1, 5), (2, 130), (3, 64))]
    n_new = 40
    outs = eng.generate(prompts, max_tokens=n_new)
    for p, got in zip(prompts, outs):
        want, logits = om.generate(p, n_new, keep_logits=True)
        assert len(got) == n_new
        for i, (a, b) in enumerate(zip(got, want)):
            if a != b:
                m = float(O.top2_margin(logits[i]))
                assert m < MARGIN, f"diverged at step {i} with oracle margin {m:.3f}"
                break
    assert outs[0][:8] == g["tokens"].tolist()[:8]
    assert len(eng.blocks.free) == r.n_blocks
    r.close()


def test_engine_sampling_is_seeded_and_mixes_with_greedy(golden_dir):
    """Non-greedy requests through the serving engine: a seed replays its tokens, another seed does not, a
    greedy request in the same batch keeps the oracle-checked greedy tokens, top_k = 1 is greedy."""
    g = np.load(f"{golden_dir}/tiny.npz")
    cfg = O.CONFIGS["tiny"]
    w = O.make_weights(cfg, seed=int(g["seed"]), norm_jitter=float(g["norm_jitter"]))
    r = make_runner(cfg, w)
    E = pkg("engine")
    prompt = g["prompt"].tolist()

    def run(specs, n_new=24):
        eng = E.LLMEngine(r, max_num_batched_tokens=64, max_num_seqs=8, max_model_len=1024)
        reqs = [E.Request(f"r{i}", list(prompt), max_tokens=n_new, ignore_eos=True, **kw) for i, kw in enumerate(specs)]
        for q in reqs:
            eng.add_request(q)
        while eng.has_work():
            eng.step()
        assert len(eng.blocks.free) == r.n_blocks
        return [q.output_ids for q in reqs]

    # same batch shape in every run: the rows of a step are independent, but a different row count changes the
    # split-K plan and with it the last bits of near-tied random-init logits
    greedy = run([{}] * 5)
    a = run([dict(temperature=1.5, seed=11), {}, dict(temperature=1.5, seed=12), dict(temperature=0.9, top_k=1, seed=3),
             dict(temperature=1.5, top_p=0.9, top_k=50, seed=11)])
    b = run([dict(temperature=1.5, seed=11), dict(temperature=0.7, seed=5), {}, {}, dict(temperature=2.0, seed=99)])
    assert a[1] == greedy[1] and b[2] == greedy[2]    # a greedy row is untouched by its neighbours' sampling
    assert a[3] == greedy[3]                          # top_k = 1
    assert a[0] == b[0]                               # same seed, same tokens (whatever else is in the batch)
    assert a[0] != a[2] and a[0] != greedy[0]         # another seed / not the argmax path
    assert all(0 <= t < cfg.vocab for o in a for t in o)
    # logprobs of a greedy request: the chosen token is the most likely one, values are log-probabilities
    eng = E.LLMEngine(r, max_num_batched_tokens=64, max_num_seqs=8, max_model_len=1024)
    q = E.Request("lp", list(prompt), max_tokens=6, ignore_eos=True, logprobs=3)
    eng.add_request(q)
    while eng.has_work():
        eng.step()
    assert len(q.logprob_data) == 6
    for tok, (lp, top) in zip(q.output_ids, q.logprob_data):
        assert top[0][0] == tok and abs(top[0][1] - lp) < 1e-6 and lp <= 0 and top[0][1] >= top[1][1] >= top[2][1]
    r.close()


def test_batch_of_decode_rows_matches_single_sequence_runs():
    """Continuous batching must not change a sequence's logits beyond accumulation-order noise:
    3 sequences of different lengths decoded together vs one by one."""
    cfg = O.CONFIGS["tiny"]
    w = O.make_weights(cfg, norm_jitter=0.1)
    r = make_runner(cfg, w)
    om = O.OracleModel(cfg, w, capacity=512)
    seqs = [O.make_prompt(cfg, 10 + i, n) for i, n in enumerate((3, 129, 200))]
    bs = r.block_size
    tables = [[5], [9, 2], [7, 11]]
    # prefill each (all but the last token), then one batched decode step with the last tokens
    for ids, tb in zip(seqs, tables):
        teacher_forced_logits(r, ids[:-1], block_ids=tb + [0] * 0)
    T = len(seqs)
    bt = torch.zeros(T, 2, dtype=torch.int32)
    for i, tb in enumerate(tables):
        bt[i, :len(tb)] = torch.tensor(tb)
    pos = torch.tensor([len(s) - 1 for s in seqs], dtype=torch.int32)
    slots = torch.tensor([tables[i][int(p) // bs] * bs + int(p) % bs for i, p in enumerate(pos)], dtype=torch.int32)
    logits = torch.empty(T, cfg.vocab, dtype=torch.bfloat16, device="cuda")
    r.step_device(torch.tensor([s[-1] for s in seqs], dtype=torch.int32).cuda(), pos.cuda(), slots.cuda(), bt.cuda(),
                  (pos + 1).cuda(), int(pos.max()) + 1, out_logits=logits)
    torch.cuda.synchronize()
    for i, ids in enumerate(seqs):
        want = om.forward(om.new_seq(), ids)[-1].float()
        assert_logits_close(logits[i].float().cpu()[None], want[None])
    r.close()


def test_full_width_8b_two_layers_vs_oracle():
    """Shape-faithful Llama-3.1-8B (h 4096, I 14336, 32/8 heads, V 128256) truncated to 2 layers,
    oracle run live: decode rows at the real GEMV/attention shapes."""
    cfg = O.truncated(O.CONFIGS["llama-3.1-8b"], 2)
    w = O.make_weights(cfg, seed=7)
    r = make_runner(cfg, w, max_tokens=64, max_model_len=512, n_blocks=8)
    ids = O.make_prompt(cfg, 0, 20)
    want = O.OracleModel(cfg, w, capacity=64).forward(O.OracleModel(cfg, w, capacity=64).new_seq(), ids).float()
    got = teacher_forced_logits(r, ids, chunk=1)
    assert_logits_close(got, want, softmax_tol=2e-3)
    got = teacher_forced_logits(r, ids, chunk=20)
    assert_logits_close(got, want, softmax_tol=2e-3)
    r.close()


@pytest.mark.parametrize("name,layers,vocab", [("qwen2-32b", 2, 8192), ("llama-3.1-70b", 1, 8192)])
def test_full_width_other_families_vs_oracle(name, layers, vocab):
    """Shape-faithful DeepSeek-R1-Distill-Qwen-32B (h 5120, 40/8 heads = G 5, qkv bias, I 27648) and
    Llama-3.1-70B (h 8192, 64/8 heads = G 8, I 28672) layers, truncated in depth and vocabulary so that the
    CPU oracle finishes in seconds: decode rows and a prefill chunk against the oracle run live."""
    cfg = O.truncated(O.CONFIGS[name], layers, vocab=vocab)
    w = O.make_weights(cfg, seed=11, norm_jitter=0.05)
    r = make_runner(cfg, w, max_tokens=32, max_model_len=256, n_blocks=4)
    ids = O.make_prompt(cfg, 0, 12)
    om = O.OracleModel(cfg, w, capacity=32)
    want = om.forward(om.new_seq(), ids).float()
    assert_logits_close(teacher_forced_logits(r, ids, chunk=1), want, softmax_tol=2e-3)
    assert_logits_close(teacher_forced_logits(r, ids, chunk=12), want, softmax_tol=2e-3)
    r.close()


def test_step_argument_validation():
    cfg = O.CONFIGS["tiny"]
    r = make_runner(cfg, O.make_weights(cfg), max_tokens=8)
    abi = pkg("_abi")
    z = torch.zeros(16, dtype=torch.int32, device="cuda")
    with pytest.raises(abi.B200Error, match="n_tokens"):
        r.step_device(z[:9], z[:9], z[:9], z[:1].view(1, 1), z[:9] + 1, 1)
    with pytest.raises(abi.B200Error, match="max_ctx_len"):
        r.step_device(z[:1], z[:1], z[:1], z[:1].view(1, 1), z[:1] + 1, 10 ** 6)
    r.close()


def test_openai_server_end_to_end_on_the_gpu():
    """The chart-facing surface over the real runner: POST /v1/completions (temperature 0) returns the
    engine's greedy tokens; /health and /metrics respond."""
    from fastapi.testclient import TestClient
    S, E = pkg("server"), pkg("engine")
    cfg = O.CONFIGS["tiny"]
    w = O.make_weights(cfg, norm_jitter=0.1)
    r = make_runner(cfg, w)
    eng = E.LLMEngine(r, max_num_batched_tokens=64, max_num_seqs=8, max_model_len=1024)
    tok = S.ByteTokenizer(cfg.vocab)
    app = S.create_app(eng, tok, "tiny", 1024)
    prompt = "What is Deep Learning?"
    ids = tok.encode(prompt)
    want, logits = O.OracleModel(cfg, w, capacity=128).generate(ids, 16, keep_logits=True)
    with TestClient(app) as c:
        assert c.get("/health").status_code == 200
        out = c.post("/v1/completions", json={"model": "tiny", "prompt": ids, "max_tokens": 16, "temperature": 0,
                                              "ignore_eos": True}).json()
        assert out["usage"]["completion_tokens"] == 16
        # several concurrent requests exercise continuous batching through HTTP
        import concurrent.futures as cf
        with cf.ThreadPoolExecutor(4) as ex:
            res = list(ex.map(lambda i: c.post("/v1/completions", json={"model": "tiny", "prompt": ids, "max_tokens": 8,
                                                                         "temperature": 0, "ignore_eos": True}).json(),
                           range(4)))
        assert all(x["choices"][0]["text"] == res[0]["choices"][0]["text"] for x in res)
        assert "vllm:generation_tokens_total" in c.get("/metrics").text
    got_text = out["choices"][0]["text"]
    # compare token-wise up to the first near-tie
    n_ok = 0
    for i, t in enumerate(want):
        if tok.decode(want[: i + 1]) != got_text[: len(tok.decode(want[: i + 1]))]:
            assert float(O.top2_margin(logits[i])) < MARGIN
            break
        n_ok += 1
    assert n_ok >= 1
    r.close()


def test_server_boots_from_a_checkpoint_directory_on_the_gpu(tmp_path, monkeypatch):
    """(f4) `--model <hf id>` end to end on the device: snapshot resolved under HF_HOME, sharded safetensors loaded and
    fused, config.json's llama3 rope_scaling (factor 32, as Llama-3.2 ships) honoured, HF tokenizer + chat template; the
    greedy tokens of /v1/chat/completions equal the oracle's on the same checkpoint (margin-aware)."""
    from fastapi.testclient import TestClient
    from ckpt_util import MODEL_ID, write_checkpoint
    S = pkg("server")
    snap, ocfg, w = write_checkpoint(str(tmp_path))
    monkeypatch.setenv("HF_HOME", str(tmp_path))
    args = S.make_arg_parser().parse_args(["--model", MODEL_ID, "--max-model-len", "512", "--max-num-batched-tokens", "64",
                                           "--max-num-seqs", "4", "--block-size", "128", "--kv-cache-gib", "0.05"])
    engine, tok, workers = S.build_engine(args)
    assert engine.runner.cfg.rope_factor == 32.0
    app = S.create_app(engine, tok, MODEL_ID, args.max_model_len, default_sampling=S.load_default_sampling(snap))
    msgs = [{"role": "user", "content": "what is deep learning ? tell me about tensor cores and memory bandwidth please"}]
    prompt_ids = tok.encode(tok.apply_chat_template(msgs, add_generation_prompt=True, tokenize=False), add_special_tokens=False)
    n_new = 24
    want, logits = O.OracleModel(ocfg, w, capacity=128).generate(prompt_ids, n_new, keep_logits=True)
    with TestClient(app) as c:
        r = c.post("/v1/chat/completions", json={"model": MODEL_ID, "messages": msgs, "max_tokens": n_new, "temperature": 0,
                                                 "ignore_eos": True, "logprobs": True, "top_logprobs": 1})
        assert r.status_code == 200, r.text
        out = r.json()
    assert out["usage"]["prompt_tokens"] == len(prompt_ids) and out["usage"]["completion_tokens"] == n_new
    got = [tok.convert_tokens_to_ids(e["token"]) for e in out["choices"][0]["logprobs"]["content"]]
    for i, (a, b) in enumerate(zip(got, want)):
        if a != b:
            assert float(O.top2_margin(logits[i])) < MARGIN, f"token {i} differs from the oracle outside a near-tie"
            break
    engine.runner.close()


def test_engine_penalties_and_logit_bias_vs_oracle(golden_dir):
    """Greedy requests with logit_bias / repetition / frequency / presence penalties through the engine: every emitted token
    is the argmax of the oracle's logits (teacher-forced on the engine's own tokens) after oracle.adjust_logits — vLLM's
    own arithmetic, tests/golden/penalties.npz — rounded to bf16 as the device does, wherever that argmax is not a
    near-tie; a +100 bias forces its token; an untouched request in the same batch keeps the plain greedy tokens."""
    g = np.load(f"{golden_dir}/tiny.npz")
    cfg = O.CONFIGS["tiny"]
    w = O.make_weights(cfg, seed=int(g["seed"]), norm_jitter=float(g["norm_jitter"]))
    r = make_runner(cfg, w)
    E = pkg("engine")
    prompt = g["prompt"].tolist()
    n_new = 24
    specs = [dict(repetition_penalty=1.3, frequency_penalty=0.4, presence_penalty=0.2, logit_bias={11: 4.0, 500: -3.0}),
             dict(), dict(logit_bias={77: 100.0}), dict(frequency_penalty=1.5)]
    eng = E.LLMEngine(r, max_num_batched_tokens=64, max_num_seqs=8, max_model_len=1024)
    reqs = [E.Request(f"p{i}", list(prompt), max_tokens=n_new, ignore_eos=True, **kw) for i, kw in enumerate(specs)]
    for q in reqs:
        eng.add_request(q)
    while eng.has_work():
        eng.step()
    assert reqs[1].output_ids[:8] == g["tokens"].tolist()[:8]
    assert reqs[2].output_ids == [77] * n_new
    om = O.OracleModel(cfg, w, capacity=256)
    checked = 0
    for q, kw in zip(reqs, specs):
        if not kw:
            continue
        logits = om.forward(om.new_seq(), prompt + q.output_ids[:-1])[len(prompt) - 1:]
        for i, tok in enumerate(q.output_ids):
            x = O.adjust_logits(logits[i], prompt, q.output_ids[:i], kw.get("repetition_penalty", 1.0), kw.get("frequency_penalty", 0.0),
                                kw.get("presence_penalty", 0.0), kw.get("logit_bias")).to(torch.bfloat16).float()
            if int(x.argmax()) != tok:
                assert float(O.top2_margin(x)) < MARGIN, f"request {q.request_id} token {i}: not the argmax of the adjusted logits"
            checked += 1
    assert checked == 3 * n_new
    # the frequency penalty changes what plain greedy would have produced (it repeats tokens on this fixture)
    assert reqs[3].output_ids != reqs[1].output_ids
    assert len(eng.blocks.free) == r.n_blocks
    r.close()
