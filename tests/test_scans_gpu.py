"""The recurrences' kernels at the edges of their stages and chunks, against the same recurrence row by row in float64."""
import pytest
import torch

from conftest import pkg

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _i32(x):
    return torch.tensor(x, dtype=torch.int32, device=DEV)


def _mlstm(x, gates, state, heads, dim, vdim):
    """Rows x [n][2 hd + hv], log gates, state (S [heads][vdim][dim], n [heads][dim], m [heads]) -> outputs, what one relative
    error of all terms of a sum can do to them, new state; float64."""
    S, nn, m = (t.clone() for t in state)
    hd, out, span = heads * dim, [], []
    for t in range(x.shape[0]):
        q = x[t, :hd].reshape(heads, dim) * dim ** -0.5
        k, v = x[t, hd:2 * hd].reshape(heads, dim), x[t, 2 * hd:2 * hd + heads * vdim].reshape(heads, vdim)
        i, f = gates[t, :heads], gates[t, heads:]
        mn = torch.maximum(f + m, i)
        a, b, m = torch.exp(f + m - mn), torch.exp(i - mn), mn
        S = a[:, None, None] * S + v[:, :, None] * (b[:, None] * k)[:, None, :]
        nn = a[:, None] * nn + b[:, None] * k
        den = torch.maximum((nn * q).sum(-1).abs(), torch.exp(-m)) + 1e-6
        o = (S @ q[:, :, None])[..., 0] / den[:, None]
        out.append(o.reshape(-1))
        span.append(((S.abs() @ q.abs()[:, :, None])[..., 0] / den[:, None] + o.abs() * ((nn * q).abs().sum(-1) / den)[:, None]).reshape(-1))
    return torch.stack(out), torch.stack(span), (S, nn, m)


# portions of two sequences, several steps: one row, less than a stage of 16, the border between the walk and the chunks (96 rows), whole and
# ragged chunks; both slots start dirty
STEPS = [([3], [70]), ([1], [64]), ([15, 66], [1, 2]), ([130], [16]), ([97], [256]), ([96], [193])]


@pytest.mark.parametrize("f32,heads,dim,vdim,pad", [(0, 2, 128, 64, 0), (0, 3, 64, 40, 0), (0, 1, 40, 24, 0), (0, 2, 16, 8, 8), (0, 2, 36, 20, 0),
                                                    (0, 1, 128, 48, 4), (0, 1, 200, 32, 0), (1, 2, 128, 32, 0), (1, 1, 50, 7, 0)])
def test_mlstm_scan_portions_and_hard_gates(f32, heads, dim, vdim, pad):
    """pad: columns of other data behind a row (4: rows that do not start at 16-byte addresses)."""
    lib, check = pkg("_abi").lib(), pkg("_abi").check
    g = torch.Generator().manual_seed(dim * 10 + vdim)
    adt = torch.float32 if f32 else torch.bfloat16
    hd, hv, nz = heads * dim, heads * vdim, (vdim + 31) // 32
    floats, ld = int(lib.b200_mlstm_state_floats(heads, dim, vdim)), 2 * hd + hv + pad
    assert floats == heads * vdim * dim + heads * nz * dim + heads * nz
    stride = floats + 6
    state = torch.full((4, stride), 7.5, device=DEV)                      # whatever a slot held: a sequence at position 0 starts from zeros
    slots, pos = [2, 0], [0, 0]
    oracle = [tuple(torch.zeros(s, dtype=torch.float64) for s in ((heads, vdim, dim), (heads, dim), (heads,))) for _ in range(2)]
    for a, b in STEPS:
        for cuts in (list(zip(a, b)) if len(a) == len(b) else [(a[0], b[0])]):
            T = sum(cuts)
            x = torch.randn(T, ld, generator=g).to(adt)
            gates = torch.randn(T, 2 * heads, generator=g) * 2
            gates[:, heads:] = torch.nn.functional.logsigmoid(gates[:, heads:] + 3)
            if T > 20:
                gates[11, heads:] = -14.9      # all but forgotten
                gates[17, :heads] = 14.0       # a row that dwarfs what is there
                gates[18:, :heads] -= 6.0
            start = [0, cuts[0], T]
            out = torch.full((T, hv), float("nan"), device=DEV)
            xd, gd = x.to(DEV), gates.to(DEV)
            p = list(range(pos[0], pos[0] + cuts[0])) + list(range(pos[1], pos[1] + cuts[1]))
            ptd, std, sld = _i32(p), _i32(start), _i32(slots)
            check(lib.b200_mlstm_scan(f32, xd.data_ptr(), ld, 0, hd, 2 * hd, gd.data_ptr(), ptd.data_ptr(), std.data_ptr(), sld.data_ptr(),
                                      state.data_ptr(), stride, out.data_ptr(), 2, heads, dim, vdim, None))
            torch.cuda.synchronize()
            for s in range(2):
                lo, hi = start[s], start[s + 1]
                want, span, oracle[s] = _mlstm(x[lo:hi].double(), gates[lo:hi].double(), oracle[s], heads, dim, vdim)
                got = out[lo:hi].double().cpu()
                # f + m - m' of a row is rounded twice in fp32 at |f| + |m| < 32 (2^-20 each): 2e-6 of a weight a row of the walk, a few rows' worth
                # lives on (the chunks take these sums in 64 bits, but start from what the walk left).  The division magnifies what happens to a
                # small |n . q|, so the results are held to what such an error of every term could do to them
                tol = 1e-5
                assert ((got - want).abs() <= tol * span + 1e-7 * want.abs()).all(), (cuts, s, float(((got - want).abs() / span).max()))
                st = state[slots[s]].double().cpu()
                S = st[:heads * vdim * dim].reshape(heads, vdim, dim)
                n = st[heads * vdim * dim:heads * vdim * dim + heads * nz * dim].reshape(heads, nz, dim)
                m = st[heads * vdim * dim + heads * nz * dim:floats].reshape(heads, nz)
                for z in range(nz):
                    assert (n[:, z] - oracle[s][1]).norm() < tol * oracle[s][1].norm() and (m[:, z] - oracle[s][2]).abs().max() < 1e-5
                assert (S - oracle[s][0]).norm() < tol * oracle[s][0].norm()
                assert (st[floats:] == 7.5).all()
                pos[s] += cuts[s]
    assert (state[[1, 3]] == 7.5).all()


@pytest.mark.parametrize("what", ["value", "key", "forget gate", "input gate"])
@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
@pytest.mark.parametrize("row", [0, 37, 100])
def test_mlstm_chunks_are_causal_for_what_is_not_finite(what, bad, row, T=130, heads=2):
    """An infinity or NaN of one row reaches that row and the later ones (a value's its own column, anything else's its head), and no earlier row."""
    if what in ("forget gate", "input gate") and bad == float("inf"):   # ("gate of +inf" below: an input gate)
        bad = float("nan")
    lib, check = pkg("_abi").lib(), pkg("_abi").check
    dim, vdim, col = 64, 64, 21
    g = torch.Generator().manual_seed(5)
    hd, hv = heads * dim, heads * vdim
    floats, ld = int(lib.b200_mlstm_state_floats(heads, dim, vdim)), 2 * hd + hv
    x = torch.randn(T, ld, generator=g).to(torch.bfloat16)
    gates = torch.randn(T, 2 * heads, generator=g)
    gates[:, heads:] = torch.nn.functional.logsigmoid(gates[:, heads:] + 3)
    zero = tuple(torch.zeros(s, dtype=torch.float64) for s in ((heads, vdim, dim), (heads, dim), (heads,)))
    want, span, (S, _, _) = _mlstm(x.double(), gates.double(), zero, heads, dim, vdim)
    hit = torch.zeros(T, heads, vdim, dtype=torch.bool)      # everything in head 1
    if what == "value":
        x[row, 2 * hd + vdim + col] = bad
        hit[row:, 1, col] = True
    else:
        hit[row:, 1] = True
        if what == "key":
            x[row, hd + dim + 9] = bad
        else:
            gates[row, (heads if what == "forget gate" else 0) + 1] = bad
    state, out = torch.zeros(1, floats, device=DEV), torch.full((T, hv), float("nan"), device=DEV)
    xd, gd, ptd, std, sld = x.to(DEV), gates.to(DEV), _i32(list(range(T))), _i32([0, T]), _i32([0])
    check(lib.b200_mlstm_scan(0, xd.data_ptr(), ld, 0, hd, 2 * hd, gd.data_ptr(), ptd.data_ptr(), std.data_ptr(), sld.data_ptr(), state.data_ptr(), floats,
                              out.data_ptr(), 1, heads, dim, vdim, None))
    torch.cuda.synchronize()
    got, hit = out.double().cpu(), hit.reshape(T, hv)
    assert not torch.isfinite(got[hit]).any()
    near = (got - want).abs() <= 1e-5 * span + 1e-7 * want.abs()   # (as above)
    assert near[~hit].all()
    st = state[0, :heads * vdim * dim].double().cpu().reshape(heads, vdim, dim)
    if what == "value":
        assert not torch.isfinite(st[1, col]).any() and torch.isfinite(st[1, :col]).all() and torch.isfinite(st[1, col + 1:]).all()
    else:
        assert not torch.isfinite(st[1, :, 9]).any()
    assert (st[0] - S[0]).norm() < 1e-5 * S[0].norm()


# Segments of a cluster: the border to the chunks (192 rows), two segments with one row in the second's last tile, both tiles of a segment (513 rows), whole
# rounds and one row more; then a step that starts from what the first one left.  vdim 96: a column block of 32, 40: of 40; `off` floats: outputs that
# do not start at 16-byte addresses.
@pytest.mark.parametrize("rows", [192, 193, 257, 513, 1024, 1025])
@pytest.mark.parametrize("heads,dim,vdim,off", [(2, 128, 64, 0), (1, 128, 96, 0), (1, 40, 40, 1), (2, 64, 64, 0)])
def test_mlstm_segments(rows, heads, dim, vdim, off):
    lib, check = pkg("_abi").lib(), pkg("_abi").check
    g = torch.Generator().manual_seed(rows + dim + vdim)
    hd, hv, nz = heads * dim, heads * vdim, (vdim + 31) // 32
    floats, ld = int(lib.b200_mlstm_state_floats(heads, dim, vdim)), 2 * hd + hv
    state = torch.full((2, floats), 7.5, device=DEV)
    oracle = tuple(torch.zeros(s, dtype=torch.float64) for s in ((heads, vdim, dim), (heads, dim), (heads,)))
    at = 0
    for T in (rows, 260):
        x = torch.randn(T, ld, generator=g).to(torch.bfloat16)
        gates = torch.randn(T, 2 * heads, generator=g) * 1.5
        gates[:, heads:] = torch.nn.functional.logsigmoid(gates[:, heads:] + 3)
        gates[T // 2, heads:] = -14.9      # all but forgotten
        gates[T // 2 + 9, :heads] = 9.0    # a row that dwarfs what is there
        buf = torch.full((T * hv + off,), float("nan"), device=DEV)
        out = buf[off:].view(T, hv)
        xd, gd, ptd, std, sld = x.to(DEV), gates.to(DEV), _i32(list(range(at, at + T))), _i32([0, T]), _i32([1])
        check(lib.b200_mlstm_scan(0, xd.data_ptr(), ld, 0, hd, 2 * hd, gd.data_ptr(), ptd.data_ptr(), std.data_ptr(), sld.data_ptr(), state.data_ptr(),
                                  floats, out.data_ptr(), 1, heads, dim, vdim, None))
        torch.cuda.synchronize()
        want, span, oracle = _mlstm(x.double(), gates.double(), oracle, heads, dim, vdim)
        got, tol = out.double().cpu(), 1e-5     # (as above)
        assert ((got - want).abs() <= tol * span + 1e-7 * want.abs()).all(), (T, float(((got - want).abs() / span).max()))
        st = state[1].double().cpu()
        assert (st[:hv * dim].reshape(heads, vdim, dim) - oracle[0]).norm() < tol * oracle[0].norm()
        n = st[hv * dim:hv * dim + heads * nz * dim].reshape(heads, nz, dim)
        assert (n - oracle[1][:, None]).norm() < tol * nz ** 0.5 * oracle[1].norm()
        assert (st[hv * dim + heads * nz * dim:].reshape(heads, nz) - oracle[2][:, None]).abs().max() < 1e-5
        at += T
    assert (state[0] == 7.5).all()


# Two row tiles a segment (513 rows: of 144), whole rounds and two of them, while another stream copies memory: a row that the products do not wait for
# would come late.  The same bits as alone, whose results the test above holds to the oracle.
@pytest.mark.parametrize("rows", [513, 1024, 2048])
@pytest.mark.parametrize("dim", [64, 128])
def test_mlstm_segments_beside_copies(rows, dim):
    lib, check = pkg("_abi").lib(), pkg("_abi").check
    heads, vdim = 8, 256
    g = torch.Generator(device=DEV).manual_seed(rows + dim)
    hd, hv = heads * dim, heads * vdim
    floats, ld = int(lib.b200_mlstm_state_floats(heads, dim, vdim)), 2 * hd + hv
    x, gates = torch.randn(rows, ld, generator=g, device=DEV).to(torch.bfloat16), torch.randn(rows, 2 * heads, generator=g, device=DEV)
    gates[:, heads:] = torch.nn.functional.logsigmoid(gates[:, heads:] + 3)
    state, out = torch.zeros(1, floats, device=DEV), torch.empty(rows, hv, device=DEV)
    ptd, std, sld = _i32(list(range(rows))), _i32([0, rows]), _i32([0])
    big, side, outs = torch.empty(2, 1 << 28, dtype=torch.uint8, device=DEV), torch.cuda.Stream(), []
    torch.cuda.synchronize()
    for run in range(40):
        if run:
            with torch.cuda.stream(side):
                big[1].copy_(big[0])
        check(lib.b200_mlstm_scan(0, x.data_ptr(), ld, 0, hd, 2 * hd, gates.data_ptr(), ptd.data_ptr(), std.data_ptr(), sld.data_ptr(), state.data_ptr(),
                                  floats, out.data_ptr(), 1, heads, dim, vdim, torch.cuda.current_stream().cuda_stream))
        outs.append((out.clone(), state.clone()))
    torch.cuda.synchronize()
    assert torch.isfinite(outs[0][0]).all() and all(torch.equal(a, b) for o in outs[1:] for a, b in zip(o, outs[0]))


@pytest.mark.parametrize("what", ["value", "key", "forget gate", "input gate"])
@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
@pytest.mark.parametrize("row", [0, 127, 200, 540])
def test_mlstm_segments_are_causal_for_what_is_not_finite(what, bad, row):
    """600 rows: segments of 160, with a second row tile; otherwise as the chunks' test."""
    test_mlstm_chunks_are_causal_for_what_is_not_finite(what, bad, row, T=600)


# An input gate of +inf makes a head's later rows NaN, as the recurrence has it (the running maximum is infinite); gates of -inf are rows without weight, also where a
# whole group of 32 rows, a segment's first rows or the sequence's have none: in chunks (130 rows), segments with one row tile and with two.
@pytest.mark.parametrize("T", [130, 300, 600])
def test_mlstm_infinite_input_gates(T):
    test_mlstm_chunks_are_causal_for_what_is_not_finite("gate of +inf", float("inf"), T // 2, T=T)
    lib, check = pkg("_abi").lib(), pkg("_abi").check
    heads, dim, vdim = 2, 64, 64
    g = torch.Generator().manual_seed(T)
    hd, hv = heads * dim, heads * vdim
    floats, ld = int(lib.b200_mlstm_state_floats(heads, dim, vdim)), 2 * hd + hv
    x, gates = torch.randn(T, ld, generator=g).to(torch.bfloat16), torch.randn(T, 2 * heads, generator=g)
    gates[:, heads:] = torch.nn.functional.logsigmoid(gates[:, heads:] + 3)
    for lo, hi in ((0, 3), (32, 64), (77, 78), (T - 40, T)) + (((150, 330),) if T > 400 else ()):
        gates[lo:hi, 1] = float("-inf")
    zero = tuple(torch.zeros(s, dtype=torch.float64) for s in ((heads, vdim, dim), (heads, dim), (heads,)))
    want, span, (S, _, m) = _mlstm(x.double(), gates.double(), zero, heads, dim, vdim)
    state, out = torch.zeros(1, floats, device=DEV), torch.full((T, hv), float("nan"), device=DEV)
    xd, gd, ptd, std, sld = x.to(DEV), gates.to(DEV), _i32(list(range(T))), _i32([0, T]), _i32([0])
    check(lib.b200_mlstm_scan(0, xd.data_ptr(), ld, 0, hd, 2 * hd, gd.data_ptr(), ptd.data_ptr(), std.data_ptr(), sld.data_ptr(), state.data_ptr(), floats,
                              out.data_ptr(), 1, heads, dim, vdim, None))
    torch.cuda.synchronize()
    assert ((out.double().cpu() - want).abs() <= 1e-5 * span + 1e-7 * want.abs()).all()     # (as above)
    st = state[0].double().cpu()
    assert (st[:hv * dim].reshape(heads, vdim, dim) - S).norm() < 1e-5 * S.norm() and (st[-heads * 2:].reshape(heads, 2) - m[:, None]).abs().max() < 1e-5


# The chunks' own kernel, which takes launches of more than 33 clusters of segments: one CTA an SM (36 heads) and two (70)
@pytest.mark.parametrize("what", ["value", "key", "forget gate", "input gate", "gate of +inf"])
@pytest.mark.parametrize("heads,T", [(36, 130), (70, 260)])
@pytest.mark.parametrize("row", [37, 100])
def test_mlstm_chunk_kernel_is_causal_for_what_is_not_finite(what, heads, T, row):
    test_mlstm_chunks_are_causal_for_what_is_not_finite(what, float("inf"), row, T=T, heads=heads)


# Steps whose CTAs outnumber the SMs: two sequences of 8 heads of 256 columns (256 CTAs, two to an SM, short portions walked beside the chunks),
# four (512 CTAs: chunks and walk in a launch each, whole portions on both sides of 97 rows), five (the walk alone); the second step
# starts from the state the first one left.
@pytest.mark.parametrize("dim", [64, 128])
@pytest.mark.parametrize("steps", [([130, 30], [20, 97]), ([97, 96, 5, 161], [64, 1, 100, 98]), ([30, 1, 17, 100, 2], [1, 1, 1, 1, 1])])
def test_mlstm_scan_of_many_ctas(dim, steps, heads=8, vdim=256):
    lib, check = pkg("_abi").lib(), pkg("_abi").check
    S = len(steps[0])
    g = torch.Generator().manual_seed(dim + S)
    hd, hv, nz = heads * dim, heads * vdim, (vdim + 31) // 32
    floats, ld = int(lib.b200_mlstm_state_floats(heads, dim, vdim)), 2 * hd + hv
    state = torch.full((S + 1, floats), 7.5, device=DEV)
    slots, pos = [S - s for s in range(S)], [0] * S
    oracle = [tuple(torch.zeros(s, dtype=torch.float64) for s in ((heads, vdim, dim), (heads, dim), (heads,))) for _ in range(S)]
    for cuts in steps:
        T = sum(cuts)
        x, gates = torch.randn(T, ld, generator=g).to(torch.bfloat16), torch.randn(T, 2 * heads, generator=g)
        gates[:, heads:] = torch.nn.functional.logsigmoid(gates[:, heads:] + 3)
        start = [0]
        for n in cuts:
            start.append(start[-1] + n)
        out = torch.full((T, hv), float("nan"), device=DEV)
        xd, gd = x.to(DEV), gates.to(DEV)
        ptd, std, sld = _i32([pos[s] + i for s in range(S) for i in range(cuts[s])]), _i32(start), _i32(slots)
        check(lib.b200_mlstm_scan(0, xd.data_ptr(), ld, 0, hd, 2 * hd, gd.data_ptr(), ptd.data_ptr(), std.data_ptr(), sld.data_ptr(), state.data_ptr(), floats,
                                  out.data_ptr(), S, heads, dim, vdim, None))
        torch.cuda.synchronize()
        for s in range(S):
            lo, hi = start[s], start[s + 1]
            want, span, oracle[s] = _mlstm(x[lo:hi].double(), gates[lo:hi].double(), oracle[s], heads, dim, vdim)
            got, tol = out[lo:hi].double().cpu(), 1e-5     # (as above)
            assert ((got - want).abs() <= tol * span + 1e-7 * want.abs()).all(), (cuts, s, float(((got - want).abs() / span).max()))
            st = state[slots[s]].double().cpu()
            assert (st[:hv * dim].reshape(heads, vdim, dim) - oracle[s][0]).norm() < tol * oracle[s][0].norm()
            n = st[hv * dim:hv * dim + heads * nz * dim].reshape(heads, nz, dim)
            assert (n - oracle[s][1][:, None]).norm() < tol * nz ** 0.5 * oracle[s][1].norm()
            assert (st[hv * dim + heads * nz * dim:].reshape(heads, nz) - oracle[s][2][:, None]).abs().max() < 1e-5
            pos[s] += cuts[s]
    assert (state[0] == 7.5).all()


# The chunks' own kernel over many chunks, which reuse its buffers, beside short portions: columns that leave a block ragged, one CTA an SM and two, and the walk in a
# launch of its own (four sequences of 40 heads)
@pytest.mark.parametrize("heads,dim,vdim,steps", [(20, 128, 72, [[300, 40], [5, 420]]), (36, 64, 64, [[420], [64], [230]]), (37, 40, 32, [[97], [300]]),
                                                  (40, 64, 72, [[97, 1, 200, 40], [30, 130, 1, 96]])])
def test_mlstm_chunk_kernel_over_many_chunks(heads, dim, vdim, steps):
    test_mlstm_scan_of_many_ctas(dim, steps, heads, vdim)


# channel decays / one per head, delta rule / plain, heads sharing keys, sizes that leave lanes and columns idle; strided decays (g_chan 2);
# zero decays forget everything, as do rows of zeros; rows that are not 16-byte aligned
@pytest.mark.parametrize("rule", ["channel", "head", "plain", "plain channel", "strided"])
@pytest.mark.parametrize("heads,kv,dim,vdim", [(2, 2, 128, 128), (4, 1, 64, 40), (3, 3, 50, 7), (2, 1, 160, 33)])
def test_linear_scans_portions(rule, heads, kv, dim, vdim):
    lib, check = pkg("_abi").lib(), pkg("_abi").check
    g = torch.Generator().manual_seed(dim + vdim)
    delta, chan = rule in ("channel", "head", "strided"), rule in ("channel", "plain channel", "strided")
    step = 2 if rule == "strided" else 1
    floats = heads * vdim * dim
    stride = floats + (4 if dim % 4 == 0 else 3)
    state = torch.full((4, stride), 7.5, device=DEV)
    slots, pos = [2, 0], [0, 0]
    oracle = [torch.zeros(heads, vdim, dim, dtype=torch.float64) for _ in range(2)]
    for cuts in [(3, 70), (1, 1), (2, 17), (16, 15), (33, 32)]:
        T = sum(cuts)
        q, k = (torch.nn.functional.normalize(torch.randn(T, kv, dim, generator=g), dim=-1) for _ in range(2))
        v, beta = torch.randn(T, heads, vdim, generator=g), torch.sigmoid(torch.randn(T, heads, generator=g))
        decay = torch.rand(T, heads, dim if chan else 1, generator=g) ** 0.1
        if T > 20:
            decay[7] = 0.0
            k[9] = 0.0
        wide = torch.zeros(T, heads, decay.shape[2] * step).reshape(T, heads, -1)
        wide[:, :, ::step] = decay
        t = [x.to(DEV).contiguous() for x in (q, k, v, beta, wide)]
        start = [0, cuts[0], T]
        p = list(range(pos[0], pos[0] + cuts[0])) + list(range(pos[1], pos[1] + cuts[1]))
        ptd, std, sld, out = _i32(p), _i32(start), _i32(slots), torch.full((T, heads * vdim), float("nan"), device=DEV)
        check(lib.b200_linear_scan(int(delta), *[x.data_ptr() for x in t], heads * wide.shape[2], wide.shape[2], step if chan else 0, ptd.data_ptr(),
                                   std.data_ptr(), sld.data_ptr(), state.data_ptr(), stride, out.data_ptr(), 2, heads, kv, dim, vdim, None))
        torch.cuda.synchronize()
        for s in range(2):
            S = oracle[s]
            for r in range(start[s], start[s + 1]):
                kk, qq = (x[r].double().repeat_interleave(heads // kv, 0) for x in (k, q))
                S = S * decay[r].double()[:, None, :]
                u = v[r].double() - ((S @ kk[:, :, None])[..., 0] if delta else 0.0)
                S = S + (beta[r].double()[:, None] * u)[:, :, None] * kk[:, None, :]
                want = (S @ qq[:, :, None])[..., 0].reshape(-1)
                # fp32 throughout: sums of up to 160 terms and the roundings of some tens of live rows, 2^-24 each
                assert (out[r].double().cpu() - want).norm() < 2e-6 * max(float(want.norm()), float(S.norm()) * 0.05), (cuts, s, r)
            oracle[s] = S
            st = state[slots[s]].double().cpu()
            assert (st[:floats].reshape(S.shape) - S).norm() < 2e-6 * S.norm() and (st[floats:] == 7.5).all()
            pos[s] += cuts[s]
    assert (state[[1, 3]] == 7.5).all()


def _delta(q, k, v, beta, decay, S):
    """Rows one by one in float64: [T][heads][vdim] and the state [heads][vdim][dim] after them."""
    y = torch.empty(v.shape, dtype=torch.float64, device=v.device)
    for r in range(len(v)):
        S = S * decay[r][:, None, :]
        u = v[r] - (S @ k[r][:, :, None])[..., 0]
        S = S + (beta[r][:, None] * u)[:, :, None] * k[r][:, None, :]
        y[r] = (S @ q[r][:, :, None])[..., 0]
    return y, S


# The delta rule in blocks of eight rows: one, two and three CTAs an SM, portions on both sides of the length from which it takes them (64; 128 with three
# CTAs an SM), blocks and rounds that are not full, clusters of one to four CTAs, half a warp's columns and channels missing; the second step starts from
# the state that the first one left.
@pytest.mark.parametrize("chan", [True, False])
@pytest.mark.parametrize("heads,kv,dim,vdim,steps", [
    (16, 16, 128, 128, [[300], [65]]), (2, 1, 128, 128, [[63], [64], [66], [72], [97]]), (3, 3, 100, 16, [[129], [80]]), (1, 1, 68, 40, [[200], [71]]),
    (16, 4, 128, 128, [[64, 90], [130, 7]]), (40, 8, 128, 48, [[70, 1], [67, 256]]),
    (16, 16, 128, 128, [[128, 127, 20], [1, 140, 161]]), (16, 16, 64, 128, [[128, 20, 200], [140, 129, 1]]), (8, 2, 64, 128, [[128], [145]]), (16, 4, 64, 128, [[160, 200], [5, 129]]), (4, 4, 36, 24, [[131], [250]]),
])
def test_delta_blocks(heads, kv, dim, vdim, steps, chan):
    lib, check = pkg("_abi").lib(), pkg("_abi").check
    g = torch.Generator(device=DEV).manual_seed(dim + vdim + heads)
    S, rnd = len(steps[0]), lambda *s: torch.randn(*s, generator=g, device=DEV)
    floats = heads * vdim * dim
    state = torch.full((S + 1, floats), 7.5, device=DEV)
    slots, pos = [S - s for s in range(S)], [0] * S
    oracle = [torch.zeros(heads, vdim, dim, dtype=torch.float64, device=DEV) for _ in range(S)]
    for cuts in steps:
        T = sum(cuts)
        q, k = (torch.nn.functional.normalize(rnd(T, kv, dim), dim=-1) for _ in range(2))
        v, beta = rnd(T, heads, vdim), torch.sigmoid(rnd(T, heads))
        decay = torch.rand(T, heads, dim if chan else 1, generator=g, device=DEV) ** 0.1
        decay[T // 2], k[T // 3], decay[T // 4, 0] = 0.0, 0.0, 1e-30
        start = [0]
        for n in cuts:
            start.append(start[-1] + n)
        out = torch.full((T, heads * vdim), float("nan"), device=DEV)
        ptd, std, sld = _i32([pos[s] + i for s in range(S) for i in range(cuts[s])]), _i32(start), _i32(slots)
        check(lib.b200_linear_scan(1, *[x.data_ptr() for x in (q, k, v, beta, decay)], heads * decay.shape[2], decay.shape[2], int(chan), ptd.data_ptr(),
                                   std.data_ptr(), sld.data_ptr(), state.data_ptr(), floats, out.data_ptr(), S, heads, kv, dim, vdim, None))
        torch.cuda.synchronize()
        wide = [x.double().repeat_interleave(heads // kv, 1) for x in (q, k)] + [x.double() for x in (v, beta, decay)]
        for s in range(S):
            lo, hi = start[s], start[s + 1]
            want, oracle[s] = _delta(*[x[lo:hi] for x in wide], oracle[s])
            # fp32 throughout, as above: 2^-24 for sums of up to 128 terms and the roundings of some tens of live rows
            err, size = (out[lo:hi].double().reshape(want.shape) - want).flatten(1).norm(dim=1), want.flatten(1).norm(dim=1)
            assert (err < 2e-6 * torch.maximum(size, 0.05 * oracle[s].norm())).all(), (cuts, s, float((err / size).max()))
            assert (state[slots[s]].double().reshape(oracle[s].shape) - oracle[s]).norm() < 2e-6 * oracle[s].norm()
            pos[s] += cuts[s]
    assert (state[0] == 7.5).all()


# Portions in the order of their length (equal ones, empty ones, the longest first and last), more CTAs than the device has places for, two and three of them
# an SM, keys of 64 on CTAs of one and three an SM, and more CTAs than go in blocks (walked); the bound is that of the test above.
@pytest.mark.parametrize("heads,kv,dim,vdim,steps", [
    (16, 16, 128, 128, [[70, 300, 1, 129], [129, 129, 64, 0]]), (16, 8, 128, 128, [[2, 200, 130, 128, 5, 31], [0, 64, 0, 90, 160, 64]]), (40, 40, 64, 128, [[5, 140, 131]]),
    (16, 4, 64, 128, [[130, 7, 1, 256, 130, 64], [5, 0, 129, 0, 128, 64]]), (8, 2, 64, 128, [[129, 260]]), (16, 16, 100, 48, [[128, 7, 300, 300, 66]]),
])
def test_delta_blocks_of_ordered_portions(heads, kv, dim, vdim, steps):
    test_delta_blocks(heads, kv, dim, vdim, steps, True)


@pytest.mark.parametrize("what", ["value", "key", "query", "decay", "beta"])
@pytest.mark.parametrize("bad", [float("inf"), float("nan")])
@pytest.mark.parametrize("row", [0, 37, 99])
def test_delta_blocks_are_causal_for_what_is_not_finite(what, bad, row):
    """A row's value that is not finite reaches its own column only, everything else the head's later rows only; a query its own row."""
    lib, check = pkg("_abi").lib(), pkg("_abi").check
    g = torch.Generator(device=DEV).manual_seed(row)
    T, heads, dim, vdim, rnd = 100, 2, 128, 32, lambda *s: torch.randn(*s, generator=g, device=DEV)
    q, k = (torch.nn.functional.normalize(rnd(T, heads, dim), dim=-1) for _ in range(2))
    v, beta, decay = rnd(T, heads, vdim), torch.sigmoid(rnd(T, heads)), torch.rand(T, heads, dim, generator=g, device=DEV) ** 0.1
    outs = []
    for clean in (True, False):
        if not clean:
            {"value": v, "key": k, "query": q, "decay": decay, "beta": beta[:, :, None]}[what][row, 1, -1] = bad
        state, out = torch.zeros(1, heads * vdim * dim, device=DEV), torch.empty(T, heads, vdim, device=DEV)
        pos, start, slot = _i32(list(range(T))), _i32([0, T]), _i32([0])
        check(lib.b200_linear_scan(1, *[x.data_ptr() for x in (q, k, v, beta, decay)], heads * dim, dim, 1, pos.data_ptr(), start.data_ptr(), slot.data_ptr(),
                                   state.data_ptr(), state.shape[1], out.data_ptr(), 1, heads, heads, dim, vdim, None))
        torch.cuda.synchronize()
        outs.append(out.cpu())
    a, b = outs
    same = torch.ones(T, heads, vdim, dtype=torch.bool)
    same[row:row + 1 if what == "query" else T, 1, -1 if what == "value" else 0:] = False
    assert torch.equal(a[same], b[same]) and not torch.isfinite(b[row, 1, -1])
