"""The tcgen05 linear on pairs of SMs (more than 128 tokens): edges of token tiles, slabs, k blocks and shares of k."""
import importlib

import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


@pytest.fixture(scope="module")
def abi():
    return importlib.import_module("enterprise-inference_b200._abi")


def _operands(T, n_out, k, ldx):
    g = torch.Generator(device="cuda").manual_seed(T * 7 + n_out + k)
    x = torch.randn(T, ldx, generator=g, device="cuda").to(BF)
    w = (0.05 * torch.randn(n_out, k, generator=g, device="cuda")).to(BF)
    return g, x, w


def _bound(x, w, y):
    """Half a unit of bf16 (8 bits), and k additions of fp32 products (24 bits; the tensor core may truncate: one unit each)."""
    return y.abs() * 2.0 ** -8 + x.shape[1] * 2.0 ** -23 * (x.abs() @ w.abs().T)


@pytest.mark.parametrize("T,n_out,k,pad", [
    (129, 8, 8, 0),             # one slab, one k block, both mostly empty
    (129, 264, 72, 8),          # a slab of 8 rows, the last k block of 8; rows of x and y with a gap
    (160, 384, 256, 0),         # an odd number of slabs: a pair's second CTA has none
    (255, 1000, 4096, 0),       # k shared by clusters
    (257, 256, 4160, 0),        # uneven shares of 65 k blocks
    (300, 2048, 2048, 0), (200, 4096, 1536, 0), (256, 6144, 1024, 16),
    (513, 2048, 1000, 0),
    (2048, 4096, 256, 0),       # two tiles a pair
    (5000, 1024, 128, 0),       # token tiles in groups of unequal size, several tiles a pair
])
def test_linear_pairs_of_sms(abi, T, n_out, k, pad):
    lib, P = abi.lib(), abi.ptr
    g, x, w = _operands(T, n_out, k, k + pad)
    b = torch.randn(n_out, generator=g, device="cuda").to(BF)
    wsb = int(lib.b200_linear_workspace_bytes(T, n_out, k))
    ws = torch.zeros(wsb, dtype=torch.uint8, device="cuda")
    xd, wd = x[:, :k].double(), w.double()
    want = xd @ wd.T + b.double()
    for bias in (b, None):
        y = torch.full((T, n_out + pad), float("nan"), dtype=BF, device="cuda")
        abi.check(lib.b200_linear_bf16(P(x), k + pad, P(w), P(bias) if bias is not None else None, P(y), n_out + pad, T, n_out, k, 0, P(ws), wsb, None))
        torch.cuda.synchronize()
        ref = want if bias is not None else want - b.double()
        assert (y[:, :n_out].double() - ref).abs().le(_bound(xd, wd, ref)).all()
        assert torch.isnan(y[:, n_out:].float()).all(), "columns beyond the output were written"


@pytest.mark.parametrize("T,I,k", [(129, 192, 512), (300, 64, 4096), (700, 1600, 256)])
def test_gate_up_epilogue_on_pairs_of_sms(abi, T, I, k):
    """SiLU * mul over interleaved slabs, odd numbers of them included, equals the plain linear and b200_silu_mul bit for bit."""
    lib, P = abi.lib(), abi.ptr
    _, x, w = _operands(T, 2 * I, k, k)
    il = torch.stack([w[:I].reshape(-1, 64, k), w[I:].reshape(-1, 64, k)], 1).reshape(2 * I, k).contiguous()
    wsb = int(lib.b200_linear_workspace_bytes(T, 2 * I, k))
    ws = torch.zeros(wsb, dtype=torch.uint8, device="cuda")
    gu, ref = torch.empty(T, 2 * I, dtype=BF, device="cuda"), torch.empty(T, I, dtype=BF, device="cuda")
    got = torch.full((T + 1, I), float("nan"), dtype=BF, device="cuda")
    abi.check(lib.b200_linear_bf16(P(x), k, P(w), None, P(gu), 2 * I, T, 2 * I, k, 0, P(ws), wsb, None))
    abi.check(lib.b200_silu_mul(P(gu), P(ref), T, I, None))
    abi.check(lib.b200_linear_fused_bf16(P(x), k, P(il), None, P(got), I, T, 2 * I, k, 1, None, None, None, None, None, 0, 0, 0, P(ws), wsb, None))
    torch.cuda.synchronize()
    assert torch.equal(got[:T], ref) and torch.isnan(got[T].float()).all()


@pytest.mark.parametrize("width,ff,experts,top,rows,gated,weight_input", [
    (64, 64, 2, 1, 130, True, 0),        # one slab of 64 gate and up rows a pair; runs of whole and part units
    (264, 192, 5, 2, 400, True, 0),      # odd numbers of slabs, the last k block of 8, an expert without rows
    (512, 96, 3, 3, 300, True, 0),       # ff not a multiple of 64: gate|up, then the activation on its own
    (256, 320, 4, 2, 515, False, 0),     # one projection, activated in the epilogue
    (256, 128, 6, 2, 900, False, 1),     # the mixing weight belongs to the input
    (128, 128, 1, 1, 1025, True, 0),     # one expert, five tiles
])
def test_experts_on_pairs_of_sms(abi, width, ff, experts, top, rows, gated, weight_input):
    """Routed experts with uneven runs (more than 64 rows in the mean): every (token, slot) row against fp64 from the same bf16 operands.

    The bound: bf16 roundings of gate, up, their activations and product (half a unit, 2^-9, each; silu takes up to twice a gate's for
    |gate| < 3, relu2 twice), i.e. less than 8 of them on every term of the closing sum."""
    lib, P = abi.lib(), abi.ptr
    g = torch.Generator(device="cuda").manual_seed(width + ff + rows)
    x = torch.randn(rows, width, generator=g, device="cuda").to(BF)
    wu = (0.5 * width ** -0.5 * torch.randn(experts, (2 if gated else 1) * ff, width, generator=g, device="cuda")).to(BF)
    wd = (0.05 * torch.randn(experts, width, ff, generator=g, device="cuda")).to(BF)
    p = torch.arange(1, experts + 1, device="cuda", dtype=torch.float32) ** 2   # uneven loads; expert 1 of many is left out
    if experts > top + 1:
        p[1] = 0
    ids = torch.multinomial(p.expand(rows, experts), top, generator=g).to(torch.int32)
    wts = torch.rand(rows, top, generator=g, device="cuda")
    parts = torch.full((rows, top, width), float("nan"), device="cuda")
    ws = torch.zeros(int(lib.b200_moe_workspace_bytes(rows, top, experts, width, ff)), dtype=torch.uint8, device="cuda")
    if gated:
        abi.check(lib.b200_moe_experts(0, P(x), P(wu), P(wd), P(ids), P(wts), rows, width, ff, experts, top, P(parts), P(ws), None))
    else:
        abi.check(lib.b200_moe_experts_form(0, P(x), P(wu), P(wd), P(ids), P(wts), rows, width, ff, experts, top, P(parts), P(ws), 0, abi.ACT_RELU2,
                                            weight_input, None))
    torch.cuda.synchronize()
    for e in range(experts):
        t, j = (ids == e).nonzero(as_tuple=True)
        xe, w = x[t].double(), wts[t, j, None].double()
        if weight_input:
            xe, w = (xe.float() * wts[t, j, None]).to(BF).double(), torch.ones_like(w)
        u = xe @ wu[e].double().T
        a = torch.nn.functional.silu(u[:, :ff]) * u[:, ff:] if gated else torch.relu(u) ** 2
        want, room = (a @ wd[e].double().T) * w, (a.abs() @ wd[e].abs().double().T) * w * 2.0 ** -6
        assert (parts[t, j].double() - want).abs().le(room + 1e-6).all(), e


# Narrow outputs over deep rows of more than 128 tokens (eight shares of k in tiles of 128 x 128) and their neighbours on pairs of SMs: up to 18 tiles and more,
# 64 k blocks and fewer, uneven shares, part tiles of either side.
@pytest.mark.parametrize("T,n_out,k", [(129, 8, 4096), (300, 200, 4160), (1024, 264, 4104), (2304, 128, 4096), (2305, 128, 4096), (129, 1152, 4096), (129, 1153, 4096),
                                       (200, 512, 4032), (257, 1280, 4160), (255, 2312, 4096), (160, 1024, 14336)])
def test_narrow_outputs_over_deep_rows(abi, T, n_out, k):
    test_linear_pairs_of_sms(abi, T, n_out, k, 8)


@pytest.mark.parametrize("T,I,k", [(160, 128, 4096), (700, 64, 4096)])
def test_gate_up_epilogue_of_narrow_outputs(abi, T, I, k):
    test_gate_up_epilogue_on_pairs_of_sms(abi, T, I, k)


@pytest.mark.parametrize("T,hq,hkv,k,bias", [(200, 2, 1, 4096, True), (700, 1, 1, 4160, False)])
def test_rope_kv_epilogue_of_narrow_outputs(abi, T, hq, hkv, k, bias):
    importlib.import_module("test_kernels_gpu").test_linear_fused_rope_kv_is_bit_identical_to_unfused(abi.lib(), abi, T, hq, hkv, k, bias)


# Plain outputs written in rows of 16-byte pieces, several tiles a pair: slabs that are whole and one that is not, tiles of an odd number of 32-token pieces, short k;
# and the same where the rows of y are no such pieces (four features at a time), bit for bit.
@pytest.mark.parametrize("T,n_out,k", [(6000, 1160, 128), (4097, 2048, 64), (2000, 4104, 64), (1300, 8192, 72), (161, 9000, 256), (700, 520, 512)])
def test_whole_slabs_and_odd_rows_of_outputs(abi, T, n_out, k):
    lib, P = abi.lib(), abi.ptr
    g, x, w = _operands(T, n_out, k, k)
    b = torch.randn(n_out, generator=g, device="cuda").to(BF)
    wsb = int(lib.b200_linear_workspace_bytes(T, n_out, k))
    ws, want, ys = torch.zeros(wsb, dtype=torch.uint8, device="cuda"), x.double() @ w.double().T + b.double(), []
    for ldy, off in ((n_out + 8, 0), (n_out + 3, 0), (n_out + 8, 4)):
        y = torch.full((T * ldy + 8,), float("nan"), dtype=BF, device="cuda")
        abi.check(lib.b200_linear_bf16(P(x), k, P(w), P(b), P(y[off:]), ldy, T, n_out, k, 0, P(ws), wsb, None))
        torch.cuda.synchronize()
        rows = y[off:off + T * ldy].reshape(T, ldy)
        assert torch.isnan(rows[:, n_out:].float()).all()
        ys.append(rows[:, :n_out])
    assert (ys[0].double() - want).abs().le(_bound(x.double(), w.double(), want)).all()
    assert torch.equal(ys[0], ys[1]) and torch.equal(ys[0], ys[2])
