"""Launches: which carry the programmatic attribute, read from the edges of a captured call; what a wait that ran out leaves behind."""
import threading

import pytest
import torch

from conftest import pkg

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _latent_call():
    """One call of an entry point that launches two kernels (run plan, attention)."""
    lib, check = pkg("_abi").lib(), pkg("_abi").check
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)   # noqa: E731
    q, kc = torch.randn(2, 4, 80, device=DEV), torch.randn(2, 1, 64, 80, device=DEV).to(torch.bfloat16)
    bt, sq, cx, out = i32([[0], [1]]), i32([0, 1]), i32([5, 60]), torch.empty(2, 4, 64, dtype=torch.bfloat16, device=DEV)
    ws = torch.zeros(int(lib.b200_paged_attn_anydim_workspace_bytes(2)), dtype=torch.uint8, device=DEV)
    keep = (q, kc, bt, sq, cx, out, ws)
    return keep, lambda s: check(lib.b200_latent_attn(q.data_ptr(), kc.data_ptr(), bt.data_ptr(), 1, sq.data_ptr(), cx.data_ptr(), out.data_ptr(), 2, 4,
                                                      80, 64, 64, 0.1, None, ws.data_ptr(), 1, None, s))


def _overlaps(switch):
    """That call captured in a thread of its own (the switch is the thread's): is the edge between its kernels a programmatic one?"""
    from cuda.bindings import runtime as rt
    keep, call = _latent_call()
    call(None)
    torch.cuda.synchronize()
    found, stream = [], torch.cuda.Stream()

    def work():
        if switch is not None:
            pkg("_abi").check(pkg("_abi").lib().b200_set_launch_pdl(switch))
        ok = lambda r: r[1:] if r[0] == rt.cudaError_t.cudaSuccess else pytest.fail(str(r[0]))   # noqa: E731
        ok(rt.cudaStreamBeginCapture(stream.cuda_stream, rt.cudaStreamCaptureMode.cudaStreamCaptureModeThreadLocal))
        call(stream.cuda_stream)
        g, = ok(rt.cudaStreamEndCapture(stream.cuda_stream))
        err = rt.cudaGraphGetEdges(g, 4)[0]      # (the query without edge data refuses edges that are not plain)
        found.append({rt.cudaError_t.cudaSuccess: False, rt.cudaError_t.cudaErrorLossyQuery: True}.get(err, err))
        ok(rt.cudaGraphDestroy(g))

    t = threading.Thread(target=work)
    t.start()
    t.join()
    assert found, "the capture failed"
    return found[0]


def test_the_launch_switch_reaches_the_kernels_of_one_call(monkeypatch):
    monkeypatch.delenv("B200_PDL", raising=False)
    assert _overlaps(None) is True     # the attention overlaps its plan
    assert _overlaps(1) is True
    assert _overlaps(0) is False
    monkeypatch.setenv("B200_PDL", "0")
    assert _overlaps(None) is False


def test_a_wait_that_runs_out_is_reported_once_by_the_next_call():
    """A small kernel gives up a wait at a barrier that nothing arrives at and ends: the context stays usable, the next call says so."""
    lib = pkg("_abi").lib()
    keep, call = _latent_call()
    call(None)
    torch.cuda.synchronize()
    want = keep[5].clone()
    assert lib.b200_debug_expired_wait(100, None) == 0
    torch.cuda.synchronize()
    with pytest.raises(Exception, match="ran out"):
        call(None)
    call(None)
    torch.cuda.synchronize()
    assert torch.equal(keep[5], want)
