"""What the operators on few rows hand to their kernels: the launch is caught and the addresses are read back on the host."""
import ctypes as C

import pytest
import torch

from socket_b200 import _lib, few_rows


def _read(address, ld, rows, n):
    """rows x n bf16 as a kernel given (address, ld) reads them."""
    raw = torch.tensor([[C.c_uint16.from_address(address + 2 * (r * ld + i)).value for i in range(n)] for r in range(rows)])
    return raw.to(torch.int32).to(torch.int16).view(torch.bfloat16)


@pytest.fixture
def caught(monkeypatch):
    """Every launch of the module, by name: what `read` makes of the parameters while the call is still running."""
    seen, read = [], {}

    def launch(library, name, *args):
        seen.append(read[name](*args))

    def params(x, w, chained, library="blocks"):
        p = _lib.LinearParams()
        p.rows, p.k = x.shape
        return p

    monkeypatch.setattr(few_rows, "_launch", launch)
    monkeypatch.setattr(few_rows, "_linear_params", params)
    monkeypatch.setattr(few_rows, "_require_cuda", lambda *tensors: None)
    monkeypatch.setattr(few_rows, "stream_ptr", lambda device=None: 0)
    return seen, read


@pytest.mark.parametrize("rows", [1, 2, 8])
@pytest.mark.parametrize("layout", ["dense", "strided", "broadcast", "turned"])
def test_residual_rows(caught, rows, layout):
    seen, read = caught
    n, k = 24, 16
    x, w = torch.randn(rows, k).bfloat16(), torch.randn(n, k).bfloat16()
    big = torch.randn(9, n + 8).bfloat16()                        # what lies behind a broadcast row belongs to this buffer too
    res = {"dense": torch.randn(rows, n).bfloat16(), "strided": big[:rows, :n], "broadcast": big[:1, 8:].expand(rows, n),
           "turned": torch.randn(n, rows).bfloat16().t()}[layout]
    read["linear_rows"] = lambda p, stream: _read(p._obj.res, p._obj.res_ld, rows, n)
    few_rows.linear(x, w, res=res)
    assert torch.equal(seen[0], res)


@pytest.mark.parametrize("rows", [1, 2, 8, 9])
@pytest.mark.parametrize("layout", ["dense", "strided", "broadcast", "turned"])
def test_logit_rows(caught, rows, layout):
    seen, read = caught
    n = 24
    big = torch.randn(10, n + 8).bfloat16()
    logits = {"dense": torch.randn(rows, n).bfloat16(), "strided": big[:rows, :n], "broadcast": big[:1, 8:].expand(rows, n),
              "turned": torch.randn(n, rows).bfloat16().t()}[layout]
    read["pick_token"] = lambda address, dtype, ld, batch, vocab, *rest: _read(address, ld, batch, vocab)
    few_rows.pick_token(logits, torch.zeros(rows, 1, dtype=torch.int64), torch.zeros(1, dtype=torch.int64),
                        torch.zeros(rows, dtype=torch.int32), "blocks")
    assert torch.equal(seen[0], logits)


@pytest.mark.parametrize("taken,change", [(1, {}), (1, dict(rows=8)), (1, dict(x_ld=72)), (0, dict(rows=0)), (0, dict(rows=9)), (0, dict(k=0)),
                                          (0, dict(x_ld=0)), (0, dict(w_ld=0)), (0, dict(w_ld=48)), (0, dict(x_ld=56)), (0, dict(k=56)),
                                          (0, dict(dtype=_lib.SK_F32)), (0, dict(w=4096 + 16)), (0, dict(x=4096 + 8))])
def test_what_the_projection_takes(taken, change):
    """What linear_rows would refuse is not applicable, so that linear() sends it to the library."""
    p = _lib.LinearParams(x=4096, w=4096, out=4096, x_ld=64, w_ld=64, out_ld=32, rows=2, n=32, k=64, dtype=_lib.SK_BF16)
    for name, value in change.items():
        setattr(p, name, value)
    assert _lib.blocks().skb_linear_rows_applicable(C.byref(p)) == taken
    assert _lib.lib().sk_linear_rows_applicable(C.byref(p)) == taken


def test_tensors_elsewhere_are_refused(caught):
    """One tensor of each call on another device; nothing is launched (a launch would find no reader here)."""
    x, w, there = torch.randn(2, 64).bfloat16(), torch.randn(24, 64).bfloat16(), dict(dtype=torch.bfloat16, device="meta")
    tok, pos, seq = torch.zeros(2, 1, dtype=torch.int64), torch.zeros(1, dtype=torch.int64), torch.zeros(2, dtype=torch.int32)
    for call in (lambda: few_rows.linear(x, w.to("meta")), lambda: few_rows.linear(x, w, res=torch.empty(2, 24, **there)),
                 lambda: few_rows.linear_glu(x, w, 0, 8, 8, 0, act=torch.empty(2, 8, **there)),
                 lambda: few_rows.rms_norm(x, torch.empty(64, **there), 1e-5),
                 lambda: few_rows.pick_token(x, tok.to("meta"), pos, seq, "step"),
                 lambda: few_rows.pick_token(x, tok, pos.to("meta"), seq, "step"),
                 lambda: few_rows.pick_token(x, tok, pos, seq.to("meta"), "step")):
        with pytest.raises(RuntimeError, match="tensors of one call"):
            call()


def test_counts_of_another_layout_are_refused(caught):
    logits, tok, pos = torch.randn(2, 64).bfloat16(), torch.zeros(2, 1, dtype=torch.int64), torch.zeros(1, dtype=torch.int64)
    for p, seq in ((pos, torch.zeros(4, dtype=torch.int32)[::2]), (torch.zeros(2, dtype=torch.int64), torch.zeros(2, dtype=torch.int32))):
        with pytest.raises(AssertionError):
            few_rows.pick_token(logits, tok, p, seq, "step")


@pytest.mark.parametrize("chained", [False, True])
def test_products_are_chained_only_inside_a_stack(monkeypatch, chained):
    """A mixer called by itself may stand right behind a kernel that wrote its weights; a decoder's stack says it does not."""
    from socket_b200 import mixers as m

    seen = []

    class Stop(Exception):
        pass

    def product(x, w, *args, chained=False, **kw):
        seen.append(chained)
        raise Stop

    monkeypatch.setattr(m.ops, "linear", product)
    monkeypatch.setattr(m.ops, "linear_glu", product)
    h, at = torch.zeros(2, 64), m.Portion(2, 1, 0, **({"chained": True} if chained else {}))
    memory = m.MatrixMemory(64, 2, 8, 8, 15.0, 1e-5)
    calls = [lambda: m.ChunkedAttention(64, 2, 1, 8, 8, 16, 1.0, 8, 4.0)(h, None, at),
             lambda: m.LatentAttention(64, 2, 8, 8, 8, 16, 8, 1e4, 1.0, 1e-5)(h, None, at),
             lambda: m.Mamba2(64, 2, 8, 8, 1, 4, 1, 1e-5)(h, None, at),
             lambda: m.ParallelLayer(64, memory, 16)(h, None, at), lambda: m.ParallelLayer(64, memory, 0)(h, None, at),
             lambda: memory.mix([], h, m.MemoryState(2, 2, 8, 8, "cpu"), at, h),
             lambda: m.ClampedFeedForward(64, 16, 7.0)(h, *([True] if chained else []))]
    for call in calls:
        with pytest.raises(Stop):
            call()
    assert seen == [chained] * len(calls)
