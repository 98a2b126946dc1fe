"""Row norms on both sides of the rules that request weights with the rows (few rows, one or two vectors a thread, short rows) and that
choose a block's threads: against float64, every way in and out."""
import pytest
import torch

from socket_b200 import block_ops as ops
from socket_b200 import few_rows

pytestmark = pytest.mark.gpu
DEV, BF16, F32 = "cuda:0", torch.bfloat16, torch.float32
EPS = 1e-3


def _r(g, *s, dtype=F32):
    return torch.randn(*s, generator=g, device=DEV).to(dtype)


def _rms(x, w):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS) * w


def _near(got, want):
    # fp32 sums of up to 8192 squares, then a rounding to the result's type: half a unit in its last place of the value
    tol = 2e-5 if got.dtype == F32 else 2.0 ** -8
    assert ((got.double() - want).abs() <= tol * want.abs() + 2e-5).all()


@pytest.mark.parametrize("width", [54, 1024, 2048, 3001, 4096, 5120, 8190, 8192])
@pytest.mark.parametrize("rows", [1, 32, 33, 148, 149, 295, 296, 400])
def test_residual_rows(rows, width):
    g = torch.Generator(device=DEV).manual_seed(rows * width)
    x, x0, y = _r(g, rows, width), _r(g, rows, width), _r(g, rows, width, dtype=BF16)
    wi, wo = _r(g, width, dtype=BF16), _r(g, width, dtype=BF16)
    xd, yd, wid, wod = x.double(), y.double(), wi.double(), wo.double()
    for y_in, kw, stream in ((None, {}, xd), (y, dict(w_in=wi), xd + _rms(yd, wid)), (y, {}, xd + yd),
                             (y.float(), dict(w_in=wi, replace=True), yd + wid)):
        for out in ("none", "norm", "layer", "x0"):
            if y_in is None and out == "none":
                continue
            s = x.clone()
            okw = {"none": {}, "norm": dict(w_out=wo), "layer": dict(w_out=wo, centred=True), "x0": dict(x0=x0, dtype=BF16)}[out]
            o = ops.residual_norm(s, EPS, **(dict(y=y_in) if y_in is not None else {}), **kw, **okw)
            _near(s, stream)
            if out == "norm":
                _near(o, _rms(stream, wod))
            elif out == "layer":
                _near(o, _rms(stream - stream.mean(-1, keepdim=True), wod))
            elif out == "x0":
                _near(o, torch.cat([stream, x0.double()], -1))


@pytest.mark.parametrize("width", [54, 2048, 5120])
@pytest.mark.parametrize("rows", [1, 200])
def test_the_stream_itself_as_second_half(rows, width):
    g = torch.Generator(device=DEV).manual_seed(width)
    x, y, w = _r(g, rows, width), _r(g, rows, width, dtype=BF16), _r(g, width, dtype=BF16)
    o = ops.residual_norm(x, EPS, y=y, w_in=w, x0=x, dtype=BF16)
    assert torch.equal(o, torch.cat([x, x], -1).to(BF16))


@pytest.mark.parametrize("inner,parts", [(4096, 8), (8192, 1), (8192, 8), (4096, 1), (3000, 3), (512, 1)])
@pytest.mark.parametrize("rows", [1, 18, 19, 148, 149, 300])
def test_gated_rows(rows, inner, parts):
    g = torch.Generator(device=DEV).manual_seed(rows + inner)
    y, z, w = _r(g, rows, inner, dtype=BF16), _r(g, rows, inner + 8, dtype=BF16), _r(g, inner, dtype=BF16)
    t = y.double() * torch.nn.functional.silu(z[:, :inner].double())
    want = _rms(t.view(rows, parts, -1), 1.0).reshape(rows, inner) * w.double()
    _near(ops.gated_group_norm(y, z, w, parts, EPS), want)


@pytest.mark.parametrize("dtype", [BF16, torch.float16, F32])
@pytest.mark.parametrize("width", [54, 2048, 4096, 4097, 8192, 16384, 20000])
@pytest.mark.parametrize("rows", [1, 148, 149, 300])
def test_rms_rows(rows, width, dtype):
    g = torch.Generator(device=DEV).manual_seed(rows + width)
    x, w = _r(g, rows, width, dtype=dtype), _r(g, width, dtype=dtype)
    _near(few_rows.rms_norm(x, w, EPS), _rms(x.double(), w.double()))


@pytest.mark.parametrize("dtype", [BF16, torch.float16, F32])
@pytest.mark.parametrize("vocab", [1, 31, 1024, 4095, 4096, 4097, 8200])
def test_pick_on_both_sides_of_the_cluster_rule(vocab, dtype):
    g = torch.Generator(device=DEV).manual_seed(vocab)
    x = _r(g, 3, vocab, dtype=dtype)
    x[0] = float("-inf")
    x[1, vocab // 2] = float("nan")
    want = torch.stack([x[0].new_zeros((), dtype=torch.long), x[0].new_full((), vocab // 2, dtype=torch.long), x[2].argmax()])
    tok, pos, seq = torch.zeros(3, 1, dtype=torch.int64, device=DEV), torch.zeros(1, dtype=torch.int64, device=DEV), torch.zeros(3, dtype=torch.int32, device=DEV)
    few_rows.pick_token(x, tok, pos, seq, "step")
    assert torch.equal(x[2, tok[2, 0]], x[2].max()) and torch.equal(tok[:2, 0], want[:2])
    assert int(tok[2, 0]) == int((x[2] == x[2].max()).nonzero()[0])
