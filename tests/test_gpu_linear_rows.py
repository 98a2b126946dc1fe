"""Projections of a few rows against float64: edges of tiles (16 and 32 weight rows), of the pieces of 64 along k, of the
division of k among 8 and 16 warps, several tiles per CTA, and the gated unit beside plain rows."""
import pytest
import torch

pytestmark = pytest.mark.gpu


EPS = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11, torch.float32: 2.0 ** -23}


def _sums(x, w, library=False):
    """Per result, how far an fp32 sum may be off: each addition at most 2^-23 of the magnitudes added.  The kernel adds a
    warp's part of k (an eighth of its pieces of up to 128 elements), then 16 warps; of the library's order nothing is known."""
    k = x.shape[1]
    adds = k if library else min(k, k // 8 + 128) + 16
    return x.double().abs() @ w.double().abs().t() * adds * 2.0 ** -23


def _bound(x, w, dtype, f32, library=False):
    """Those sums, then one rounding to the type."""
    return _sums(x, w, library), 0.0 if f32 else EPS[dtype]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows,n,k", [(1, 1, 16), (8, 16, 64), (3, 17, 48), (2, 33, 1040), (5, 2369, 528), (8, 4752, 128), (1, 2368, 2064),
                                      (7, 9600, 192), (4, 19008, 64), (8, 100, 14336)])
def test_plain_products(rows, n, k, dtype):
    from socket_b200 import block_ops as ops
    g = torch.Generator(device="cuda").manual_seed(n + k)
    x = torch.randn(rows, k + 8, generator=g, device="cuda").to(dtype)[:, :k]          # strided rows
    w = torch.randn(n, k + 16, generator=g, device="cuda").to(dtype)[:, :k]
    res = torch.randn(rows, n, generator=g, device="cuda").to(dtype)
    assert ops._linear_params(x, w, False) is not None
    want = x.double() @ w.double().t()
    for f32, r, chained in ((True, None, False), (False, None, True), (False, res, False)):
        got = ops.linear(x, w, f32=f32, res=r, chained=chained).double()
        ref = want if r is None else want + r.double()
        tol, eps = _bound(x, w, dtype, f32)
        assert got.shape == ref.shape and bool(((got - ref).abs() <= tol + eps * ref.abs() + 1e-7).all())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows,k,ff,plain", [(1, 64, 16, 0), (8, 128, 33, 40), (3, 1040, 5632, 3072), (8, 512, 100, 4800)])
@pytest.mark.parametrize("kind", [0, 1])
def test_gated_unit(rows, k, ff, plain, kind, dtype):
    from socket_b200 import block_ops as ops
    g = torch.Generator(device="cuda").manual_seed(ff)
    x = torch.randn(rows, k, generator=g, device="cuda").to(dtype)
    w = (torch.randn(plain + 2 * ff + 8, k, generator=g, device="cuda") * 2 * k ** -0.5).to(dtype)
    wide = torch.full((rows, ff + 24), 3.0, device="cuda", dtype=dtype)
    out, act = ops.linear_glu(x, w, plain, plain + ff + 8, ff, kind, limit=1.5, slope=1.7, plain=plain, act=wide[:, 8:8 + ff])
    y, off = x.double() @ w.double().t(), _sums(x, w)
    gates, ups = slice(plain, plain + ff), slice(plain + ff + 8, plain + 2 * ff + 8)
    slope, a, b = (1.7, y[:, gates].clamp(max=1.5), y[:, ups].clamp(-1.5, 1.5) + 1) if kind == ops.GLU_CLAMPED else (1.0, y[:, gates], y[:, ups])
    want = a * torch.sigmoid(slope * a) * b
    # a sigmoid(slope a) has slopes up to 1.1 and is at most |a|; the exponential is off by 2 + 1.18 |slope a| units in the last
    # place, the division by 2, three more roundings; then one to the type (fp16: at least half a denormal step)
    d_gate, d_up = off[:, gates], off[:, ups]
    unit = 1.1 * d_gate * (b.abs() + d_up) + a.abs() * d_up + want.abs() * (8 + 1.2 * (slope * a).abs()) * 2.0 ** -23
    assert bool(((act.double() - want).abs() <= unit + EPS[dtype] * (want.abs() + unit) + 2.0 ** -25).all())
    assert bool((wide[:, :8] == 3).all()) and bool((wide[:, 8 + ff:] == 3).all())
    tol, eps = _bound(x, w[:plain], dtype, False)
    assert bool(((out.double() - y[:, :plain]).abs() <= tol + eps * y[:, :plain].abs() + 1e-7).all())


@pytest.mark.parametrize("rows", [1, 8])
@pytest.mark.parametrize("graph", [False, True])
def test_chained_products_behind_one_another(rows, graph):
    """Projections of all forms (16 and 32 rows a tile, 16 warps, the unit), each reading what the one before wrote: chained or
    not, the same bits."""
    from socket_b200 import block_ops as ops
    g = torch.Generator(device="cuda").manual_seed(rows)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda")
    sizes = [512, 9600, 2048, 4800, 256, 512]
    ws = [(r(n, k) * k ** -0.5).bfloat16() for k, n in zip(sizes, sizes[1:])]
    glu = (r(1024, 512) * 512 ** -0.5).bfloat16()

    def chain(x, chained):
        for _ in range(3):
            for w in ws:
                x = ops.linear(x, w, chained=chained)
            x = ops.linear_glu(x, glu, 0, 512, 512, ops.GLU_SILU, chained=chained)[1]
        return x

    x0 = r(rows, 512).bfloat16()
    want = chain(x0, False)
    x = x0.clone()                                                # unchained, behind everything that made the weights
    if not graph:
        assert torch.equal(chain(x, True), want)
        return
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        chain(x, True)
        recorded = torch.cuda.CUDAGraph()
        with torch.cuda.graph(recorded, stream=side):
            got = chain(x.clone(), True)
    torch.cuda.current_stream().wait_stream(side)
    for _ in range(3):
        got.zero_()
        recorded.replay()
        assert torch.equal(got, want)


def test_shapes_outside_go_to_the_library():
    from socket_b200 import block_ops as ops
    x, w = torch.randn(9, 64, device="cuda").bfloat16(), torch.randn(24, 64, device="cuda").bfloat16()
    for a, b in ((x, w), (x[:2, :40], w[:, :40]), (x[:2].float(), w.float())):
        assert ops._linear_params(a, b, False) is None
        torch.testing.assert_close(ops.linear(a, b), torch.mm(a, b.t()))
        assert ops.linear_glu(a, b, 0, 8, 8, ops.GLU_SILU) is None


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("batch,vocab", [(1, 1), (3, 33), (2, 4096), (8, 32768), (1, 50257)])
def test_pick_token(batch, vocab, dtype):
    from socket_b200 import few_rows
    g = torch.Generator(device="cuda").manual_seed(vocab)
    wide = torch.randn(batch, vocab + 8, generator=g, device="cuda").to(dtype)
    logits = wide[:, :vocab]
    rows = [logits.clone() for _ in range(4)]
    rows[1][:, vocab // 2:] = rows[1].amax()                      # equal largest ones: the first of them
    rows[2][:] = -float("inf")
    rows[3][:, vocab // 3] = float("nan")
    for library in ("step", "blocks"):
        for x in [logits] + rows:
            tok = torch.full((batch, 1), -1, dtype=torch.int64, device="cuda")
            pos = torch.tensor([41], device="cuda")
            seq = torch.arange(batch, dtype=torch.int32, device="cuda")
            few_rows.pick_token(x, tok, pos, seq, library)
            v = x.double().cpu()
            v = torch.where(v.isnan(), torch.full_like(v, float("inf")), v)
            want = torch.tensor([[int((r == r.max()).nonzero()[0])] for r in v])
            assert torch.equal(tok.cpu(), want) and int(pos) == 42 and torch.equal(seq.cpu(), torch.arange(1, batch + 1, dtype=torch.int32))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows,width", [(1, 8), (2, 33), (8, 4096), (3, 5000), (1, 16384), (2, 2049), (2, 16392), (3, 16387), (2, 131080), (1, 70001)])
def test_rms_norm_rows(rows, width, dtype):
    from socket_b200 import few_rows
    g = torch.Generator(device="cuda").manual_seed(width)
    x, w = torch.randn(rows, width, generator=g, device="cuda").to(dtype), torch.randn(width, generator=g, device="cuda").to(dtype)
    want = x.double() / torch.sqrt((x.double() ** 2).mean(-1, keepdim=True) + 1e-5) * w.double()
    # the sum of squares in fp32: a thread's additions in order, then 10 of the tree, each off by at most 2^-24 of the sum, and the
    # square root halves that; some roundings of the factors; one to the type
    adds = max(16, width / 512) + 10
    eps = {torch.float32: 0.0, torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}[dtype] + (adds / 2 + 5) * 2.0 ** -24
    assert bool(((few_rows.rms_norm(x, w, 1e-5).double() - want).abs() <= eps * want.abs() + 6e-8).all())


@pytest.mark.parametrize("rows", [1, 2, 8, 9])
@pytest.mark.parametrize("layout", ["strided", "broadcast", "turned"])
def test_residual_layouts(rows, layout):
    from socket_b200 import block_ops as ops
    n, k = 72, 128
    g = torch.Generator(device="cuda").manual_seed(rows)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda").bfloat16()
    x, w = r(rows, k), r(n, k)
    res = {"strided": r(rows, n + 8)[:, 8:], "broadcast": r(1, n).expand(rows, n), "turned": r(n, rows).t()}[layout]
    want = x.double() @ w.double().t() + res.double()
    tol, eps = _bound(x, w, torch.bfloat16, False, library=rows > 8)
    if rows > 8:                                                  # the library rounds the product before the sum
        tol = tol + eps * (want - res.double()).abs()
    assert bool(((ops.linear(x, w, res=res).double() - want).abs() <= tol + eps * want.abs() + 1e-7).all())


@pytest.mark.parametrize("rows", [1, 2, 8, 9])
@pytest.mark.parametrize("layout", ["broadcast", "turned"])
def test_pick_token_layouts(rows, layout):
    from socket_b200 import few_rows
    g = torch.Generator(device="cuda").manual_seed(rows)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda")
    logits = r(1, 1000).expand(rows, 1000) if layout == "broadcast" else r(1000, rows).t()
    tok = torch.zeros(rows, 1, dtype=torch.int64, device="cuda")
    pos, seq = torch.zeros(1, dtype=torch.int64, device="cuda"), torch.zeros(rows, dtype=torch.int32, device="cuda")
    few_rows.pick_token(logits, tok, pos, seq, "step")
    assert torch.equal(tok, logits.argmax(-1, keepdim=True))


@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("form", ["expanded rows", "expanded weights", "no rows", "no columns", "no weights", "one weight row"])
def test_what_only_the_library_takes(form, f32):
    from socket_b200 import block_ops as ops
    r = lambda *s: torch.randn(*s, device="cuda").bfloat16()
    x, w = r(3, 64), r(24, 64)
    x, w = {"expanded rows": (x[:1].expand(3, 64), w), "expanded weights": (x, w[:1].expand(24, 64)), "no rows": (x[:0], w),
            "no columns": (x[:, :0], w[:, :0]), "no weights": (x, w[:0]), "one weight row": (x, r(64, 1).t())}[form]
    got = ops.linear(x, w, f32=f32)
    assert got.shape == (x.shape[0], w.shape[0]) and got.dtype == (torch.float32 if f32 else torch.bfloat16)
    want = x.double() @ w.double().t()
    tol, eps = _bound(x, w, torch.bfloat16, f32, library=True)
    assert bool(((got.double() - want).abs() <= tol + eps * want.abs() + 1e-7).all())
    if form in ("expanded rows", "no rows", "no columns"):
        assert ops.linear_glu(x, w, 0, 8, 8, ops.GLU_SILU) is None


def test_doubles_go_to_the_library():
    from socket_b200 import block_ops as ops
    x, w = torch.randn(2, 64, device="cuda", dtype=torch.float64), torch.randn(24, 64, device="cuda", dtype=torch.float64)
    torch.testing.assert_close(ops.linear(x, w), x @ w.t())
