"""Prefill attention where its rules change: many heads of few key/value heads or of their own, biases whose table ends inside, at
and far before a half tile of 64 keys, rows that end anywhere in a query tile, head sizes with a ragged last MMA step."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _case(S, H, G, D, E, start, kv_start, bias_len, chunk, window, cap, sink, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = lambda *s: torch.randn(*s, generator=g, device="cuda")
    T = start + S - kv_start
    q, k, v = r(1, S, H, D).bfloat16(), r(1, T, G, D).bfloat16(), r(1, T, G, E).bfloat16()
    kw = dict(scale=2.0 * D ** -0.5, start=start, kv_start=kv_start, chunk=chunk, window=window, softcap=cap)
    if bias_len:
        kw["bias"] = 2.0 * r(H, bias_len)
    if sink:
        kw["sink"] = r(H)
    return q, k, v, kw


def _plain(q, k, v, kw, i, h):
    """Row i of head h in float64, and the sum of weights times |v|."""
    g = h // (q.shape[2] // k.shape[2])
    s = k[0, :, g].double() @ q[0, i, h].double() * kw["scale"]
    if kw["softcap"]:
        s = kw["softcap"] * torch.tanh(s / kw["softcap"])
    pos, j = kw["start"] + i, kw["kv_start"] + torch.arange(k.shape[1], device="cuda")
    if "bias" in kw:
        s = s + kw["bias"][h].double()[(pos - j).clamp(0, kw["bias"].shape[1] - 1)]
    seen = j <= pos
    if kw["chunk"]:
        seen &= j // kw["chunk"] == pos // kw["chunk"]
    if kw["window"]:
        seen &= pos - j < kw["window"]
    s = s.masked_fill(~seen, -float("inf"))
    if "sink" in kw:
        s = torch.cat([s, kw["sink"][h:h + 1].double()])
    p = torch.softmax(s, 0)[:k.shape[1]]
    return p @ v[0, :, g].double(), p @ v[0, :, g].double().abs()


@pytest.mark.parametrize("S,H,G,D,E,start,kv_start,bias_len,chunk,window,cap,sink", [
    (300, 11, 11, 192, 128, 9000, 0, 0, 0, 0, 0.0, True),        # an odd number of heads, each its own keys, 6 MB a head
    (515, 20, 10, 192, 128, 14000, 0, 0, 0, 0, 0.0, False),      # two query heads a key/value head, a ragged last block
    (700, 4, 2, 128, 128, 0, 0, 33, 0, 0, 0.0, False),           # bias constant beyond 32, inside the diagonal tiles
    (385, 4, 2, 128, 128, 640, 512, 193, 512, 0, 0.0, False),    # and at a half tile's edge, behind the chunk's first rows
    (257, 2, 2, 128, 64, 511, 0, 5000, 512, 0, 0.0, True),       # table longer than any distance
    (129, 3, 1, 72, 40, 200, 0, 70, 0, 0, 0.0, True),            # ragged head sizes
    (640, 2, 1, 128, 128, 900, 773, 0, 0, 128, 30.0, True),      # window as long as a tile, weights relative to zero
    (640, 2, 1, 128, 128, 900, 773, 100, 0, 128, 30.0, False),   # the same with a bias: running maximum under a cap
    (200, 2, 1, 144, 128, 100, 0, 0, 0, 65, 200.0, False),       # a cap too high for that
])
def test_forms(S, H, G, D, E, start, kv_start, bias_len, chunk, window, cap, sink):
    from socket_b200 import block_ops as ops
    q, k, v, kw = _case(S, H, G, D, E, start, kv_start, bias_len, chunk, window, cap, sink, S + D)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    got = ops.attn(q, k, v, path="prefill_tc", status=status, **kw)[0].double()
    assert int(status) == 0
    for i in sorted({0, 1, 31, 32, 63, 64, 127, 128, 255, 256, S // 2, S - 1} & set(range(S))):
        for h in range(H):
            want, mag = _plain(q, k, v, kw, i, h)
            # weights rounded to bf16 (2^-9 each, their sum is not), fp32 scores of at most 2^7 off by 2^-17, the result rounded
            assert bool(((got[i, h] - want).abs() <= 2.0 ** -8 * mag + 2.0 ** -8 * want.abs() + 1e-6).all()), (i, h)


@pytest.mark.parametrize("growth", [0.1, 0.6, -0.6])
@pytest.mark.parametrize("D,E,window,cap,bias_len", [(128, 128, 0, 0.0, 0), (192, 128, 300, 0.0, 0), (128, 64, 0, 0.0, 90), (64, 128, 0, 900.0, 0)])
def test_maximum_that_moves(growth, D, E, window, cap, bias_len):
    """Scores that rise from key to key, so that a tile's first weights are taken again and the sums before are scaled, or fall."""
    from socket_b200 import block_ops as ops
    q, k, v, kw = _case(400, 2, 1, D, E, 260, 0, bias_len, 0, window, cap, True, D + E)
    q[..., 0], k[..., 0] = 8.0, (growth * torch.arange(k.shape[1], device="cuda"))[None, :, None].bfloat16()
    q[:, ::3, :, 0] = 0.0                                          # every third row as it was, in the same warps
    kw["scale"] = 0.125
    got = ops.attn(q, k, v, path="prefill_tc", **kw)[0].double()
    for i in (0, 1, 2, 95, 127, 128, 255, 256, 300, 398, 399):
        for h in range(2):
            want, mag = _plain(q, k, v, kw, i, h)
            # as above; scores of at most 2^9 in fp32
            assert bool(((got[i, h] - want).abs() <= 2.0 ** -8 * mag + 2.0 ** -8 * want.abs() + 1e-6).all()), (i, h)


@pytest.mark.parametrize("S,H,G,D,E,start,bias_len,chunk,window,cap,sink", [
    (129, 2, 1, 128, 128, 3000, 0, 0, 0, 0.0, True),             # few blocks of many key tiles
    (40, 1, 1, 64, 128, 100, 50, 0, 0, 0.0, False),              # fewer tiles than parts
    (700, 2, 2, 192, 128, 0, 0, 0, 0, 0.0, True),                # first blocks of two tiles
    (300, 2, 1, 128, 72, 900, 0, 0, 200, 30.0, True),            # relative to zero; a part without one of the query tiles
    (257, 3, 1, 256, 40, 700, 90, 512, 0, 50.0, False),
])
def test_keys_shared_by_blocks(S, H, G, D, E, start, bias_len, chunk, window, cap, sink):
    """One sequence, whose blocks are shared by CTAs, against many, whose blocks are not."""
    from socket_b200 import block_ops as ops
    q, k, v, kw = _case(S, H, G, D, E, start, 0, bias_len, chunk, window, cap, sink, S)
    one = ops.attn(q, k, v, path="prefill_tc", **kw)[0].float()
    n = 592 // (H * ((S + 255) // 256)) + 1
    many = ops.attn(*(x.expand(n, *x.shape[1:]).contiguous() for x in (q, k, v)), path="prefill_tc", **kw).float()
    assert torch.equal(many[0].expand_as(many), many)
    # weights rounded to bf16 relative to another maximum, the results rounded
    assert bool(((one - many[0]).abs() <= 2.0 ** -7 * one.abs() + 2.0 ** -8 * v.abs().max().item()).all())


@pytest.mark.parametrize("kv_start", [2 ** 31 - 300, 2 ** 31 + 7, 2 ** 40])
@pytest.mark.parametrize("chunk,window,cap", [(0, 0, 0.0), (0, 200, 30.0), (2 ** 30, 0, 0.0)])
def test_positions_beyond_two_billion(kv_start, chunk, window, cap):
    """Key rows count from kv_start; where the first position lies must not matter without a chunk's edge in between."""
    from socket_b200 import block_ops as ops
    if chunk and kv_start < 2 ** 31:
        kv_start = 2 ** 31 - 2 ** 20                              # its chunk begins and ends far from these rows
    q, k, v, kw = _case(300, 2, 1, 128, 64, 250, 0, 0, 0, window, cap, False, 7)
    want = ops.attn(q, k, v, path="prefill_tc", **kw)
    kw.update(start=kv_start + 250, kv_start=kv_start, chunk=chunk)
    assert torch.equal(ops.attn(q, k, v, path="prefill_tc", **kw), want)
