"""Sparse decode attention at row counts and list lengths on both sides of the rules that deal a row's entries to clusters of CTAs, to
several clusters, or to CTAs without clusters: against float64, called by itself and inside a captured graph."""
import pytest
import torch

from socket_b200.kernels.sparse import sparse_attention_fwd

pytestmark = pytest.mark.gpu
DEV, T = "cuda:0", 5000
# error of fp32 sums of up to 4100 weighted values, and half a unit of the output type at the largest value (below 4)
TOL = {torch.float32: 2e-5, torch.bfloat16: 2.0 ** -7, torch.float16: 2.0 ** -10}


def _plain(q, k, v, lst, n):
    B, H, D = q.shape
    rep = H // k.shape[1]
    out = torch.empty(B, H, D, dtype=torch.float64, device=DEV)
    for b in range(B):
        for h in range(H):
            rows = lst[b, h, :int(n[b, h])].long()
            p = torch.softmax(k[b, h // rep, rows].double() @ q[b, h].double() / D ** 0.5, 0)
            out[b, h] = p @ v[b, h // rep, rows].double()
    return out


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("entries", [1, 63, 337, 1216, 2368, 4100])
@pytest.mark.parametrize("rows", [1, 4, 15, 16, 24, 33, 48, 64, 83, 96, 128, 149, 160])
def test_rows_and_entries(rows, entries, dtype):
    g = torch.Generator(device=DEV).manual_seed(rows * 10000 + entries)
    H = 4 if rows % 4 == 0 else 1
    B = rows // H
    r = lambda *s: torch.randn(*s, generator=g, device=DEV).to(dtype)  # noqa: E731
    q, k, v = r(B, H, 128), r(B, 1, T, 128), r(B, 1, T, 128)
    lst = torch.rand(B, H, T, generator=g, device=DEV).topk(entries).indices.int()
    n = torch.full((B, H), entries, dtype=torch.int32, device=DEV)
    n[0, 0] = max(1, entries // 3)                       # some CTAs of the first row have nothing
    want = _plain(q, k, v, lst, n)
    got = sparse_attention_fwd(q, k, v, lst, n)
    assert (got.double() - want).abs().max() <= TOL[dtype]
    assert torch.equal(got, sparse_attention_fwd(q, k, v, lst, n))          # tickets are back at zero, sums in one order
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        again = sparse_attention_fwd(q, k, v, lst, n)
    graph.replay()
    assert torch.equal(got, again)
