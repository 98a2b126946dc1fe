"""The ends of a decode step in one launch each: the clustered greedy pick around the sizes its blocks divide, and the start on
given tokens."""
import pytest
import torch

from socket_b200 import few_rows

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("vocab", [1, 7, 8, 2047, 8192, 16384, 16392, 65536, 65537, 151936])
def test_pick_finds_a_peak_anywhere(vocab, dtype):
    x = torch.zeros(3, vocab, dtype=dtype, device=DEV)
    tok, pos = torch.zeros(3, 1, dtype=torch.int64, device=DEV), torch.zeros(1, dtype=torch.int64, device=DEV)
    seq = torch.zeros(3, dtype=torch.int32, device=DEV)
    for i, at in enumerate((0, vocab - 1, vocab // 2, vocab // 3)):
        x.zero_()
        x[:, at] = 1
        x[1, vocab - 1] = 1                                  # an equal one behind it
        few_rows.pick_token(x, tok, pos, seq, "blocks")
        assert tok.flatten().tolist() == [at] * 3 and int(pos) == i + 1 and seq.tolist() == [i + 1] * 3


@pytest.mark.parametrize("library", ["step", "blocks"])
@pytest.mark.parametrize("batch,n", [(1, 0), (8, 1), (130, 64), (3, 65), (2, 200)])
def test_begin_token(batch, n, library):
    first = torch.randint(0, 1 << 40, (batch, 1), device=DEV)
    tok, pos = torch.zeros_like(first), torch.zeros(1, dtype=torch.int64, device=DEV)
    seq = torch.zeros(batch, dtype=torch.int32, device=DEV)
    lengths = [torch.zeros((), dtype=torch.int32, device=DEV) for _ in range(n)]
    few_rows.begin_token(first, tok, pos, seq, 70001, lengths, library)
    assert torch.equal(tok, first) and int(pos) == 70001 and seq.tolist() == [70001] * batch
    assert all(int(t) == 70001 for t in lengths)
