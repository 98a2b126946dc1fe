"""The state-space recurrence in chunks of 128 tokens on the tensor cores, which portions from 65 tokens up take: against the plain
form, and its state against the token-by-token form."""
import pytest
import torch

from socket_b200 import block_ops as ops
from test_gpu_radapel_blocks import _close, _plain_ssm, _ssm_inputs

pytestmark = pytest.mark.gpu
DEV, BF16 = "cuda:0", torch.bfloat16
CASES = [dict(H=4, P=24, N=16, G=2, taps=3), dict(H=2, P=64, N=128, G=1, taps=4), dict(H=3, P=40, N=24, G=3, taps=2),
         dict(H=2, P=72, N=72, G=2, taps=4), dict(H=2, P=8, N=8, G=1, taps=1)]


def _scan(proj, w, c, B, S, inner, state, conv, path="auto", start=0):
    return ops.ssm(proj, inner, w["conv_w"], w["conv_b"], w["dt_bias"], w["A_log"], w["D"], conv, state, S=S, groups=c["G"], path=path,
                   start=start)


@pytest.mark.parametrize("case", range(len(CASES)))
@pytest.mark.parametrize("sizes", [[65], [128], [129], [300], [128, 172], [70, 1, 229], [100, 200]])
def test_portions_of_all_sizes(case, sizes):
    c, B, S = CASES[case], 2, sum(sizes)
    proj, w, inner, ch = _ssm_inputs(c, B, S, BF16)
    want, want_st = _plain_ssm(c, proj, w, inner, ch, B, S)
    w, rows = {k: v.to(DEV) for k, v in w.items()}, proj.to(DEV).view(B, S, -1)
    conv = torch.full((B, c["taps"] - 1, ch), 5.0, dtype=BF16, device=DEV)
    state = torch.full((B, c["H"], c["N"], c["P"]), 3.0, device=DEV)      # not seen by a portion at position 0
    out, at = [], 0
    for n in sizes:
        y = _scan(rows[:, at:at + n].reshape(B * n, -1), w, c, B, n, inner, state, conv, start=at)
        out.append(y.view(B, n, inner))
        at += n
    _close(torch.cat(out, 1), want, BF16)
    _close(state, want_st, BF16, tol16=1e-2)


@pytest.mark.parametrize("decay", [-6.0, 1.0, 4.0])
def test_the_state_keeps_more_than_bf16(decay):
    """As in the block form: at most 3e-5 of the largest state after 1000 tokens, whatever the decay."""
    c, B, S = dict(H=2, P=32, N=64, G=1, taps=1), 1, 1000
    proj, w, inner, ch = _ssm_inputs(c, B, S, BF16, seed=9)
    w["A_log"] = torch.tensor([decay, decay - 0.5])
    w = {k: v.to(DEV) for k, v in w.items()}
    states, ys = [], []
    for path in ("steps", "auto"):
        conv, state = torch.zeros(B, 0, ch, dtype=BF16, device=DEV), torch.zeros(B, 2, 64, 32, device=DEV)
        ys.append(_scan(proj.to(DEV), w, c, B, S, inner, state, conv, path=path).float())
        states.append(state)
    assert (states[0] - states[1]).abs().max() <= 3e-5 * states[0].abs().max()
    # both round their outputs to bf16: neighbours at most, where the sums are not near zero
    assert (ys[0] - ys[1]).abs().max() <= 2.0 ** -7 * ys[0].abs().max()


def test_many_chunks_and_heads():
    """More blocks than the GPU holds at a time, each going round its barriers many times."""
    c, B, S = dict(H=64, P=64, N=128, G=8, taps=4), 3, 1701
    proj, w, inner, ch = _ssm_inputs(c, B, S, BF16, seed=3)
    w = {k: v.to(DEV) for k, v in w.items()}
    got = []
    for path in ("chunks", "auto"):
        conv, state = torch.zeros(B, 3, ch, dtype=BF16, device=DEV), torch.zeros(B, 64, 128, 64, device=DEV)
        y = _scan(proj.to(DEV), w, c, B, S, inner, state, conv, path=path).float()
        got.append((y, state))
    assert torch.isfinite(got[1][0]).all()
    assert (got[0][1] - got[1][1]).abs().max() <= 6e-5 * got[0][1].abs().max()
    assert (got[0][0] - got[1][0]).abs().max() <= 2.0 ** -7 * got[0][0].abs().max()


def test_the_skip_is_one_fp32_product():
    """Without queries an output is the skip alone: D x in fp32, rounded once to the output's type, as the block form leaves it."""
    c, B, S = dict(H=64, P=24, N=16, G=2, taps=1), 2, 333     # many skips: an input has 128 mantissas only
    proj, w, inner, ch = _ssm_inputs(c, B, S, BF16, seed=5)
    n_qk = c["G"] * c["N"]
    w["conv_b"][inner + n_qk:inner + 2 * n_qk] = 0
    proj[:, inner + inner + n_qk:inner + inner + 2 * n_qk] = 0
    w["D"] *= 10.0 ** torch.linspace(-3, 3, c["H"])
    w = {k: v.to(DEV) for k, v in w.items()}
    got = []
    for path in ("chunks", "auto"):
        conv, state = torch.zeros(B, 0, ch, dtype=BF16, device=DEV), torch.zeros(B, c["H"], c["N"], c["P"], device=DEV)
        got.append(_scan(proj.to(DEV), w, c, B, S, inner, state, conv, path=path))
    assert (got[0] != 0).float().mean() > 0.9
    assert torch.equal(got[0], got[1])


@pytest.mark.parametrize("value", [float("inf"), float("nan")])
@pytest.mark.parametrize("at", [0, 37, 127, 128, 200, 383])
def test_a_value_that_is_not_finite_reaches_no_token_before_its_16(at, value):
    """One such x: its column from its 16 tokens on, as in the block form; every other output as without it, bit for bit."""
    c, B, S, col = dict(H=2, P=72, N=24, G=1, taps=1), 1, 400, 72 + 67      # head 1, beyond its first 64 columns
    proj, w, inner, ch = _ssm_inputs(c, B, S, BF16, seed=7)
    w = {k: v.to(DEV) for k, v in w.items()}
    got = []
    for x in (None, value):
        rows = proj.clone()
        if x is not None:
            rows[at, inner + col] = x
        conv, state = torch.zeros(B, 0, ch, dtype=BF16, device=DEV), torch.zeros(B, 2, 24, 72, device=DEV)
        got.append((_scan(rows.to(DEV), w, c, B, S, inner, state, conv), state.transpose(2, 3).reshape(B, inner, -1)))
    (y0, st0), (y1, st1) = got
    assert torch.isfinite(y0).all() and not torch.isfinite(y1[at, col]) and not torch.isfinite(st1[:, col]).any()
    first = at // 16 * 16
    assert torch.equal(y0[:first], y1[:first])
    others = torch.arange(inner, device=DEV) != col
    assert torch.equal(y0[:, others], y1[:, others]) and torch.equal(st0[:, others], st1[:, others])
