"""Which form of the state-space recurrence a call takes (no GPU)."""
import ctypes as C

import pytest

from socket_b200 import _lib

AUTO, STEPS, CHUNKS, TENSOR = 0, 1, 2, 3


def _params(**kw):
    p = _lib.SsmParams()
    f = dict(xbc=1 << 20, y=1 << 21, state=1 << 22, B=2, S=300, H=8, P=64, N=128, G=2, taps=4, dtype=_lib.SK_BF16, path=AUTO,
             xbc_ld=8 * 64 + 2 * 2 * 128, in_ld=4096)
    for k, v in {**f, **kw}.items():
        setattr(p, k, v)
    return p


@pytest.mark.parametrize("kw,path", [
    ({}, TENSOR), (dict(S=65), TENSOR), (dict(S=64), CHUNKS), (dict(S=15), STEPS), (dict(N=200), CHUNKS), (dict(N=12), STEPS),
    (dict(P=12), STEPS), (dict(P=8, N=8), TENSOR), (dict(pos=1 << 23), STEPS), (dict(dtype=_lib.SK_F32), STEPS),
    (dict(xbc=(1 << 20) + 8), STEPS), (dict(xbc_ld=1028), STEPS), (dict(y=(1 << 21) + 2), CHUNKS), (dict(state=(1 << 22) + 4), CHUNKS),
    (dict(path=CHUNKS), CHUNKS), (dict(path=STEPS), STEPS)])
def test_route_and_workspace(kw, path):
    p = _params(**kw)
    lib = _lib.blocks()
    assert lib.skb_ssm_path(C.byref(p)) == path
    blocks = {TENSOR: -(-p.S // 128) * 128, CHUNKS: -(-p.S // 64) * 64, STEPS: 0}[path]
    assert lib.skb_ssm_workspace_bytes(C.byref(p)) == 8 * p.B * p.H * blocks
