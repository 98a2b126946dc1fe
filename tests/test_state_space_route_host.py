"""Which form of the state-space recurrence a call takes (no GPU)."""
import ctypes as C

import pytest
import torch

from socket_b200 import _lib, block_ops, mixers

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


@pytest.mark.parametrize("off", [4, 8, 12])
def test_a_workspace_off_16_bytes(off):
    """The tensor-core forms move their scratch 16 bytes at a time.  The state space takes the blocks of 64 tokens instead, for which the
    scratch asked for without a workspace is enough; the matrix memory refuses before any launch."""
    lib, p = _lib.blocks(), _params()
    asked = lib.skb_ssm_workspace_bytes(C.byref(p))
    p.workspace = (1 << 24) + off
    assert lib.skb_ssm_path(C.byref(p)) == CHUNKS and lib.skb_ssm_workspace_bytes(C.byref(p)) <= asked
    p.workspace = (1 << 24) + 16
    assert lib.skb_ssm_path(C.byref(p)) == TENSOR and lib.skb_ssm_workspace_bytes(C.byref(p)) == asked
    m = _lib.MlstmParams()
    for name in ("q", "k", "v", "z", "norm_w", "gates", "i_bias", "f_bias", "S_state", "n_state", "m_state", "num", "den", "m_next", "out"):
        setattr(m, name, 1 << 20)
    m.dtype, m.B, m.S, m.H, m.N, m.P, m.cap = _lib.SK_BF16, 1, 300, 4, 64, 64, 15.0
    m.in_ld, m.gates_ld, m.out_ld = 2048, 8, 256
    assert lib.skb_mlstm_path(C.byref(m)) == TENSOR
    m.workspace, m.workspace_bytes = (1 << 24) + off, lib.skb_mlstm_workspace_bytes(C.byref(m))
    assert lib.skb_mlstm(C.byref(m), None) == -3 and b"workspace" in lib.skb_last_error()


def test_the_models_status_word_reaches_the_scan(monkeypatch):
    """A wait that runs out in the tensor-core form is reported in the word that `device_flags()` reads."""
    seen = []

    class Library:
        def skb_ssm_workspace_bytes(self, p):
            return 0

        def skb_ssm_conv(self, p, stream):
            return 0

        def skb_ssm_scan(self, p, stream):
            seen.append(p._obj.status)
            return 0

    monkeypatch.setattr(block_ops, "blocks", Library)
    monkeypatch.setattr(block_ops, "_require_cuda", lambda *t: None)
    monkeypatch.setattr(block_ops, "stream_ptr", lambda device: None)
    monkeypatch.setattr(block_ops, "gated_group_norm", lambda y, *a: torch.zeros_like(y))
    layer = mixers.Mamba2(32, heads=4, vdim=8, state=16, groups=2, taps=4, norm_groups=2, eps=1e-5)
    layer.finish_loading()
    cache = layer.make_cache(1, 200, torch.float32, "cpu")
    status = torch.zeros(1, dtype=torch.int32)
    layer(torch.zeros(100, 32), cache, mixers.Portion(1, 100, 0, status=status))
    layer(torch.zeros(100, 32), cache, mixers.Portion(1, 100, 100))
    assert seen == [status.data_ptr(), None]
