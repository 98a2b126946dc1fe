"""Row kernels of a prompt in the forms that its size or its layout selects."""
import pytest
import torch

from socket_b200 import block_ops as ops

pytestmark = pytest.mark.gpu
DEV, BF16 = "cuda:0", torch.bfloat16


@pytest.mark.parametrize("P", [8, 40, 256, 264])
def test_memory_outputs_by_warps_and_by_blocks(P):
    """A portion whose (token, head) pairs get a warp each, against a shorter one of the same tokens, whose pairs get a block."""
    H, N, S, short = 8, 16, 640, 512
    g = torch.Generator(device=DEV).manual_seed(P)
    r = lambda *s: torch.randn(*s, generator=g, device=DEV)  # noqa: E731
    rows, gates = r(S, 2 * H * (N + P)).to(BF16), r(S, 2 * H)
    bias, w = (torch.zeros(H, device=DEV), torch.full((H,), 3.0, device=DEV)), 1 + 0.1 * r(H * P)
    outs, states = [], []
    for n in (S, short):
        q, k, v, z = rows[:n].split([H * N, H * N, H * P, H * P], 1)
        state = [torch.zeros(1, H, N, P, device=DEV), torch.zeros(1, H, N, device=DEV), torch.zeros(1, H, device=DEV)]
        out = torch.empty(n, H * P, dtype=BF16, device=DEV)
        ops.mlstm(q, k, v, z, gates[:n], *bias, w.to(BF16), *state, out, S=n, cap=15.0, q_scale=N ** -0.5, eps=1e-5)
        outs.append(out.float())
        states.append(state[2])
    a, b = outs[0][:short], outs[1]
    assert torch.isfinite(outs[0]).all() and not torch.equal(states[0], states[1])
    assert ((a - b).abs() <= 2.0 ** -7 * torch.maximum(a.abs(), b.abs()) + 1e-3).all()      # roundings of num and of out


@pytest.mark.parametrize("dtype", [BF16, torch.float32])
@pytest.mark.parametrize("G,D,E,pad", [(4, 128, 128, 0), (1, 8, 24, 0), (3, 5, 7, 0), (2, 16, 16, 1), (8, 128, 64, 8), (2, 40, 40, 3)])
def test_ring_append_of_every_layout(G, D, E, pad, dtype):
    B, S, ring, start = 2, 21, 16, 5
    wide = torch.randn(B, S, G * (D + E) + pad, device=DEV).to(dtype)
    k, v = wide[..., :G * D].unflatten(-1, (G, D)), wide[..., G * D:G * (D + E)].unflatten(-1, (G, E))
    kc, vc = torch.zeros(B, ring, G, D, dtype=dtype, device=DEV), torch.zeros(B, ring, G, E, dtype=dtype, device=DEV)
    ops.ring_append(k, v, kc, vc, start=start)
    first = (start + S - 1) // ring * ring                   # the chunk of the last token
    for s in range(max(first - start, 0), S):
        slot = (start + s) % ring
        assert torch.equal(kc[:, slot], k[:, s]) and torch.equal(vc[:, slot], v[:, s])


@pytest.mark.parametrize("N,P,S", [(128, 256, 300), (136, 264, 700), (40, 72, 129), (256, 512, 257)])
def test_memory_states_of_every_width(N, P, S):
    """A head's state in parts of 16, 32 and 64 value columns, by how many sequences there are."""
    H = 8
    g = torch.Generator(device=DEV).manual_seed(N)
    r = lambda *s: torch.randn(*s, generator=g, device=DEV)  # noqa: E731
    base, base_gates = r(S, 2 * H * (N + P)).to(BF16), r(S, 2 * H)
    bias, w = (torch.zeros(H, device=DEV), torch.full((H,), 3.0, device=DEV)), (1 + 0.1 * r(H * P)).to(BF16)

    def run(B):
        rows, gates = base.repeat(B, 1), base_gates.repeat(B, 1)
        q, k, v, z = rows.split([H * N, H * N, H * P, H * P], 1)
        state = [torch.zeros(B, H, N, P, device=DEV), torch.zeros(B, H, N, device=DEV), torch.zeros(B, H, device=DEV)]
        out = torch.empty(B * S, H * P, dtype=BF16, device=DEV)
        ops.mlstm(q, k, v, z, gates, *bias, w, *state, out, S=S, cap=15.0, q_scale=N ** -0.5, eps=1e-5)
        return out.view(B, S, -1), state[0]

    runs = [run(B) for B in (1, 2, 4, 9)]
    for out, state in runs[1:]:                                # the same sums in the same order, in every sequence
        assert torch.equal(out, runs[0][0].expand_as(out)) and torch.equal(state, runs[0][1].expand_as(state))


@pytest.mark.parametrize("start,S,chunk,length", [(5, 40, 64, 256), (5, 59, 64, 256), (5, 60, 64, 256), (70, 50, 64, 256), (60, 100, 64, 256), (9, 70, 512, 100)])
def test_portion_inside_a_chunk_and_across(start, S, chunk, length):
    """A portion that attends on the ring's own rows, and one whose rows replace them, against both halves in one portion."""
    from socket_b200 import mixers
    torch.manual_seed(S)
    m = mixers.ChunkedAttention(64, 4, 2, 16, 24, chunk, 0.25, 12, 50.0).to(DEV).to(BF16)
    for p in m.parameters():
        p.data.copy_(0.3 * torch.randn_like(p))
    m.finish_loading()
    h = torch.randn(2, start + S, 64, device=DEV).to(BF16)
    whole, parts = (m.make_cache(2, length, BF16, DEV) for _ in range(2))
    flat = lambda x: x.reshape(-1, 64).contiguous()  # noqa: E731
    want = m(flat(h), whole, mixers.Portion(2, start + S, 0)).view(2, start + S, -1)
    m(flat(h[:, :start]), parts, mixers.Portion(2, start, 0))
    got = m(flat(h[:, start:]), parts, mixers.Portion(2, S, start)).view(2, S, -1)
    err = (got.float() - want[:, start:].float()).abs().max()
    assert err <= 2.0 ** -6 * want.float().abs().max(), float(err)               # weights, outputs and the projection in bf16
    kept = (start + S - 1) % chunk + 1                         # rows of the last token's chunk
    assert torch.equal(parts.k[:, :kept], whole.k[:, :kept]) and torch.equal(parts.v[:, :kept], whole.v[:, :kept])
