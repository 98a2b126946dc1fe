"""The original-layout scorer at the edges of its blocks of 1024 keys and on both sides of its rule (tables, table size): the same
bits as adding the tables one by one in fp32."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,L,R,T", [(148, 32, 256, 1), (148, 32, 256, 511), (160, 32, 64, 513), (150, 16, 256, 1024), (75, 32, 256, 1025),
                                     (37, 16, 128, 4096), (3, 32, 256, 1500), (149, 24, 256, 700), (150, 32, 512, 600), (1, 32, 256, 1),
                                     (2, 16, 256, 1025), (1, 32, 384, 2048), (1, 32, 385, 2048)])
def test_same_bits_as_table_by_table(H, L, R, T):
    from socket_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(T)
    q = torch.rand(1, H, 1, L, R, generator=g, device="cuda")
    codes = torch.randint(0, R, (1, H, L, T), generator=g, device="cuda").to(torch.int16)
    allowed = torch.rand(1, H, 1, T, generator=g, device="cuda") < 0.9
    v = torch.rand(1, H, 1, T, generator=g, device="cuda")
    got = ops.soft_hash_collision(q, codes, allowed, v)
    s = torch.zeros(1, H, T, device="cuda")
    for table in range(L):
        s = s + q[:, :, 0, table].gather(-1, codes[:, :, table].long())
    want = (s * v[:, :, 0]).masked_fill(~allowed[:, :, 0], -float("inf"))
    assert torch.equal(got[:, :, 0], want)
