"""Cache appends of 16-bit rows in one tensor-core launch, against the general kernel (which fp32 planes of the same values
select): the same cache rows, codes, norms and length, bit for bit.  Both let fp32 sums decide a sign outside the same band, so
codes and norms of both are also compared with float64 sums."""
import pytest
import torch

from socket_b200 import _lib, ops

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _cache(B, Hkv, T, dtype):
    z = lambda *s, dt=dtype: torch.full(s, 7, dtype=dt, device=DEV)  # noqa: E731
    return [z(B, Hkv, T, 128), z(B, Hkv, T, 128), z(B, Hkv, T, 32, dt=torch.uint8), z(B, Hkv, T, dt=torch.float16),
            torch.zeros((), dtype=torch.int32, device=DEV)]


def _against_fp64(cache, pos, k, v, planes):
    """Codes of the rows at their positions: signs of float64 sums, where no order of summing 128 products can change them.  Norms: float64
    ones rounded to fp32 and then to fp16."""
    live = (pos >= 0) & (pos < cache[0].shape[2])
    k, v, at = k[:, live].double(), v[:, live].double(), pos[live]
    flat = planes.double().view(256, 128)
    for h in range(k.shape[2]):
        kh = k[:, :, h]
        prod = (kh @ flat.t()).nan_to_num(nan=-1.0, posinf=1.0, neginf=-1.0)
        finite = torch.isfinite(kh).all(-1, keepdim=True) & torch.isfinite(flat).all(-1)
        band = 1e-13 * kh.nan_to_num(0.0, 0.0, 0.0).norm(dim=-1, keepdim=True) * flat.nan_to_num(0.0, 0.0, 0.0).norm(dim=-1)
        sure = (prod.abs() > band) | (prod == 0) | ~finite
        codes = cache[2][:, h, at]
        bits = (codes[..., None] >> torch.arange(7, -1, -1, device=DEV) & 1).bool().flatten(2)
        assert torch.equal(bits & sure, (prod >= 0) & sure)
        assert torch.equal(cache[3][:, h, at], (v[:, :, h] ** 2).sum(-1).sqrt().float().half())


def _both(B, S, Hkv, T, pos, k, v, planes):
    got, want = _cache(B, Hkv, T, k.dtype), _cache(B, Hkv, T, k.dtype)
    flags = [torch.zeros((), dtype=torch.int32, device=DEV) for _ in range(2)]
    ops.kv_append(*got, pos, k, v, planes, status=flags[0])
    ops.kv_append(*want, pos, k, v, planes.float(), status=flags[1])
    for name, g, w in zip(("keys", "values", "codes", "norms", "length"), got, want):
        assert torch.equal(g.view(torch.uint8) if g.dim() else g, w.view(torch.uint8) if w.dim() else w), name
    assert int(flags[0]) == int(flags[1])
    _against_fp64(got, pos, k, v, planes)
    return got, int(flags[0])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,S,Hkv,start", [(1, 1024, 1, 0), (1, 1025, 1, 3), (3, 347, 1, 0), (2, 257, 5, 100), (1, 8192, 8, 0),
                                           (4, 1999, 8, 1)])
def test_append_on_tensor_cores_equals_the_exact_kernel(B, S, Hkv, start, dtype):
    g = torch.Generator(device=DEV).manual_seed(B * S + Hkv)
    r = lambda *s: torch.randn(*s, generator=g, device=DEV)  # noqa: E731
    k, v = (r(B, S, Hkv, 128) * torch.exp(r(128))).to(dtype), r(B, S, Hkv, 128).to(dtype)
    pos = start + torch.randperm(S, generator=g, device=DEV)
    _both(B, S, Hkv, start + S + 5, pos, k, v, r(32, 8, 128).to(dtype))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_append_of_hostile_rows_is_exact(dtype):
    """Rows of zeros, orthogonal to planes, tiny, huge, infinite and NaN; planes of zeros and tiny ones; positions outside the
    cache."""
    g = torch.Generator(device=DEV).manual_seed(3)
    S = 1300
    planes = torch.randn(32, 8, 128, generator=g, device=DEV).to(dtype)
    k = torch.randn(1, S, 1, 128, generator=g, device=DEV).to(dtype)
    v = torch.randn(1, S, 1, 128, generator=g, device=DEV).to(dtype)
    planes[0, 0] = 0
    planes[1, 1] *= 1e-3
    planes[5, :, 64:] = 0
    k[0, 5] = 0
    k[0, 6] = 0
    k[0, 6, 0, 0], k[0, 6, 0, 1] = planes[3, 2, 1], -planes[3, 2, 0]
    k[0, 200:600, :, :64] = 0                                # orthogonal to a whole table
    k[0, 600:620] *= 1e-4 if dtype == torch.float16 else 1e-25
    k[0, 620:640] *= 6e4 if dtype == torch.float16 else 1e37
    k[0, 640, 0, 3] = float("inf")
    k[0, 641, 0, 3] = float("-inf")
    k[0, 642, 0, 3] = float("nan")
    k[0, 643, 0, 3], k[0, 643, 0, 4] = float("inf"), float("inf")
    pos = torch.arange(S, device=DEV)
    pos[7], pos[9] = -1, S + 100
    _, flags = _both(1, S, 1, S + 2, pos, k, v, planes)
    assert flags != 0
    if dtype == torch.bfloat16:                              # planes whose squares vanish in fp32
        _both(1, S, 1, S + 2, torch.arange(S, device=DEV), k, v, (planes.float() * 1e-25).to(dtype))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
def test_the_exact_kernel_against_fp64(dtype):
    """Its fp32 sums decide only what fp64 would decide alike: hostile rows, few rows (the general kernel for every type)."""
    g = torch.Generator(device=DEV).manual_seed(11)
    S = 397
    planes, k, v = (torch.randn(*s, generator=g, device=DEV).to(dtype) for s in ((32, 8, 128), (1, S, 1, 128), (1, S, 1, 128)))
    planes[0, 0] = 0
    planes[5, :, 64:] = 0
    k[0, 5] = 0
    k[0, 6] = 0
    k[0, 6, 0, 0], k[0, 6, 0, 1] = planes[3, 2, 1], -planes[3, 2, 0]
    k[0, 20:60, :, :64] = 0
    k[0, 60:70] *= 1e-4 if dtype == torch.float16 else 1e-25
    k[0, 70:80] *= 6e4 if dtype == torch.float16 else 1e37
    v[0, 70:80] *= 1e3
    v[0, 60:70] *= 1e-6
    v[0, 5] = 0
    k[0, 81, 0, 3], k[0, 82, 0, 3], k[0, 83, 0, 3] = float("inf"), float("-inf"), float("nan")
    cache = _cache(1, 1, S, dtype)
    ops.kv_append(*cache, torch.arange(S, device=DEV), k, v, planes)
    prod = (k.double().view(S, 1, 128) * planes.double().view(1, 256, 128)).sum(-1)
    sure = ~(prod.abs() <= 1e-13 * k.double().view(S, 1, 128).norm(dim=-1) * planes.double().view(1, 256, 128).norm(dim=-1)) | (prod == 0)
    bits = (prod >= 0).view(S, 32, 8)
    got = (cache[2][0, 0, :, :, None] >> torch.arange(7, -1, -1, device=DEV) & 1).bool()
    assert torch.equal(got & sure.view(S, 32, 8), bits & sure.view(S, 32, 8))
    want = (v.double() ** 2).sum(-1).sqrt().float().half()[0, :, 0]
    assert torch.equal(cache[3][0, 0], want)


def test_append_where_every_projection_is_near_zero():
    S, planes = 4000, torch.randn(32, 8, 128, device=DEV).bfloat16()
    planes[:, :, 64:] = 0
    k = torch.zeros(1, S, 1, 128, device=DEV)
    k[..., 64:] = torch.randn(1, S, 1, 64, device=DEV)
    (_, _, codes, _, _), _ = _both(1, S, 1, S, torch.arange(S, device=DEV), k.bfloat16(), k.bfloat16(), planes)
    assert (codes[:, :, :S] == 255).all()


def test_rows_that_do_not_start_on_16_bytes_take_the_general_kernel():
    S = 1500
    planes = torch.randn(32, 8, 128, device=DEV).half()
    raw = torch.randn(2, S * 128 + 1, device=DEV).half()
    k, v = (t[1:].view(1, S, 1, 128) for t in raw)
    _both(1, S, 1, S, torch.arange(S, device=DEV), k, v, planes)


def test_entry_points_by_name_with_strides_rows_elsewhere_and_no_workspace():
    """`sk_hash_keys_tc` on rows 136 elements apart, whose codes go to rows 48 bytes apart in another order (negative: nowhere), and
    `sk_kv_append_tc`: neither reads a workspace."""
    g = torch.Generator(device=DEV).manual_seed(23)
    N, planes = 1000, torch.randn(32, 8, 128, generator=g, device=DEV).bfloat16()
    wide = torch.randn(N, 136, generator=g, device=DEV).bfloat16()
    wide[40:400, :64] = 0                                    # near zero against a table's planes: decided from the rows in memory
    planes[5, :, 64:] = 0
    k, st = wide[:, :128].contiguous(), torch.cuda.current_stream().cuda_stream
    want = ops.hash_keys(k, planes)
    to = torch.randperm(N, generator=g, device=DEV)
    to[::7] = -1
    codes = torch.full((N, 48), 9, dtype=torch.uint8, device=DEV)
    lib = _lib.lib()
    assert lib.sk_hash_keys_tc_workspace_bytes(N) == lib.sk_kv_append_tc_workspace_bytes(1, N, 1) == 0
    assert lib.sk_hash_keys_tc(wide.data_ptr(), 136, planes.data_ptr(), N, 128, 32, 8, codes.data_ptr(), 48, to.data_ptr(), None, 0, None, st) == 0
    expect = torch.full_like(codes, 9)
    expect[to[to >= 0], :32] = want[to >= 0]
    assert torch.equal(codes, expect)
    v, pos = torch.randn(1, N, 1, 128, generator=g, device=DEV).bfloat16(), torch.arange(N, device=DEV)
    for S in (100, N):                                       # fewer rows than the general entry point would bring here, and more
        got, ref = _cache(1, 1, N, torch.bfloat16), _cache(1, 1, N, torch.bfloat16)
        kc, vc, cc, nc, length = got
        assert lib.sk_kv_append_tc(k.data_ptr(), v.data_ptr(), _lib.SK_BF16, pos.data_ptr(), planes.data_ptr(), _lib.SK_BF16, kc.data_ptr(),
                                   vc.data_ptr(), cc.data_ptr(), nc.data_ptr(), length.data_ptr(), None, 1, S, 1, 128, N, 32, 8, None, 0, st) == 0
        ops.kv_append(*ref, pos[:S], k.view(1, N, 1, 128)[:, :S], v[:, :S], planes.float())
        assert all(torch.equal(a, b) for a, b in zip(got, ref))
