"""RoPE + cache append inside the attention kernel, the single-tensor RMSNorm and the arg-max over logits, where they can go
wrong: the new position at the edges of splits and tiles, more splits than tiles, ties, NaN, rows of -inf, odd widths."""
import pytest
import torch

from gpu_ipc_example_b200._ext import load

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("G", [1, 2, 4, 8])
@pytest.mark.parametrize("pos,splits", [(0, 1), (0, 4), (15, 2), (16, 3), (63, 4), (64, 4), (1000, 32), (2047, 8)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_rope_decode_attention_is_the_two_kernels(G, pos, splits, dtype):
    """The same roundings in the same places: the caches and the result are bit-identical."""
    C = load()
    B, hkv, D, max_ctx, theta = 3, 2, 128, 2048, 5e5
    hq = hkv * G
    g = torch.Generator(device="cuda").manual_seed(pos + G)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g).to(dtype)
    qkv, kc, vc = rnd(B, (hq + 2 * hkv) * D), rnd(B, hkv, max_ctx, D), rnd(B, hkv, max_ctx, D)
    ws = torch.zeros(C.attention_workspace_bytes(B, hq, hkv, splits), dtype=torch.uint8, device="cuda")
    q2, k2, v2 = qkv.clone(), kc.clone(), vc.clone()
    torch.ops.b200ipc.rope_kv_append(q2, k2, v2, hq, hkv, pos, theta)
    want = torch.ops.b200ipc.decode_attention(q2, k2, v2, ws, hq, hkv, pos + 1, splits)
    before = qkv.clone()
    got = torch.ops.b200ipc.rope_decode_attention(qkv, kc, vc, ws, hq, hkv, pos, splits, theta)
    torch.cuda.synchronize()
    assert torch.equal(got, want) and torch.equal(kc, k2) and torch.equal(vc, v2) and torch.equal(qkv, before)


def test_rope_decode_attention_refuses_a_position_outside_the_cache():
    C = load()
    qkv, kc = torch.zeros(1, 3 * 128, device="cuda").half(), torch.zeros(1, 1, 16, 128, device="cuda").half()
    ws = torch.zeros(C.attention_workspace_bytes(1, 1, 1, 1), dtype=torch.uint8, device="cuda")
    for pos in (-1, 16):
        with pytest.raises(RuntimeError):
            torch.ops.b200ipc.rope_decode_attention(qkv, kc, kc.clone(), ws, 1, 1, pos, 1, 5e5)


@pytest.mark.parametrize("rows,cols", [(1, 1), (3, 7), (2, 512), (33, 16032), (4, 4099)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_row_argmax(rows, cols, dtype):
    load()
    g = torch.Generator(device="cuda").manual_seed(cols)
    x = torch.randn(rows, cols, device="cuda", generator=g).to(dtype)
    x[0] = 0.5  # all equal: the first one
    if rows > 1:
        x[1] = float("-inf")
    if rows > 2:
        x[2, cols // 2:] = float("nan")  # the first NaN
    v, i = torch.ops.b200ipc.row_argmax(x)
    f = x.float().cpu()
    for r in range(rows):
        nan = torch.isnan(f[r]).nonzero()
        want = int(nan[0]) if len(nan) else int((f[r] == f[r].max()).nonzero()[0])
        assert int(i[r]) == want and torch.equal(v[r].cpu(), f[r, want]) or bool(torch.isnan(v[r])) and int(i[r]) == want


@pytest.mark.parametrize("rows,hidden", [(1, 8), (5, 1000), (64, 8192), (3, 12288)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_rmsnorm(rows, hidden, dtype):
    load()
    g = torch.Generator(device="cuda").manual_seed(hidden)
    x, gam = torch.randn(rows, hidden, device="cuda", generator=g).to(dtype), (1 + 0.1 * torch.randn(hidden, device="cuda", generator=g)).to(dtype)
    want = x.double() * torch.rsqrt(x.double().pow(2).mean(-1, keepdim=True) + 1e-5) * gam.double()
    u = 2.0 ** -11 if dtype == torch.float16 else 2.0 ** -8  # one rounding
    torch.testing.assert_close(torch.ops.b200ipc.rmsnorm(x, gam, 1e-5).double(), want, atol=1e-6, rtol=1.01 * u)


def test_rmsnorm_of_strided_and_unaligned_operands():
    load()
    g = torch.Generator(device="cuda").manual_seed(0)
    x, gam = torch.randn(5, 64, device="cuda", generator=g).half(), torch.randn(64, device="cuda", generator=g).half()
    want = torch.ops.b200ipc.rmsnorm(x, gam, 1e-5)
    shifted = torch.zeros(72, device="cuda").half()
    shifted[1:65] = gam
    spread = torch.zeros(64, 2, device="cuda").half()
    spread[:, 1] = gam
    for ga in (shifted[1:65], spread[:, 1]):
        assert torch.equal(torch.ops.b200ipc.rmsnorm(x, ga, 1e-5), want)
        assert torch.equal(torch.ops.b200ipc.rmsnorm(x.t().contiguous().t(), ga, 1e-5), want)
