"""The weight-streaming GEMM of a process that drives every rank, at the edges of its rule and tiles, against fp64 products (the
bounds of test_gpu_gemm_local.py)."""
import pytest
import torch

from gpu_ipc_example_b200 import Communicator

pytestmark = pytest.mark.gpu
HALF_ULP = {torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8}


def _rand(g, dtype, *shape, scale=1.0):
    return (torch.randn(*shape, device="cuda", generator=g) * scale).to(dtype)


def _close(got, want, dtype):
    # fp32 sums of K products of N(0, 1) x N(0, 0.02): off by less than K * 2^-24 * 0.02 * 4; one rounding to 16 bit
    torch.testing.assert_close(got.double(), want, atol=1e-4, rtol=1.01 * HALF_ULP[dtype])


def _check_kernel(comm, tiles, splits):
    """One tile per CTA (cluster) is this kernel; the other one reports all of its tiles as steps."""
    if splits:
        assert comm.last_info.steps == 1 and comm.last_info.ctas == tiles * splits
    else:
        assert comm.last_info.steps > 1


# rows: one, the accumulator's steps, one less and one more; no split, two, four, eight; a last tile of 64 rows of W; K that fills
# no block; ranks that meet inside a share of K; splits 0: the other kernel's side of the rule
@pytest.mark.parametrize("world,M,K,N,splits", [
    (1, 1, 72, 4864, 1), (1, 16, 448, 4864, 1), (1, 17, 448, 4864, 0), (1, 16, 1024, 8192, 2), (1, 17, 1024, 8192, 2), (1, 16, 2048, 3136, 4),
    (1, 5, 8192, 1280, 8), (1, 17, 2056, 6016, 4), (1, 32, 3000, 4928, 4), (1, 33, 2048, 6464, 4), (1, 64, 2056, 6464, 4),
    (1, 64, 2056, 6016, 0), (1, 64, 448, 4864, 0), (1, 65, 2048, 8192, 0), (2, 48, 1000, 8192, 4), (2, 15, 1000, 5120, 4), (2, 31, 1792, 8192, 4),
    (4, 3, 264, 6144, 2), (8, 16, 136, 8192, 2), (8, 24, 456, 4864, 4)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_linear(world, M, K, N, splits, dtype):
    g = torch.Generator(device="cuda").manual_seed(M + K)
    xs = [_rand(g, dtype, M, K) for _ in range(world)]
    ws = [_rand(g, dtype, N, K, scale=0.02) for _ in range(world)]
    res = [_rand(g, dtype, M, N) for _ in range(world)]
    gam = [1 + _rand(g, dtype, N, scale=0.1) for _ in range(world)]
    y = sum(x.double() @ w.double().t() for x, w in zip(xs, ws))
    with Communicator.virtual(world, 0, staging_bytes=96 << 20) as comm:
        outs = comm.linear_allreduce(xs, ws)
        _check_kernel(comm, -(-N // 128), splits)
        for o in outs:
            _close(o, y, dtype)
        for o, s, r in zip(*comm.linear_allreduce(xs, ws, res), res):
            _close(s, y + r.double(), dtype)
            assert torch.equal(o, s)
        first = None
        for _ in range(20):  # back to back: every launch sets up while the one in front runs
            outs, sums = comm.linear_allreduce(xs, ws, res, gam, 1e-5)
            if first is None:
                first = [t.clone() for t in outs + sums]
        for a, b in zip(first, outs + sums):
            assert torch.equal(a, b), "the result must not depend on timing"
        for o, s, r, ga in zip(outs, sums, res, gam):
            _close(s, y + r.double(), dtype)
            want = s.double() * torch.rsqrt(s.double().pow(2).mean(-1, keepdim=True) + 1e-5) * ga.double()
            _close(o, want, dtype)
        torch.cuda.synchronize()
        comm.check()


# one shard; shards with padding rows between them and without; more rows than the kernel takes
@pytest.mark.parametrize("world,rows,K,N,splits", [(1, 7, 520, 4160, 1), (2, 3, 1000, 3136, 2), (2, 8, 1024, 4096, 2), (2, 16, 2048, 4096, 4),
                                                   (2, 17, 2048, 4096, 0), (4, 1, 2048, 1600, 4), (4, 8, 2056, 1600, 4), (4, 9, 2048, 3136, 0)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_gather_linear(world, rows, K, N, splits, dtype):
    g = torch.Generator(device="cuda").manual_seed(rows + K)
    xs = [_rand(g, dtype, rows, K) for _ in range(world)]
    ws = [_rand(g, dtype, N, K, scale=0.02) for _ in range(world)]
    full = torch.cat(xs).double()
    with Communicator.virtual(world, 0, staging_bytes=32 << 20) as comm:
        outs = comm.allgather_linear(xs, ws)
        _check_kernel(comm, -(-N // 128) * world, splits)
        for o, w in zip(outs, ws):
            _close(o, full @ w.double().t(), dtype)
        torch.cuda.synchronize()
        comm.check()
