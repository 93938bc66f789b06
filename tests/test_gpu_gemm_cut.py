"""The tiles behind the last full wave of the GEMM of a process that drives every rank, taken in parts, against fp64 products (the
bounds of test_gpu_gemm_local.py)."""
import pytest
import torch

from gpu_ipc_example_b200 import Communicator

pytestmark = pytest.mark.gpu
HALF_ULP = {torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8}


def _rand(g, dtype, *shape, scale=1.0):
    return (torch.randn(*shape, device="cuda", generator=g) * scale).to(dtype)


def _close(got, want, dtype):
    torch.testing.assert_close(got.double(), want, atol=1e-4, rtol=1.01 * HALF_ULP[dtype])


# on 74 pairs of SMs: 34 tiles left, in two parts; the same with a last row of tiles of which a part is empty; two ranks; two tiles
# left, in four parts
@pytest.mark.parametrize("world,M,K,N", [(1, 2048, 2056, 8192), (1, 1800, 2048, 8128), (2, 2000, 1024, 8192), (1, 512, 2104, 9728)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_linear(world, M, K, N, dtype):
    g = torch.Generator(device="cuda").manual_seed(M + K)
    xs = [_rand(g, dtype, M, K) for _ in range(world)]
    ws = [_rand(g, dtype, N, K, scale=0.02) for _ in range(world)]
    res = [_rand(g, dtype, M, N) for _ in range(world)]
    y = sum(x.double() @ w.double().t() for x, w in zip(xs, ws))
    with Communicator.virtual(world, 0, staging_bytes=512 << 20) as comm:
        for o in comm.linear_allreduce(xs, ws):
            _close(o, y, dtype)
        for o, s, r in zip(*comm.linear_allreduce(xs, ws, res), res):
            _close(s, y + r.double(), dtype)
            assert torch.equal(o, s)
        torch.cuda.synchronize()
        comm.check()


@pytest.mark.parametrize("world,rows,K,N", [(1, 2048, 2048, 8192), (2, 1024, 2048, 3584), (2, 1000, 2056, 3584)])
def test_gather_linear(world, rows, K, N):
    g = torch.Generator(device="cuda").manual_seed(rows + K)
    xs = [_rand(g, torch.float16, rows, K) for _ in range(world)]
    ws = [_rand(g, torch.float16, N, K, scale=0.02) for _ in range(world)]
    full = torch.cat(xs).double()
    with Communicator.virtual(world, 0, staging_bytes=32 << 20) as comm:
        for o, w in zip(comm.allgather_linear(xs, ws), ws):
            _close(o, full @ w.double().t(), torch.float16)
        torch.cuda.synchronize()
        comm.check()
