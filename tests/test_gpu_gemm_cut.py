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


def _check_cut(comm, tiles, cut):
    """The launch report counts the tiles and parts of tiles that were taken: those behind the last full wave are cut."""
    room = comm.last_info.ctas // 2
    assert comm.last_info.steps == tiles + tiles % room * (cut - 1)


# on 74 pairs of SMs: 34 tiles left, in two parts, of one rank and of two; 66 left, whole, as two parts each would not fit a wave; two
# left, in four parts; four left, of which the last one's last part is empty, of one rank and of two
@pytest.mark.parametrize("world,M,K,N,bn,cut", [
    (1, 2048, 2056, 8192, 256, 2), (2, 2048, 1032, 8192, 256, 2), (1, 1800, 2048, 8128, 224, 1), (2, 2000, 1024, 8192, 224, 1),
    (1, 512, 2104, 9728, 256, 4), (1, 700, 2056, 9728, 192, 4), (2, 700, 1032, 9728, 192, 4)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_linear(world, M, K, N, bn, cut, dtype):
    g = torch.Generator(device="cuda").manual_seed(M + K)
    xs = [_rand(g, dtype, M, K) for _ in range(world)]
    ws = [_rand(g, dtype, N, K, scale=0.02) for _ in range(world)]
    res = [_rand(g, dtype, M, N) for _ in range(world)]
    y = sum(x.double() @ w.double().t() for x, w in zip(xs, ws))
    with Communicator.virtual(world, 0, staging_bytes=512 << 20) as comm:
        outs = comm.linear_allreduce(xs, ws)
        _check_cut(comm, -(-M // bn) * -(-N // 256), cut)
        for o in outs:
            _close(o, y, dtype)
        for o, s, r in zip(*comm.linear_allreduce(xs, ws, res), res):
            _close(s, y + r.double(), dtype)
            assert torch.equal(o, s)
        torch.cuda.synchronize()
        comm.check()


# the last: of the six tiles left two have an empty part
@pytest.mark.parametrize("world,rows,K,N,bn,cut", [(1, 2048, 2048, 8192, 256, 2), (2, 1024, 2048, 3584, 256, 4), (2, 1000, 2056, 3584, 256, 4),
                                                   (2, 700, 2056, 4864, 256, 4)])
def test_gather_linear(world, rows, K, N, bn, cut):
    g = torch.Generator(device="cuda").manual_seed(rows + K)
    xs = [_rand(g, torch.float16, rows, K) for _ in range(world)]
    ws = [_rand(g, torch.float16, N, K, scale=0.02) for _ in range(world)]
    full = torch.cat(xs).double()
    with Communicator.virtual(world, 0, staging_bytes=32 << 20) as comm:
        outs = comm.allgather_linear(xs, ws)
        _check_cut(comm, -(-rows // bn) * -(-N // 256) * world * world, cut)
        for o, w in zip(outs, ws):
            _close(o, full @ w.double().t(), torch.float16)
        torch.cuda.synchronize()
        comm.check()
