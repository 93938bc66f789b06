"""All-reduce + residual + RMSNorm of a process that drives every rank: rows on one CTA and on clusters, one and two vectors
per thread, rows that do not divide over threads or CTAs, against fp64.  One rounding of the sum, one of the result."""
import pytest
import torch

from gpu_ipc_example_b200 import Communicator

pytestmark = pytest.mark.gpu
HALF_ULP = {torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8}


@pytest.mark.parametrize("world", [1, 2, 4, 8])
@pytest.mark.parametrize("rows,hidden", [(1, 8), (1, 264), (3, 1032), (16, 8192), (100, 4104), (300, 5128), (512, 8192), (2, 32768), (200, 12296), (1, 40960)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_direct(world, rows, hidden, dtype):
    g = torch.Generator(device="cuda").manual_seed(rows + hidden)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
    xs = [rnd(rows, hidden).to(dtype) for _ in range(world)]
    res = [rnd(rows, hidden).to(dtype) for _ in range(world)]
    gam = [(1 + 0.1 * rnd(hidden)).to(dtype) for _ in range(world)]
    res[-1], gam[-1] = res[0], gam[0]
    total = sum(x.double() for x in xs)
    with Communicator.virtual(world, 0, staging_bytes=16 << 20) as comm:
        outs, sums = comm.allreduce_residual_rmsnorm(xs, res, gam, 1e-5)
        torch.cuda.synchronize()
        comm.check()
    u = HALF_ULP[dtype]
    for o, s, r, ga in zip(outs, sums, res, gam):
        # fp32 sums of at most nine values of a few units: off by less than 1e-5
        torch.testing.assert_close(s.double(), total + r.double(), atol=1e-5, rtol=1.01 * u)
        want = s.double() * torch.rsqrt(s.double().pow(2).mean(-1, keepdim=True) + 1e-5) * ga.double()
        torch.testing.assert_close(o.double(), want, atol=1e-6, rtol=1.01 * u)
    assert torch.equal(outs[0], outs[-1]) and torch.equal(sums[0], sums[-1])  # same residual and gamma: the same bits


@pytest.mark.parametrize("world", [1, 2, 8])
def test_the_kernel_with_the_exchange(world):
    """An explicit CTA count asks for the kernel that runs with one process per GPU."""
    g = torch.Generator(device="cuda").manual_seed(world)
    xs = [torch.randn(16, 2048, device="cuda", generator=g).half() for _ in range(world)]
    res, gam = torch.randn(16, 2048, device="cuda", generator=g).half(), torch.ones(2048, device="cuda").half()
    with Communicator.virtual(world, 0, staging_bytes=16 << 20) as comm:
        a = comm.allreduce_residual_rmsnorm(xs, [res] * world, [gam] * world, 1e-5, ctas=8)
        assert comm.last_info.sched == "oneshot"
        b = comm.allreduce_residual_rmsnorm(xs, [res] * world, [gam] * world, 1e-5)
        torch.cuda.synchronize()
        comm.check()
        for q in range(world):
            assert torch.equal(a[1][q], b[1][q])
            torch.testing.assert_close(a[0][q], b[0][q], atol=1e-6, rtol=2.0 ** -10)
