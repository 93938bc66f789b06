"""The row norm behind a GEMM of a process that drives every rank: rows that a CTA's registers hold and longer ones, whole and
ragged vectors per thread, both CTA sizes.  The norm is checked alone, against 64 bits, from the sums that the call returns."""
import pytest
import torch

from gpu_ipc_example_b200 import Communicator

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,n", [
    (1, 64),       # a quarter of a warp
    (5, 1088),
    (7, 8192),
    (3, 16384),    # the longest row of 512 threads in registers
    (3, 16448),    # ... and one that is read again
    (300, 4160),
    (300, 8192),   # the longest row of 256 threads in registers
    (297, 8256),
])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_row_norm(rows, n, dtype):
    eps = 1e-5
    g = torch.Generator(device="cuda").manual_seed(rows + n)
    x = torch.randn(rows, 64, device="cuda", generator=g).to(dtype)
    w = (torch.randn(n, 64, device="cuda", generator=g) * 0.02).to(dtype)
    res = torch.randn(rows, n, device="cuda", generator=g).to(dtype)
    gamma = (1 + 0.1 * torch.randn(n, device="cuda", generator=g)).to(dtype)
    with Communicator.virtual(1, 0, staging_bytes=(12 * max(rows, 32) * n * 2) + (64 << 20)) as comm:
        out, s = comm.linear_allreduce([x], [w], [res], [gamma], eps)
        comm.check()
        s64 = s[0].double()
        want = s64 * torch.rsqrt(s64.pow(2).mean(-1, keepdim=True) + eps) * gamma.double()
        # one rounding to the output's type (half a unit in the last place; its smallest numbers have a fixed spacing), and in fp32
        # two products, the root and a sum of squares whose additions per thread and across threads are fewer than 128
        u = 2.0 ** -11 if dtype == torch.float16 else 2.0 ** -8
        bound = want.abs() * (u + 140 * 2.0 ** -24) * (1 + u) + 2.0 ** -25
        assert bool(((out[0].double() - want).abs() <= bound).all())
