"""Waits inside the GEMM kernels of a process that drives every rank that run out: partial sums of a K split that nobody sends.  The
kernel returns, the status says which wait it was, and the next call is right: shared and tensor memory were given back."""
import pytest
import torch

from gpu_ipc_example_b200 import Communicator
from gpu_ipc_example_b200.parallel.communicator import CollectiveError

pytestmark = pytest.mark.gpu
MUTE_SENDS = 2


# the weight-streaming kernel, its K in four parts; tiles of SM pairs, K in two (more rows than the former takes)
@pytest.mark.parametrize("M,K,N,where", [(16, 2048, 3136, 41), (80, 4096, 2048, 40)])
def test_partial_sums_unsent(M, K, N, where):
    g = torch.Generator(device="cuda").manual_seed(M)
    x, w = torch.randn(M, K, device="cuda", generator=g).half(), (torch.randn(N, K, device="cuda", generator=g) * 0.02).half()
    with Communicator.virtual(1, 0, staging_bytes=32 << 20) as comm:
        want = comm.linear_allreduce([x], [w])[0].clone()
        comm.set_timeout_ms(20)
        out = torch.empty(M, N, device="cuda", dtype=x.dtype)
        torch.ops.b200ipc.local_gemm_ar([x], [w], [], [], [out], [], 0.0, False, comm._h, MUTE_SENDS)
        torch.cuda.synchronize()
        with pytest.raises(CollectiveError, match="bounded wait ran out"):
            comm.check()
        assert comm.status()["where"] == where
        comm.reset()
        comm.set_timeout_ms(2000)
        for _ in range(3):
            assert torch.equal(comm.linear_allreduce([x], [w])[0], want)
        torch.cuda.synchronize()
        comm.check()
