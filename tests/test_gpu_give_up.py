"""Waits inside the kernels of a process that drives every rank that run out: partial sums of a K split that nobody sends, a CTA that
stays away from the decode step's meeting points.  The kernel returns, the status says which wait it was, and the next call is right:
shared and tensor memory were given back."""
import pytest
import torch

from gpu_ipc_example_b200 import Communicator
from gpu_ipc_example_b200.models.llama import LlamaConfig, LlamaTP
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


# one launch, CTAs with several tiles of the cache each; several launches, the cache longer than the rings
@pytest.mark.parametrize("world,layers,batch,pos", [(1, 2, 4, 300), (2, 6, 64, 2000)])
def test_decode_step_meeting(world, layers, batch, pos):
    cfg = LlamaConfig(layers=layers, hidden=1024, n_heads=4 * world, n_kv_heads=2 * world, ffn=512 * world, vocab=512)
    with Communicator.virtual(world, 0, staging_bytes=64 << 20) as comm:
        m = LlamaTP(cfg, comm, batch=batch, max_ctx=pos + 1, fusion="gemm", seed=1)
        assert m.one_kernel
        for caches in (m.kcache, m.vcache):
            for t in (t for rank in caches for t in rank):
                t.normal_()
        tokens = torch.arange(batch, device="cuda")

        def step(flags=0):
            m.pos = pos
            if not flags:
                return [m.decode(tokens), *m.last_hidden]
            per = lambda ws: [ws[r][l] for l in range(layers) for r in range(world)]
            return torch.ops.b200ipc.decode_step(m.embed[tokens], per(m.wqkv), per(m.wo), per(m.wgu), per(m.wdown), per(m.kcache), per(m.vcache),
                                                 m.lm_head, m.norm_attn, m.norm_mlp, m.norm_final, m.step_ws, m.hq, m.hkv, pos, cfg.eps,
                                                 cfg.rope_theta, comm._h, flags)

        want = [t.clone() for t in step()]
        comm.set_timeout_ms(20)
        assert step(MUTE_SENDS)
        torch.cuda.synchronize()
        with pytest.raises(CollectiveError, match="bounded wait ran out"):
            comm.check()
        assert comm.status()["where"] == 50
        comm.reset()
        comm.set_timeout_ms(2000)
        for _ in range(3):
            for a, b in zip(step(), want):
                assert torch.equal(a, b)
        torch.cuda.synchronize()
        comm.check()
