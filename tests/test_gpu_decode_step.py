"""The decode step as one kernel against a recomputation in 64 bits, where
its work split can go wrong: positions at the edges of a tile, fewer and more (sequence, KV head) pairs than CTAs, widths that
do not fill a tile, several launches, every head ratio."""
import pytest
import torch
import torch.nn.functional as F

from gpu_ipc_example_b200 import Communicator
from gpu_ipc_example_b200.models.llama import LlamaConfig, LlamaTP, apply_rope, full_weights_from_shards

pytestmark = pytest.mark.gpu


def _exact(m, tokens, kc, vc, pos):
    """The step in 64 bits from the model's weights and caches [layer][B, heads, pos, D]: hidden states, new k and v per layer."""
    cfg, D = m.cfg, m.cfg.head_dim
    layers, _ = full_weights_from_shards(m)
    norm = lambda x, g: x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + cfg.eps) * g.double()
    B = tokens.shape[0]
    posv = torch.full((B,), pos, device=m.dev, dtype=torch.int64)
    h = m.embed[tokens].double()
    rep = cfg.n_heads // cfg.n_kv_heads
    new_k, new_v = [], []
    for l, (wq, wk, wv, wo, wg, wu, wd) in enumerate(layers):
        x = norm(h, m.norm_attn[l])
        q = apply_rope((x @ wq.double().t()).view(B, cfg.n_heads, D), posv, cfg.rope_theta)
        new_k.append(apply_rope((x @ wk.double().t()).view(B, cfg.n_kv_heads, D), posv, cfg.rope_theta))
        new_v.append((x @ wv.double().t()).view(B, cfg.n_kv_heads, D))
        k = torch.cat([kc[l].double(), new_k[l].unsqueeze(2)], 2).repeat_interleave(rep, 1)
        v = torch.cat([vc[l].double(), new_v[l].unsqueeze(2)], 2).repeat_interleave(rep, 1)
        p = torch.softmax((q.double().unsqueeze(2) @ k.transpose(2, 3)) / D ** 0.5, -1)
        h = h + (p @ v).reshape(B, -1) @ wo.double().t()
        x = norm(h, m.norm_mlp[l])
        h = h + (F.silu(x @ wg.double().t()) * (x @ wu.double().t())) @ wd.double().t()
    return norm(h, m.norm_final), new_k, new_v


def _rel(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm())


@pytest.mark.parametrize("world,B,pos,G,hkv,hidden,ffn,vocab,layers", [
    (1, 1, 1, 1, 1, 128, 8, 40, 1),          # one position in the cache, everything smaller than a tile
    (1, 3, 63, 8, 1, 1088, 136, 1001, 2),    # a tile less one position; widths that fill no tile; an odd vocabulary
    (2, 16, 64, 2, 1, 512, 264, 320, 2),
    (1, 17, 65, 4, 2, 1024, 384, 640, 2),    # the batch's padding steps
    (4, 33, 130, 1, 1, 256, 128, 96, 1),
    (8, 5, 200, 2, 1, 512, 64, 64, 3),       # two launches
    (1, 64, 300, 1, 4, 640, 512, 500, 1),    # more sequences than CTAs: whole ones
    (1, 50, 2000, 2, 3, 384, 128, 256, 1),   # ... and cut into runs
    (1, 1, 3000, 8, 1, 256, 128, 128, 9),    # every tile of a sequence on a CTA of its own
])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_decode_step(world, B, pos, G, hkv, hidden, ffn, vocab, layers, dtype):
    cfg = LlamaConfig(layers=layers, hidden=hidden, n_heads=world * hkv * G, n_kv_heads=world * hkv, ffn=world * ffn, vocab=world * vocab, dtype=dtype)
    with Communicator.virtual(world, 0, staging_bytes=96 << 20) as comm:
        m = LlamaTP(cfg, comm, batch=B, max_ctx=pos + 2, fusion="gemm", seed=3)
        assert m.one_kernel
        g = torch.Generator(device="cuda").manual_seed(pos)
        for caches in (m.kcache, m.vcache):
            for t in (t for rank in caches for t in rank):
                t.normal_(generator=g)
                t[:, :, pos:] = float("nan")  # nothing of a position that is not there yet may be used
        for gam in m.norm_attn + m.norm_mlp + [m.norm_final]:
            gam.copy_((1 + 0.1 * torch.randn(hidden, device="cuda", generator=g)).to(dtype))
        tokens = torch.randint(0, cfg.vocab, (B,), device="cuda", generator=g)
        past = [[torch.cat([m.__dict__[c][r][l][:, :, :pos] for r in range(world)], 1) for l in range(layers)] for c in ("kcache", "vcache")]
        want, want_k, want_v = _exact(m, tokens, *past, pos)
        err, runs = {}, []
        for one in (False, True, True):
            m.one_kernel = one
            m.pos = pos
            before = comm.launches
            ids = m.decode(tokens)
            torch.cuda.synchronize()
            comm.check()
            assert m.pos == pos + 1
            if one:  # the first norm, then launches of as many layers as their tensor maps leave room for
                assert comm.launches - before == 1 + -(-layers // (48 // (6 * world)))
            new = [torch.cat([m.__dict__[c][r][l][:, :, pos] for r in range(world)], 1) for c in ("kcache", "vcache") for l in range(layers)]
            err[one] = [_rel(m.last_hidden[0], want)] + [_rel(a, b) for a, b in zip(new, want_k + want_v)]
            for h in m.last_hidden[1:]:
                assert torch.equal(h, m.last_hidden[0]), "every rank must hold the same activations"
            head = torch.cat(list(m.lm_head)).double()
            logits = m.last_hidden[0].double() @ head.t()
            # the id's logit is the greatest one, but for the rounding of logits to 16 bits
            slack = 2.1 * (2.0 ** -11 if dtype == torch.float16 else 2.0 ** -8) * logits.abs().max()
            assert bool((logits.gather(1, ids[:, None])[:, 0] >= logits.max(1).values - slack).all())
            if one:
                runs.append([ids.clone(), *(h.clone() for h in m.last_hidden), *(x.clone() for x in new)])
        for a, b in zip(*runs):
            assert torch.equal(a, b), "the result must not depend on timing"
        # A layer rounds nine times on the way to the next (two norms, q / k / v, the turned q and k, the probabilities, the
        # attention, SiLU * up, two sums); a rounding to u changes a vector by at most u / sqrt(3) of its norm on average, and
        # independent ones add up as squares.
        u = 2.0 ** -11 if dtype == torch.float16 else 2.0 ** -8
        assert max(err[True]) <= u / 3 ** 0.5 * (9 * layers + 1) ** 0.5, (err[True], err[False])


def test_what_the_kernel_does_not_take_runs_as_the_chain():
    cfg = LlamaConfig(layers=2, hidden=256, n_heads=2, n_kv_heads=1, ffn=128, vocab=64)
    with Communicator.virtual(1, 0, staging_bytes=64 << 20) as comm:
        m = LlamaTP(cfg, comm, batch=65, max_ctx=8, fusion="gemm")
        assert not m.one_kernel  # more sequences than the accumulator has columns
        m.decode(torch.zeros(65, dtype=torch.int64, device="cuda"))
        cfg.hidden = 200  # the row-parallel GEMMs refuse it, so the step does
        with pytest.raises(RuntimeError):
            m = LlamaTP(cfg, comm, batch=2, max_ctx=4, fusion="gemm")
            m.pos = 1
            m.decode(torch.zeros(2, dtype=torch.int64, device="cuda"))
        cfg.hidden = 256
        m = LlamaTP(cfg, comm, batch=2, max_ctx=4, fusion="gemm")
        tokens = torch.zeros(2, dtype=torch.int64, device="cuda")
        for step in range(4):  # an empty cache first; then a weight that is a strided view, which the chain copies
            if step == 2:
                m.wqkv[0][1] = torch.cat([m.wqkv[0][1], m.wqkv[0][1]], 1)[:, :256]
            before = comm.launches
            m.decode(tokens)
            assert (comm.launches - before == 2) == (step == 1)
        with pytest.raises(RuntimeError):
            m.decode(tokens)  # past the end of the cache
        torch.cuda.synchronize()
        comm.check()
    with Communicator.virtual(2, 0, staging_bytes=64 << 20, max_ctas=8) as comm:  # the kernel would take the whole GPU
        cfg.n_heads, cfg.n_kv_heads = 4, 2
        assert not LlamaTP(cfg, comm, batch=2, max_ctx=4, fusion="gemm").one_kernel


def test_captured_steps_replay():
    """The kernel is one cooperative launch per step: a captured step replays with new tokens in the same buffer."""
    cfg = LlamaConfig(layers=2, hidden=512, n_heads=4, n_kv_heads=2, ffn=256, vocab=128)
    with Communicator.virtual(1, 0, staging_bytes=64 << 20) as comm:
        m = LlamaTP(cfg, comm, batch=4, max_ctx=80, fusion="gemm")
        for caches in (m.kcache, m.vcache):
            for t in caches[0]:
                t.normal_()
        tokens = torch.tensor([1, 2, 3, 4], device="cuda")

        def step():
            m.pos = 70
            return m.decode(tokens)

        step()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            ids = step()
        hidden = m.last_hidden[0]
        for t in ([5, 6, 7, 8], [9, 10, 11, 12]):
            tokens.copy_(torch.tensor(t, device="cuda"))
            graph.replay()
            got = ids.clone(), hidden.clone()
            assert torch.equal(got[0], step()) and torch.equal(got[1], m.last_hidden[0])
        torch.cuda.synchronize()
        comm.check()


@pytest.mark.parametrize("name,value", [("one_kernel", False), ("kernels", False), ("local_gemm", True), ("fusion", "allreduce"), ("stage_events", [])])
def test_switches_that_are_set_later_pick_the_chain(name, value):
    cfg = LlamaConfig(layers=2, hidden=256, n_heads=2, n_kv_heads=1, ffn=128, vocab=64)
    with Communicator.virtual(1, 0, staging_bytes=64 << 20) as comm:
        m = LlamaTP(cfg, comm, batch=2, max_ctx=4, fusion="gemm")
        tokens = torch.tensor([3, 5], device="cuda")

        def step():
            m.pos, before = 1, comm.launches
            m.decode(tokens)
            return comm.launches - before, m.last_hidden[0].float()

        launches, want = step()
        assert launches == 2
        setattr(m, name, value)
        launches, got = step()
        assert launches != 2
        # the bound of test_decode_step for each of the two ways; the PyTorch ops of kernels=False round a norm twice
        assert _rel(got, want) <= 2 * 2.0 ** -11 / 3 ** 0.5 * (11 * cfg.layers + 2) ** 0.5
        if name == "stage_events":
            assert {n for n, *_ in m.stage_events} >= {"qkv_gemm", "rope_attention"}
        torch.cuda.synchronize()
        comm.check()


@pytest.mark.parametrize("batch,G,tiles,one", [(56, 8, 0, False), (55, 8, 0, True), (56, 8, -1, True), (56, 4, 0, True)])
def test_attention_heavy_steps_run_as_the_chain(batch, G, tiles, one):
    """Both sides of the rule: from 160 tiles of 64 positions per SM on (here exactly, or one tile per sequence less)."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    pos = 64 * (-(-160 * sms // (56 * 4)) + tiles)
    cfg = LlamaConfig(layers=1, hidden=256, n_heads=4 * G, n_kv_heads=4, ffn=128, vocab=64)
    with Communicator.virtual(1, 0, staging_bytes=64 << 20) as comm:
        m = LlamaTP(cfg, comm, batch=batch, max_ctx=pos + 1, fusion="gemm")
        m.pos, before = pos, comm.launches
        m.decode(torch.zeros(batch, dtype=torch.int64, device="cuda"))
        assert (comm.launches - before == 2) == one
        torch.cuda.synchronize()
        comm.check()
