"""The GEMM of a process that drives every rank (linear + all-reduce, all-gather + linear), at the edges of its tiles, splits
and shards, against fp64 products.  fp32 sums of K products of N(0, 1) x N(0, 0.02) are off by less than K * 2^-24 * 0.02 * 4
(at most 2e-5 here), the one rounding to 16 bit by half a unit in the last place."""
import pytest
import torch

from gpu_ipc_example_b200 import Communicator

pytestmark = pytest.mark.gpu
HALF_ULP = {torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8}


def _rand(g, dtype, *shape, scale=1.0):
    return (torch.randn(*shape, device="cuda", generator=g) * scale).to(dtype)


def _close(got, want, dtype):
    torch.testing.assert_close(got.double(), want, atol=1e-4, rtol=1.01 * HALF_ULP[dtype])


# one row, the edges of the 32-row tile steps, several tiles of rows, K that does not fill a 64-column block, N that does
# not fill a 256-row tile of W, few blocks per K split, ranks that meet inside a stage
@pytest.mark.parametrize("world,M,K,N", [(1, 1, 64, 64), (1, 31, 72, 192), (1, 33, 3584, 1024), (1, 257, 1000, 320), (1, 2048, 448, 1152),
                                         (2, 16, 4096, 512), (2, 300, 200, 704), (4, 97, 8, 1024), (8, 5, 1032, 8192)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_linear(world, M, K, N, dtype):
    g = torch.Generator(device="cuda").manual_seed(M + K)
    xs = [_rand(g, dtype, M, K) for _ in range(world)]
    ws = [_rand(g, dtype, N, K, scale=0.02) for _ in range(world)]
    res = [_rand(g, dtype, M, N) for _ in range(world)]
    gam = [1 + _rand(g, dtype, N, scale=0.1) for _ in range(world)]
    y = sum(x.double() @ w.double().t() for x, w in zip(xs, ws))
    with Communicator.virtual(world, 0, staging_bytes=96 << 20) as comm:
        for o in comm.linear_allreduce(xs, ws):
            _close(o, y, dtype)
        for o, s, r in zip(*comm.linear_allreduce(xs, ws, res), res):
            _close(s, y + r.double(), dtype)
            assert torch.equal(o, s)
        outs, sums = comm.linear_allreduce(xs, ws, res, gam, 1e-5)
        for o, s, r, ga in zip(outs, sums, res, gam):
            _close(s, y + r.double(), dtype)
            want = s.double() * torch.rsqrt(s.double().pow(2).mean(-1, keepdim=True) + 1e-5) * ga.double()
            _close(o, want, dtype)
        norm_only, _ = comm.linear_allreduce(xs, ws, None, gam, 1e-5)  # the sum is normalised where it lies
        for o, ga in zip(norm_only, gam):
            want = y * torch.rsqrt(y.pow(2).mean(-1, keepdim=True) + 1e-5) * ga.double()
            # two roundings: the sum's and the result's, and the statistic is taken from the rounded sums
            torch.testing.assert_close(o.double(), want, atol=2e-3, rtol=3 * HALF_ULP[dtype])
        torch.cuda.synchronize()
        comm.check()


# all shards in one tile (with padding rows between them and without), the largest such tile, one tile per shard, several
@pytest.mark.parametrize("world,rows,K,N", [(1, 3, 512, 64), (2, 1, 520, 320), (2, 128, 64, 256), (2, 129, 256, 448), (4, 8, 1000, 1024),
                                            (4, 13, 192, 7168), (4, 65, 128, 64), (2, 600, 328, 512), (1, 4100, 136, 256), (8, 9, 96, 128)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_gather_linear(world, rows, K, N, dtype):
    g = torch.Generator(device="cuda").manual_seed(rows + K)
    xs = [_rand(g, dtype, rows, K) for _ in range(world)]
    ws = [_rand(g, dtype, N, K, scale=0.02) for _ in range(world)]
    full = torch.cat(xs).double()
    with Communicator.virtual(world, 0, staging_bytes=32 << 20) as comm:
        for o, w in zip(comm.allgather_linear(xs, ws), ws):
            _close(o, full @ w.double().t(), dtype)
        torch.cuda.synchronize()
        comm.check()


def test_what_the_kernel_does_not_take_still_runs():
    """Below 4096 rows an all-gather followed by the framework's matmul took any N and K, unaligned rows, weights of
    uneven heights, a vector, and a weight that wants a gradient; it still does."""
    g = torch.Generator(device="cuda").manual_seed(0)
    with Communicator.virtual(2, 0, staging_bytes=32 << 20) as comm:
        for K, N, off in ((128, 40, 0), (36, 64, 0), (128, 64, 1)):
            flat = [_rand(g, torch.float16, 8 * K + 8) for _ in range(2)]
            xs = [f[off:off + 8 * K].view(8, K) for f in flat]
            ws = [_rand(g, torch.float16, N, K, scale=0.02) for _ in range(2)]
            for o, w in zip(comm.allgather_linear(xs, ws), ws):
                torch.testing.assert_close(o.double(), torch.cat(xs).double() @ w.double().t(), atol=2e-3, rtol=2e-3)
        xs = [_rand(g, torch.float16, 8, 128) for _ in range(2)]
        for shapes in (((64, 128), (128, 128)), ((128,), (128,))):  # uneven heights, a vector
            ws = [_rand(g, torch.float16, *s, scale=0.02) for s in shapes]
            for o, w in zip(comm.allgather_linear(xs, ws), ws):
                torch.testing.assert_close(o.double(), torch.cat(xs).double() @ w.double().t(), atol=2e-3, rtol=2e-3)
        ws = [w.detach().requires_grad_() for w in (_rand(g, torch.float16, 64, 128), _rand(g, torch.float16, 64, 128))]
        outs = comm.allgather_linear([_rand(g, torch.float16, 8, 128) for _ in range(2)], ws)
        outs[1].float().sum().backward()
        assert ws[1].grad is not None


@pytest.mark.parametrize("world", [1, 2, 8])
@pytest.mark.parametrize("M", [1, 32, 40, 300])
def test_the_kernels_with_the_exchange(world, M):
    """fused=True: what runs with one process per GPU, on an emulated world.  Every rank's partial product is rounded to the
    element type before the sum."""
    g = torch.Generator(device="cuda").manual_seed(M)
    xs = [_rand(g, torch.float16, M, 320) for _ in range(world)]
    ws = [_rand(g, torch.float16, 1024, 320, scale=0.02) for _ in range(world)]
    res, gam = _rand(g, torch.float16, M, 1024), 1 + _rand(g, torch.float16, 1024, scale=0.1)
    with Communicator.virtual(world, 0, staging_bytes=96 << 20) as comm:
        for _ in range(2):
            comm.linear_allreduce(xs, ws, [res] * world, [gam] * world)  # the two forms take turns on one set of outputs
            outs, sums = comm.linear_allreduce(xs, ws, [res] * world, [gam] * world, fused=True)
            torch.cuda.synchronize()
            comm.check()
            y = sum((x.double() @ w.double().t()).half().double() for x, w in zip(xs, ws)) + res.double()
            for o, s in zip(outs, sums):
                torch.testing.assert_close(s.double(), y, atol=2e-3, rtol=2e-3)
                want = s.double() * torch.rsqrt(s.double().pow(2).mean(-1, keepdim=True) + 1e-5) * gam.double()
                torch.testing.assert_close(o.double(), want, atol=2e-3, rtol=2e-3)


def test_a_limit_on_ctas_is_kept():
    """A communicator that may use a few SMs only (the others belong to work on another stream) keeps the kernels that can be
    told so."""
    g = torch.Generator(device="cuda").manual_seed(0)
    with Communicator.virtual(2, 0, staging_bytes=64 << 20, max_ctas=8) as comm:
        xs = [_rand(g, torch.float16, 64, 512) for _ in range(2)]
        ws = [_rand(g, torch.float16, 1024, 512, scale=0.02) for _ in range(2)]
        res, gam = [_rand(g, torch.float16, 64, 1024)] * 2, [_rand(g, torch.float16, 1024)] * 2
        comm.linear_allreduce(xs, ws, res, gam)
        assert comm.last_info.ctas <= 8
        comm.allreduce_residual_rmsnorm(res, res, gam)
        assert comm.last_info.ctas <= 8 and comm.last_info.sched == "oneshot"
        outs = comm.allgather_linear(xs, ws)
        assert comm.last_info.ctas <= 8  # the all-gather's
        torch.cuda.synchronize()
        comm.check()
        torch.testing.assert_close(outs[0].double(), torch.cat(xs).double() @ ws[0].double().t(), atol=2e-3, rtol=2e-3)


@pytest.mark.parametrize("producer", ["strided", "norm"])
@pytest.mark.parametrize("call", ["linear_allreduce", "linear_allreduce packed", "linear_allreduce exchange", "linear", "allgather_linear"])
@pytest.mark.parametrize("world", [1, 2])
def test_weight_made_by_the_kernel_right_before(world, call, producer):
    """The kernels are launched while their predecessor may still run, so a weight that it writes must not be loaded before
    the wait for it: the copy of a strided weight inside the call, and a weight that is the output of a kernel which lets its
    dependents start before it stores.  The buffers come back from call to call with other values in them."""
    M, K, N = 16, 1024, 4096
    g = torch.Generator(device="cuda").manual_seed(0)
    with Communicator.virtual(world, 0, staging_bytes=96 << 20) as comm:
        for _ in range(10):
            xs = [_rand(g, torch.float16, M, K) for _ in range(world)]
            base = [_rand(g, torch.float16, N, K, scale=0.02) for _ in range(world)]
            gam = [_rand(g, torch.float16, K, scale=0.02) for _ in range(world)]
            ws = [b.t().contiguous().t() for b in base]  # [N, K], not contiguous
            torch.cuda.synchronize()
            if producer == "norm":
                ws = comm.allreduce_residual_rmsnorm(base, base, gam)[0]
            if call == "linear_allreduce":
                outs = comm.linear_allreduce(xs, ws)
            elif call == "linear_allreduce packed":
                outs = comm.linear_allreduce(xs, [comm.pack_weight(w) for w in ws])
            elif call == "linear_allreduce exchange":
                outs = comm.linear_allreduce(xs, ws, fused=True)
            elif call == "linear":
                outs = comm.linear(xs, ws)
            else:
                outs = comm.allgather_linear(xs, ws)
            torch.cuda.synchronize()
            comm.check()
            part = [x.double() @ w.double().t() for x, w in zip(xs, ws)]
            for i, o in enumerate(outs):
                want = torch.cat(xs).double() @ ws[i].double().t() if call == "allgather_linear" else part[i] if call == "linear" else sum(part)
                # one rounding per rank and one of the sum, of values of a few units
                torch.testing.assert_close(o.double(), want, atol=4e-3, rtol=2 * HALF_ULP[torch.float16])


@pytest.mark.parametrize("world", [3, 5, 6, 7])
def test_other_world_sizes_are_refused(world):
    """A communicator can be made for them, the kernels are for 1, 2, 4 and 8."""
    with Communicator.virtual(world, 0, staging_bytes=16 << 20) as comm:
        xs = [torch.zeros(8, 128, device="cuda").half() for _ in range(world)]
        ws = [torch.zeros(64, 128, device="cuda").half() for _ in range(world)]
        outs = [torch.zeros(8 * world, 64, device="cuda").half() for _ in range(world)]
        for call in (lambda: comm.allgather_linear(xs, ws), lambda: comm.linear_allreduce(xs, ws),
                     lambda: torch.ops.b200ipc.local_ag_gemm(xs, ws, outs, comm._h),
                     lambda: torch.ops.b200ipc.local_gemm_ar(xs, ws, [], [], [o[:8] for o in outs], [], 1e-5, False, comm._h)):
            with pytest.raises(RuntimeError, match="world size"):
                call()


@pytest.mark.parametrize("fused", [None, True])
def test_operands_of_the_epilogue_are_checked(fused):
    """A residual that would have to be broadcast, a gamma of another length, 32-bit ones: refused, not read out of range or as
    16-bit values.  Any shape with the right number of elements is taken, as before."""
    g = torch.Generator(device="cuda").manual_seed(0)
    M, K, N = 8, 128, 256
    with Communicator.virtual(2, 0, staging_bytes=16 << 20) as comm:
        xs, ws = [_rand(g, torch.float16, M, K) for _ in range(2)], [_rand(g, torch.float16, N, K, scale=0.02) for _ in range(2)]
        res, gam = _rand(g, torch.float16, M, N), _rand(g, torch.float16, N)
        for r, ga in ((res[0], gam), (res[:1], gam), (res.float(), gam), (res, gam[:64]), (res, gam.float())):
            for bad in (0, 1):  # either rank's
                rs, gs = [res, res], [gam, gam]
                rs[bad], gs[bad] = r.contiguous(), ga.contiguous()
                with pytest.raises(RuntimeError, match="must hold"):
                    comm.linear_allreduce(xs, ws, rs, gs, fused=fused)
        with pytest.raises(RuntimeError, match="dtype"):
            comm.linear_allreduce(xs, [ws[0], ws[1].bfloat16()], [res] * 2, [gam] * 2, fused=fused)
        want = comm.linear_allreduce(xs, ws, [res] * 2, [gam] * 2, fused=fused)[0][0].clone()
        got = comm.linear_allreduce(xs, ws, [res.view(2, M // 2, N)] * 2, [gam.view(1, N)] * 2, fused=fused)[0][0]
        torch.cuda.synchronize()
        comm.check()
        assert torch.equal(got, want)


@pytest.mark.parametrize("world,M", [(1, 16), (1, 300), (2, 16), (2, 300)])
def test_inputs_that_lie_where_the_outputs_go(world, M):
    """Outputs take turns on two sets of buffers.  A result that is used twice is the second time an input at the place that the
    call writes; so is a residual of which every rank holds one rank's copy."""
    g = torch.Generator(device="cuda").manual_seed(M)
    N = 1024
    ws = [[_rand(g, torch.float16, N, N, scale=0.02) for _ in range(world)] for _ in range(3)]
    with Communicator.virtual(world, 0, staging_bytes=64 << 20) as comm:
        a = comm.linear_allreduce([_rand(g, torch.float16, M, N) for _ in range(world)], ws[0])
        was = [t.clone() for t in a]
        comm.linear_allreduce(a, ws[1])
        c = comm.linear_allreduce(a, ws[2])
        assert c[0].data_ptr() == a[0].data_ptr()
        want = sum(t.double() @ w.double().t() for t, w in zip(was, ws[2]))
        for o in c:
            _close(o, want, torch.float16)
        xs = [_rand(g, torch.float16, M, N) for _ in range(world)]
        r = comm.linear_allreduce(xs, ws[0], [was[0]] * world)[1]
        r0 = r[0].clone()
        comm.linear_allreduce(xs, ws[1], r)
        s = comm.linear_allreduce(xs, ws[2], [r[0]] * world)[1]
        assert s[0].data_ptr() == r[0].data_ptr()
        want = sum(t.double() @ w.double().t() for t, w in zip(xs, ws[2])) + r0.double()
        for o in s:
            _close(o, want, torch.float16)
        torch.cuda.synchronize()
        comm.check()
