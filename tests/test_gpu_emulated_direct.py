"""Collectives of an emulated world on the callers' own buffers (no staging), where they can go wrong: counts that do
not fill a vector, shards that start anywhere in a vector, grids of one and of many CTAs, in-place forms, buffers that
overlap.  Sums are compared with fp32 sums; one rounding to fp16 is at most 2^-11 of the value."""
import pytest
import torch

from gpu_ipc_example_b200 import Communicator

pytestmark = pytest.mark.gpu


def _inputs(world, n, dtype=torch.float16, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return [torch.randn(n, device="cuda", generator=g).to(dtype) for _ in range(world)]


def _close(got, want):
    eps = 2.0 ** -11 if got.dtype == torch.float16 else 2.0 ** -8
    torch.testing.assert_close(got.float(), want, atol=1e-6, rtol=1.01 * eps)


@pytest.fixture(scope="module", params=[2, 4, 8])
def comm(request):
    with Communicator.virtual(request.param, 0, staging_bytes=48 << 20) as c:
        yield c


@pytest.mark.parametrize("n", [1, 7, 8, 63, 65, 4096 * 8 + 5, 512 * 8 * 8, 1234567])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_all_reduce(comm, n, dtype):
    xs = _inputs(comm.world, n, dtype)
    want = torch.stack([x.float() for x in xs]).sum(0)
    outs = [torch.full_like(x, 9) for x in xs]
    comm.all_reduce(xs, outs)
    assert comm.last_info.sched == "bulk" and not comm.last_info.staged
    comm.all_reduce(xs)  # in place
    torch.cuda.synchronize()
    comm.check()
    for x, o in zip(xs, outs):
        _close(o, want)
        assert torch.equal(x, o)


@pytest.mark.parametrize("n", [2, 4, 6, 8, 12, 22, 4096, 4098, 70002, 70006, 262144 + 2])
def test_all_gather(comm, n):
    xs = _inputs(comm.world, n, seed=1)
    want = torch.cat(xs)
    outs = [torch.zeros(comm.world * n + 16, device="cuda", dtype=torch.float16) for _ in xs]
    got = [o[:comm.world * n] for o in outs]
    comm.all_gather(xs, got)
    assert comm.last_info.sched == "bulk" and not comm.last_info.staged
    torch.cuda.synchronize()
    comm.check()
    for o, g in zip(outs, got):
        assert torch.equal(g, want) and not bool(o[comm.world * n:].any())
    if n % 8 == 0:  # in place: every rank's input is its part of the output
        parts = [g[r * n:(r + 1) * n] for r, g in enumerate(got)]
        for r, p in enumerate(parts):
            p.copy_(xs[r] + 1)
        comm.all_gather(parts, got)
        torch.cuda.synchronize()
        comm.check()
        assert all(torch.equal(g, want + 1) for g in got)


@pytest.mark.parametrize("slice_", [1, 3, 8, 17, 4096, 4099, 65536 + 6, 100001])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_reduce_scatter(comm, slice_, dtype):
    xs = _inputs(comm.world, comm.world * slice_, dtype, seed=2)
    want = torch.stack([x.float() for x in xs]).sum(0)
    outs = comm.reduce_scatter(xs)
    assert comm.last_info.sched == "bulk" and not comm.last_info.staged
    torch.cuda.synchronize()
    comm.check()
    for r, o in enumerate(outs):
        _close(o, want[r * slice_:(r + 1) * slice_])


def test_overlapping_buffers_take_another_kernel(comm):
    """An output that lies inside an input, but not where the in-place form has it.  Above what the flag-in-data kernels take
    (8 MiB), so the inputs are staged."""
    n = 8 * 600000
    xs = _inputs(comm.world, n, seed=3)
    want = torch.stack([x.float() for x in xs]).sum(0)
    outs = [x[:n // comm.world] for x in xs]
    comm.reduce_scatter(xs, outs)
    assert comm.last_info.staged
    torch.cuda.synchronize()
    comm.check()
    for r, o in enumerate(outs):
        _close(o, want[r * (n // comm.world):(r + 1) * (n // comm.world)])


@pytest.mark.parametrize("n", [8, 4096 * 8 + 8, 1234568])
def test_by_name_it_is_the_kernel_with_the_barrier(comm, n):
    """What one process per GPU runs: staged from plain buffers, zero-copy on the symmetric heap."""
    w = comm.world
    xs = _inputs(w, n, seed=6)
    want = torch.stack([x.float() for x in xs]).sum(0)
    outs = comm.all_reduce(xs, [torch.empty_like(x) for x in xs], "bulk")
    assert comm.last_info.staged
    gathered = comm.all_gather(xs, None, "allgather_bulk")
    assert comm.last_info.staged
    scattered = comm.reduce_scatter([x[:n // (8 * w) * 8 * w] for x in xs], None, "bulk") if n >= 8 * w else None
    if scattered:
        assert comm.last_info.staged
    sym = comm.empty([n // (8 * w) * 8 * w], torch.float16) if n >= 8 * w else None
    if sym:
        for s, x in zip(sym, xs):
            s.copy_(x[:s.numel()])
        barrier = comm.last_info.first_flag  # the number of its barrier: the direct kernel takes none
        comm.all_reduce(sym, None, "bulk")
        assert not comm.last_info.staged and comm.last_info.first_flag > barrier
    torch.cuda.synchronize()
    comm.check()
    for r in range(w):
        _close(outs[r], want)
        assert torch.equal(gathered[r], torch.cat(xs))
        if scattered:
            m = scattered[r].numel()
            _close(scattered[r], want[r * m:(r + 1) * m])
            _close(sym[r], want[:sym[r].numel()])
    comm.free_symmetric()


@pytest.mark.parametrize("nbytes", [8 << 10, (8 << 10) + 2, 64 << 10, (64 << 10) + 2, 512 << 10, (512 << 10) + 2, 4 << 20])
def test_auto_at_any_size(comm, nbytes):
    w, n = comm.world, nbytes // 2
    xs = _inputs(w, n, seed=4)
    want = torch.stack([x.float() for x in xs]).sum(0)
    outs = comm.all_reduce(xs, [torch.empty_like(x) for x in xs])
    gathered = comm.all_gather([x[:n // 2 * 2] for x in xs])
    scattered = comm.reduce_scatter([x[:n // w * w] for x in xs])
    torch.cuda.synchronize()
    comm.check()
    for r in range(w):
        _close(outs[r], want)
        assert torch.equal(gathered[r], torch.cat([x[:n // 2 * 2] for x in xs]))
        _close(scattered[r], want[:n // w * w][r * (n // w):(r + 1) * (n // w)])


@pytest.mark.parametrize("nbytes", [4 << 10, 96 << 10, 1 << 20, 12 << 20])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_auto_rounds_after_each_add_where_the_flag_asks_for_it(comm, nbytes, dtype):
    """Every element is a chain of adds in T.  The schedules take the ranks in rank order, from a rank of their choice."""
    w, n = comm.world, nbytes // 2
    xs = _inputs(w, n, dtype, seed=5)

    def chains(vs):
        for order in (vs, vs[::-1]):
            for r in range(w):
                s = order[r]
                for k in range(1, w):
                    s = s + order[(r + k) % w]
                yield s

    def is_chain(got, vs):
        ok = torch.zeros_like(got, dtype=torch.bool)
        for s in chains(vs):
            ok |= got == s
        return bool(ok.all())

    # two ranks have one add; for more, a sum in fp32 is seen
    assert is_chain(sum(x.float() for x in xs).to(dtype), xs) == (w == 2)
    outs = comm.all_reduce([x.clone() for x in xs], [torch.empty_like(x) for x in xs], flags=1)
    torch.cuda.synchronize()
    comm.check()
    assert all(torch.equal(o, outs[0]) for o in outs) and is_chain(outs[0], xs)
    if nbytes <= 8 << 20:  # up to here `auto` has a reduce-scatter that looks at the flag
        m = n // (2 * w) * 2 * w
        outs = comm.reduce_scatter([x[:m].clone() for x in xs], flags=1)
        torch.cuda.synchronize()
        comm.check()
        assert is_chain(torch.cat(outs), [x[:m] for x in xs])
