"""The list calls past the dispatcher: where a mode, a profiler or a subclass would see the operator, the operator is what runs,
and both ways give the same results, launch reports and errors."""
import pytest
import torch
from torch.utils._python_dispatch import TorchDispatchMode

from gpu_ipc_example_b200 import Communicator

pytestmark = pytest.mark.gpu


class Seen(TorchDispatchMode):
    def __init__(self):
        super().__init__()
        self.names = []

    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        self.names.append(str(func))
        return func(*args, **(kwargs or {}))


class Sub(torch.Tensor):
    pass


def _calls(comm, xs, ws, res, gam):
    W = comm.world
    yield "all_reduce", lambda: comm.all_reduce(xs, [torch.empty_like(t) for t in xs])
    yield "all_reduce in place", lambda: comm.all_reduce([t.clone() for t in xs])
    yield "all_gather", lambda: comm.all_gather(xs, [t.new_empty(W * t.shape[0], t.shape[1]) for t in xs])
    yield "reduce_scatter", lambda: comm.reduce_scatter(xs, [t.new_empty(t.shape[0] // W, t.shape[1]) for t in xs])
    yield "norm", lambda: sum(comm.allreduce_residual_rmsnorm(xs, res, gam), [])
    yield "linear", lambda: [t.clone() for t in sum(comm.linear_allreduce(xs, ws, res, gam), [])]
    yield "gather_linear", lambda: comm.allgather_linear(xs, ws)


@pytest.mark.parametrize("world", [2, 8])
def test_both_ways_agree(world):
    g = torch.Generator(device="cuda").manual_seed(world)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g).half()
    xs, ws = [rnd(16, 512) for _ in range(world)], [rnd(512, 512) for _ in range(world)]
    res, gam = [rnd(16, 512)] * world, [rnd(512)] * world
    with Communicator.virtual(world, 0, staging_bytes=64 << 20) as comm:
        for name, call in _calls(comm, xs, ws, res, gam):
            fast, info = call(), comm.last_info
            seen = Seen()
            with seen:
                slow = call()
            assert comm.last_info == info, name
            for a, b in zip(fast, slow):
                assert torch.equal(a, b), name
        subs = [t.as_subclass(Sub) for t in xs]
        for a, b in zip(comm.all_reduce(subs, [torch.empty_like(t) for t in xs]), comm.all_reduce(xs, [torch.empty_like(t) for t in xs])):
            assert torch.equal(a, b)
        with torch.profiler.profile() as prof:
            comm.all_reduce(xs, [torch.empty_like(t) for t in xs])
        assert any("b200ipc::all_reduce_lists" in e.name for e in prof.events())
        torch.cuda.synchronize()
        comm.check()


def test_errors_are_the_operators():
    with Communicator.virtual(2, 0, staging_bytes=16 << 20) as comm:
        a = [torch.zeros(64, device="cuda").half() for _ in range(2)]
        for ins, outs, kw in ((a, [torch.zeros(64, device="cuda").half(), torch.zeros(32, device="cuda").half()], {}),  # sizes
                              (a, a, dict(algo="no such algorithm")), ([t.float() for t in a], None, {}), ([t.cpu() for t in a], None, {}),
                              (a, None, dict(ctas="one")), ([a[0], None], None, {})):
            errors = []
            for listen in (False, True):
                with pytest.raises((RuntimeError, TypeError, ValueError)) as e:
                    if listen:
                        with Seen():
                            comm.all_reduce(ins, outs, **kw)
                    else:
                        comm.all_reduce(ins, outs, **kw)
                errors.append((e.type, str(e.value).split("\n")[0]))
            assert errors[0] == errors[1]
        out = comm.all_reduce(a, None)  # the communicator still works
        assert torch.equal(out[0], a[0])


@pytest.mark.parametrize("key", ["AutogradCUDA", "CUDA"])
def test_a_kernel_of_the_program_is_what_runs(key):
    """A kernel that a program registers for an operator, an autograd one say, is not passed by."""
    xs = [torch.ones(2, 64, device="cuda").half() for _ in range(2)]
    seen = []

    def mine(xs, residuals, gammas, eps, comm):
        seen.append(eps)
        return [t.clone() for t in xs + residuals], [0] * 9

    with Communicator.virtual(2, 0, staging_bytes=16 << 20) as comm:
        call = lambda: comm.allreduce_residual_rmsnorm(xs, xs, [x[0] for x in xs], 0.25)
        plain = call()
        lib = torch.library.Library("b200ipc", "IMPL")
        try:
            lib.impl("ar_rmsnorm_lists", mine, key)
            out, _ = call()
            assert seen == [0.25] and torch.equal(out[0], xs[0])
        finally:
            lib._destroy()
        for a, b in zip(sum(call(), []), sum(plain, [])):
            assert torch.equal(a, b)
        assert seen == [0.25]


def test_the_direct_route_is_taken():
    """The fast calls answer for plain lists, and for nothing that somebody would see."""
    W = 2
    with Communicator.virtual(W, 0, staging_bytes=32 << 20) as comm:
        h, ones = comm._h, lambda *s: [torch.ones(*s, device="cuda").half() for _ in range(W)]
        xs, ws, res, gam = ones(16, 512), ones(512, 512), ones(16, 512), ones(512)
        calls = [lambda x: comm._fast_all_reduce(x, ones(16, 512), h, "auto", 0, 0, 0), lambda x: comm._fast_all_gather(x, ones(32, 512), h, "auto", 0, 0, 0),
                 lambda x: comm._fast_reduce_scatter(x, ones(8, 512), h, "auto", 0, 0), lambda x: comm._fast_ar_rmsnorm(x, res, gam, 1e-5, h),
                 lambda x: comm._fast_local_gemm_ar(x, ws, res, gam, ones(16, 512), ones(16, 512), 1e-5, True, h),
                 lambda x: comm._fast_local_ag_gemm(x, ws, ones(32, 512), h)]
        for call in calls:
            assert call(xs) is not None
            assert call([t.as_subclass(Sub) for t in xs]) is None
            with Seen():
                assert call(xs) is None
            with torch.profiler.profile():
                assert call(xs) is None
            assert call([xs[0], None]) is None and call(tuple(xs)) is None and call([t.cpu() for t in xs]) is None
        torch.cuda.synchronize()
        comm.check()
