"""The native operator layer (csrc/ops_ext.cpp) against the Python classes of ops.py: same kernels, so values and
words agree bit for bit and gradients to the order of their atomics."""
import pytest
import torch

from gpu_util import rel

pytestmark = pytest.mark.gpu
INF = float("inf")


def both(fn):
    """(native, Python) results of fn()."""
    from sortnet_b200 import ops
    native = fn()
    keep, ops._native = ops._native, lambda w: False
    try:
        return native, fn()
    finally:
        ops._native = keep


def operands(B, CI, CO, HW=1, groups=1, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.rand(B, CI, HW, device="cuda", generator=g, requires_grad=True)
    w = torch.randn(CO, CI // groups, device="cuda", generator=g, requires_grad=True)
    return x, w, torch.randn(B, CO, HW, device="cuda", generator=g)


def compare(a, b):
    """1e-5 as for all gradients here: a finite p sums its outputs in run-dependent order (a few 2^-24), and the
    backward raises ratios of them to the power p - 1 (30 at most)."""
    assert len(a) == len(b)
    for u, v in zip(a, b):
        assert (u is None) == (v is None)
        if u is not None:
            assert u.shape == v.shape and rel(u.detach().cpu().numpy(), v.detach().cpu().numpy()) < 1e-5


@pytest.mark.parametrize("p", [INF, 1.0, 8.0, 31.6])
@pytest.mark.parametrize("shape", [(9, 97, 33, 1, 1), (40, 12, 18, 4, 3), (70, 1024, 400, 1, 1)])
@pytest.mark.parametrize("needs", ["xw", "x", "w", ""])
def test_distance(p, shape, needs):
    from sortnet_b200 import ops
    B, CI, CO, HW, G = shape
    x, w, gy = operands(B, CI, CO, HW, G)
    x.requires_grad_("x" in needs), w.requires_grad_("w" in needs)

    def run():
        y = ops.norm_dist(x, w, p, G)
        wanted = [t for t in (x, w) if t.requires_grad]
        return [y] + (list(torch.autograd.grad(y, wanted, gy)) if wanted else [])
    compare(*both(run))


@pytest.mark.parametrize("p", [INF, 3.0])
@pytest.mark.parametrize("ascending", [False, True])
def test_masked_distance(p, ascending):
    from sortnet_b200 import ops
    from sortnet_b200.layers import sample_mask
    x, w, _ = operands(70, 300, 200)
    ci, co = sample_mask(3, 1, 300, 0.8, "cuda"), sample_mask(3, 1, 200, 0.9, "cuda")
    x = x.detach()[:, :ci.size(2)].contiguous().requires_grad_()
    gy = torch.randn(70, co.size(2), 1, device="cuda")
    op = ops.norm_dist_dropout_ascending if ascending else ops.norm_dist_dropout

    def run():
        y = op(x, w, ci, co, p)
        return [y, *torch.autograd.grad(y, (x, w), gy)]
    compare(*both(run))


@pytest.mark.parametrize("shape", [(40, 30, 20, 1, 1), (33, 12, 18, 4, 3)])
def test_sort_neuron_and_bounds(shape):
    from sortnet_b200 import ops
    B, CI, CO, HW, G = shape
    x, w, gy = operands(B, CI, CO, HW, G)
    lo, hi = (x.detach() - 0.1).requires_grad_(), (x.detach() + 0.1).requires_grad_()

    def run():
        y = ops.sort_neuron(x, w, G, q=0.8, truncate=4)
        yl, yu = ops.bound_inf_dist(lo, hi, w, G)
        out = [y, yl, yu, *torch.autograd.grad(y, (x, w), gy)]
        out += torch.autograd.grad((yl, yu), (lo, hi, w), (gy, 2 * gy), retain_graph=True)
        out += torch.autograd.grad(yu, (lo, hi), gy)            # only one of the two outputs is used
        with torch.no_grad():
            return out + [*ops.bound_sort_neuron(lo, hi, w, G, q=0.8, truncate=4), ops.sort_neuron(x, w, G, q=0.8)]
    compare(*both(run))


def test_errors_and_counter():
    from sortnet_b200 import norm_dist_cuda as C, ops
    x, w, _ = operands(8, 16, 5)
    C.reset_counters()
    y = ops.norm_dist(x, w, INF)
    y.sum().backward()
    assert C.launch_count >= 2
    with pytest.raises(RuntimeError):
        ops.norm_dist(x.detach().cpu(), w, INF)
    with pytest.raises(RuntimeError):
        ops.norm_dist(x.double(), w, INF)
    with pytest.raises(RuntimeError):
        ops.norm_dist(x.transpose(0, 1).transpose(0, 1)[::2], w, INF)   # not contiguous
    with pytest.raises(AssertionError):
        ops.norm_dist(x, w[:, :8], INF)


@pytest.mark.filterwarnings("ignore::torch.jit.TracerWarning")
@pytest.mark.parametrize("grad", [False, True])
def test_traced_calls_replay(grad):
    """torch.jit.trace records the operators and replays them on other inputs."""
    from sortnet_b200 import layers, ops
    x, w, _ = operands(40, 12, 18)
    x2, w2, _ = operands(40, 12, 18, seed=1)
    for t in (x, w, x2, w2):
        t.requires_grad_(grad)
    calls = [lambda a, b: ops.norm_dist(a, b, INF), lambda a, b: ops.norm_dist(a, b, 3.0),
             lambda a, b: ops.sort_neuron(a, b, q=0.8, truncate=4), lambda a, b: ops.bound_inf_dist(a, a + 0.1, b)[1]]
    for f in calls:
        traced = torch.jit.trace(f, (x, w), check_trace=False)
        spoil = torch.full((40, 18, 1), 7.0, device="cuda")      # what an allocation that nobody fills finds
        del spoil
        assert torch.allclose(traced(x2, w2), f(x2, w2), rtol=1e-6)
    index = layers.sample_mask(3, 2, 9, 0.8, "cuda", count=6)
    other = layers.sample_mask(3, 2, 9, 0.8, "cuda", count=6)
    traced = torch.jit.trace(lambda i: layers._plane_index(i, 18, 4), (index,), check_trace=False)
    spoil = torch.full((3, 1, 48), 7, dtype=torch.int32, device="cuda")
    del spoil
    assert torch.equal(traced(other), layers._plane_index(other, 18, 4))


def test_dual_tensors_are_refused():
    """There is no forward-mode derivative; a result without a tangent would read as a zero one."""
    from torch.autograd import forward_ad
    from sortnet_b200 import ops
    x, w, _ = operands(40, 12, 18)
    x, w = x.detach(), w.detach()
    with forward_ad.dual_level():
        dual = forward_ad.make_dual(x, torch.ones_like(x))
        for call in (lambda: ops.norm_dist(dual, w, INF), lambda: ops.norm_dist(dual, w, 3.0),
                     lambda: ops.sort_neuron(dual, w, q=0.8, truncate=4), lambda: ops.bound_inf_dist(dual, dual, w),
                     lambda: ops.norm_dist_dropout(dual, w, None, None, INF)):
            with pytest.raises(RuntimeError, match="jvp"):
                call()
    assert ops.norm_dist(x, w, INF).shape == (40, 18, 1)


def test_further_axes_of_size_one():
    """A 1 x 1 convolution's weight [CO, CI, 1, 1] and inputs [B, C, HW, 1]: gradients have the operands' shapes."""
    from sortnet_b200 import ops
    x, w, gy = operands(40, 12, 18, HW=4)
    x4, w4 = x.detach().unsqueeze(-1).requires_grad_(), w.detach()[..., None, None].requires_grad_()
    for call in (lambda a, b: ops.norm_dist(a, b, INF), lambda a, b: ops.norm_dist(a, b, 3.0),
                 lambda a, b: ops.bound_inf_dist(a, a + 0.1, b)[1]):
        def run(a=x4, b=w4):
            y = call(a, b)
            return [y, *torch.autograd.grad(y, (a, b), gy)]
        compare(*both(run))
        compare([t.reshape(-1) for t in run()], [t.reshape(-1) for t in run(x, w)])


@pytest.mark.parametrize("grad", [False, True])
def test_status_codes_arrive_as_the_library_error(grad):
    from sortnet_b200 import _lib, ops
    x, w, _ = operands(8, 40, 5)
    x.requires_grad_(grad), w.requires_grad_(grad)
    for got in both_errors(lambda: ops.sort_neuron(x, w, q=0.8, truncate=30)):      # more values than the kernels take
        assert type(got) is _lib.SortnetB200Error and "status 3" in str(got)


def both_errors(fn):
    def caught():
        with pytest.raises(Exception) as info:
            fn()
        return info.value
    return both(caught)


def test_launch_count_is_what_the_device_ran():
    """snb_launch_count against the profiler's list, over entry points of every kind."""
    from torch.profiler import ProfilerActivity, profile
    from sortnet_b200 import layers, norm_dist_cuda as C, ops
    from sortnet_b200.optim import FlatAdamW
    x, w, gy = operands(70, 1024, 1000)
    small, ws, gs = operands(9, 40, 20)
    model = layers.SortMLPModel(depth=4, width=700, input_dim=(3, 17, 17), num_classes=10, dropout=0.8).cuda().train()
    images, labels = torch.rand(70, 3, 17, 17, device="cuda"), torch.randint(0, 10, (70,), device="cuda")
    opt = FlatAdamW(model)

    def work():
        for a, b, g in ((x, w, gy), (small, ws, gs)):
            for p in (INF, 3.0, 60.0):
                torch.autograd.grad(ops.norm_dist(a, b, p), (a, b), g)
            torch.autograd.grad(ops.sort_neuron(a, b, q=0.8), (a, b), g)
            torch.autograd.grad(ops.bound_inf_dist(a, a, b)[0], (a, b), g)
            ops.bound_sort_neuron(a.detach(), a.detach(), b.detach(), q=0.8)
        for p in (INF, 3.0):
            model.set_p(p)
            model.mixture_loss(images, labels, 0.05).backward()
            opt.step()
        model.set_p(INF)
        with torch.no_grad():
            model.eval()(images, labels, 0.02, up=1.0, down=0.0)
            model.train()

    work()
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        C.reset_counters()
        work()
        torch.cuda.synchronize()
        counted = C.launch_count
    ours = [e.name for e in prof.events() if e.device_type.name == "CUDA" and "snb::" in e.name]
    assert len(ours) > 60 and counted == len(ours), (counted, len(ours))
