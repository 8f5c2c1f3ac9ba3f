"""Whole-net calls (csrc/mlp.cu) against the same net taken layer by layer: the forward is the same arithmetic in the
same order (bit-identical), gradients are fp32 sums in another order (1e-5 of the largest entry, as elsewhere)."""
import pytest
import torch

from gpu_util import rel

pytestmark = pytest.mark.gpu


def nets(depth, width, dims, classes, keep, **kw):
    from sortnet_b200.layers import SortMLPModel
    torch.manual_seed(1)
    a = SortMLPModel(depth=depth, width=width, input_dim=dims, num_classes=classes, dropout=keep, **kw).cuda()
    b = SortMLPModel(depth=depth, width=width, input_dim=dims, num_classes=classes, dropout=keep, **kw).cuda()
    b.load_state_dict(a.state_dict())
    return a, b


def layer_by_layer(fn):
    from sortnet_b200 import layers
    layers.FUSED_LAYERS = False
    try:
        return fn()
    finally:
        layers.FUSED_LAYERS = True


# ragged rows and widths, one and several sub-batches, more than 16 of them, odd class counts
CASES = [(70, 4, 700, (3, 17, 17), 10, 0.8), (33, 5, 1280, (1, 28, 28), 200, 0.9), (300, 4, 515, (3, 15, 15), 7, 1.0),
         (545, 4, 385, (1, 20, 20), 10, 0.7), (32, 4, 1024, (3, 32, 32), 10, 0.5)]


@pytest.mark.parametrize("B,depth,width,dims,classes,keep", CASES)
@pytest.mark.parametrize("flat", [False, True])
def test_training_pass(B, depth, width, dims, classes, keep, flat):
    """flat: activations hardly differ from the weights' spread, so that outputs are left to the dense kernel."""
    a, b = nets(depth, width, dims, classes, keep, std=0.02 if flat else 1.0)
    g = torch.Generator(device="cuda").manual_seed(3)
    x = torch.rand(B, *dims, device="cuda", generator=g)
    t = torch.randint(0, classes, (B,), device="cuda", generator=g)
    from sortnet_b200 import norm_dist_cuda as C
    plan = a._plan(None)
    assert plan.applies(B)
    out = []
    for net, run in ((a, lambda f: f()), (b, layer_by_layer)):
        net.train()
        xi = x.clone().requires_grad_()
        torch.manual_seed(7)
        loss = run(lambda: net.mixture_loss(xi, t, 0.05))
        run(lambda: (2 * loss).backward())
        out.append([loss.detach(), xi.grad] + [p.grad for p in net.parameters()])
        out[-1] += [l.mean_shift.running_mean for l in net.fc_dist[:-1]]
    n = len(list(a.parameters()))
    assert abs(float(out[0][0]) - float(out[1][0])) <= 2e-6 * max(1.0, abs(float(out[1][0])))
    for u, v in zip(out[0][1:2 + n], out[1][1:2 + n]):
        assert rel(u.cpu().numpy(), v.cpu().numpy()) < 1e-5
    for u, v in zip(out[0][2 + n:], out[1][2 + n:]):
        assert torch.equal(u, v)


def test_training_pass_with_sinks_and_frozen_layers():
    from sortnet_b200.optim import FlatAdamW
    a, b = nets(4, 700, (3, 17, 17), 10, 0.8)
    for net in (a, b):
        net.fc_dist[0].weight.requires_grad_(False)
        net.fc_dist[2].weight.requires_grad_(False)
    x = torch.rand(70, 3, 17, 17, device="cuda")
    t = torch.randint(0, 10, (70,), device="cuda")
    opt = FlatAdamW(a)
    for k in range(2):                      # the second backward of a step adds
        torch.manual_seed(k)
        a.mixture_loss(x, t, 0.05).backward()
        torch.manual_seed(k)
        layer_by_layer(lambda: b.mixture_loss(x, t, 0.05).backward())
    opt.gather_grads()
    for p, q in zip(a.parameters(), b.parameters()):
        if p.requires_grad:
            assert rel(p.grad_sink.cpu().numpy(), q.grad.cpu().numpy()) < 1e-5


@pytest.mark.parametrize("B,depth,width,dims,classes,keep", CASES)
@pytest.mark.parametrize("flat", [False, True])
def test_evaluation_pass(B, depth, width, dims, classes, keep, flat):
    a, _ = nets(depth, width, dims, classes, keep, std=0.02 if flat else 1.0)
    x = torch.rand(B, *dims, device="cuda")
    t = torch.randint(0, classes, (B,), device="cuda")
    from sortnet_b200.layers import update_running_means
    update_running_means(a, [x])
    a.eval()
    assert a._plan(None).applies(B)
    pixels = x.view(B, -1).size(1)
    box = (torch.rand(pixels, device="cuda") * 0.1 + 0.9, torch.rand(pixels, device="cuda") * 0.1)
    with torch.no_grad():
        for run in (lambda: a(x), lambda: a(x, t, 0.02), lambda: a(x, t, 0.02, up=1.0, down=0.0),
                    lambda: a(x, t, 0.02, up=box[0], down=box[1]), lambda: a.certified_margin(x, t, 0.02, 1.0, 0.0),
                    lambda: a.certified_margin(x, t, 0.02, 1.0, 0.0, sort_eval=False)):
            got, want = run(), layer_by_layer(run)
            for u, v in zip(got if isinstance(got, tuple) else (got,), want if isinstance(want, tuple) else (want,)):
                assert torch.equal(u, v)


@pytest.mark.parametrize("flat", [False, True])
def test_weights_written_right_before_a_pass(flat):
    """The kernels of a pass may start while the ones before them end, under capture as well: what is written to the weights and
    to the input ahead of a pass is seen by it, and replays follow one another without waiting."""
    a, b = nets(4, 700, (3, 17, 17), 10, 1.0, std=0.02 if flat else 1.0)
    a.eval(), b.eval()
    x = torch.rand(70, 3, 17, 17, device="cuda")
    t = torch.randint(0, 10, (70,), device="cuda")

    def step(net, to):
        for l in net.fc_dist:
            l.weight.mul_(1.01)
        to.mul_(0.99)
        out = net(to, t, 0.02, up=1.0, down=0.0)
        return out if isinstance(out, tuple) else (out,)

    with torch.no_grad():
        u, v = x.clone(), x.clone()
        assert a._plan(None).applies(70)
        got = [step(a, u) for _ in range(3)]
        want = [layer_by_layer(lambda: step(b, v)) for _ in range(3)]
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            last = step(a, u)
        for _ in range(3):
            graph.replay()
            got.append([o.clone() for o in last])
            want.append(layer_by_layer(lambda: step(b, v)))
        for p, q in zip(got, want):
            assert len(p) == len(q) and all(torch.equal(u, v) for u, v in zip(p, q))


@pytest.mark.parametrize("what", ["forward", "backward", "lists"])
def test_other_threads_run_while_a_pass_is_issued(what):
    """A call that waits for room in the launch queue does not hold the interpreter lock."""
    import threading
    import time
    from sortnet_b200 import norm_dist_cuda as C
    net, _ = nets(4, 700, (3, 17, 17), 10, 0.8)
    x, t = torch.rand(70, 867, device="cuda"), torch.randint(0, 10, (70,), device="cuda")
    plan = net._plan(net.draw_masks(70, x.device))
    one, grads = torch.ones((), device="cuda"), [torch.empty_like(w) for w in plan.weights]
    _, saved = C.mlp_train_forward(plan, x, t, 0.05, 1.0, 0.1, 1.0)
    uniform, seeds = torch.rand(64), torch.zeros(1, dtype=torch.int64)
    call = {"forward": lambda: C.mlp_train_forward(plan, x, t, 0.05, 1.0, 0.1, 1.0),
            "backward": lambda: C.mlp_train_backward(plan, 70, one, saved, grads, None, None),
            "lists": lambda: C.draw_lists(uniform, seeds, [64], [0.5], 3, x.device)}[what]
    call()
    torch.cuda.synchronize()
    ticks, end = [], threading.Event()

    def tick():
        while not end.is_set():
            ticks.append(time.perf_counter())
            time.sleep(0.001)

    thread = threading.Thread(target=tick)
    thread.start()
    try:
        torch.cuda._sleep(10 ** 9)                           # about half a second, behind which the launches pile up
        slept = torch.cuda.Event()
        slept.record()
        began, ended = 0.0, 0.0
        while not slept.query():
            t0 = time.perf_counter()
            call()
            t1 = time.perf_counter()
            if t1 - t0 > ended - began:
                began, ended = t0, t1
    finally:
        end.set()
        thread.join()
    assert ended - began > 0.05, "no call had to wait"
    assert sum(began < s < ended for s in ticks) > 100 * (ended - began)


@pytest.mark.parametrize("flat", [False, True])
def test_training_pass_of_many_sub_batches(flat):
    """More sub-batches than the mean shift holds the sums of in shared memory (64).  A gradient entry is a sum over up to 2085 rows:
    in fp32 2084 * 2^-24 = 1.2e-4 of the magnitudes at worst, which is the bar.  Against 64 bits the layers' atomics are off by up
    to 2.5e-5 of the largest entry at this size, the whole pass by 1.5e-6."""
    a, b = nets(4, 130, (1, 12, 12), 10, 0.8, std=0.02 if flat else 1.0)
    x = torch.rand(2085, 144, device="cuda")
    t = torch.randint(0, 10, (2085,), device="cuda")
    masks = a.draw_masks(2085, x.device)
    assert a._plan(masks).applies(2085)
    out = []
    for net, run in ((a, lambda f: f()), (b, layer_by_layer)):
        at = x.clone().requires_grad_()
        loss = run(lambda: net.mixture_loss(at, t, 0.05, masks=masks))
        grads = run(lambda: torch.autograd.grad(loss, [at, *net.parameters()]))
        out.append((loss, grads, [l.mean_shift.running_mean for l in net.fc_dist[:-1]]))
    (loss, grads, means), (loss_b, grads_b, means_b) = out
    assert abs(float(loss) - float(loss_b)) <= 2e-6 * max(1.0, abs(float(loss_b)))
    assert all(rel(p.cpu().numpy(), q.cpu().numpy()) < 1.2e-4 for p, q in zip(grads, grads_b))
    assert all(torch.equal(p, q) for p, q in zip(means, means_b))


@pytest.mark.parametrize("what", ["train", "sort"])
def test_passes_with_new_weights_follow_one_another(what):
    """The same for training passes with masks and for sort neurons: the kernels of a pass start while those before them end, and so
    do a pass and its backward.  Values bit-identical, gradients 1e-5 of the largest entry."""
    a, b = nets(4, 700, (3, 17, 17), 10, 0.8)
    x = torch.rand(70, 867, device="cuda")
    t = torch.randint(0, 10, (70,), device="cuda")
    masks = a.draw_masks(70, x.device)
    if what == "sort":
        a.eval(), b.eval()
        assert a._plan(None, sort_eval=True).applies(70)
    else:
        assert a._plan(masks).applies(70)

    def step(net, to):
        with torch.no_grad():
            for l in net.fc_dist:
                l.weight.mul_(1.01)
            to.mul_(0.99)
            if what == "sort":
                return list(net(to, t, 0.02, up=1.0, down=0.0)), []
        at = to.detach().requires_grad_()
        loss = net.mixture_loss(at, t, 0.05, masks=masks)
        grads = torch.autograd.grad(loss, [at, *net.parameters()])
        return [l.mean_shift.running_mean.clone() for l in net.fc_dist[:-1]], [loss.detach(), *grads]

    u, v = x.clone(), x.clone()
    got = [step(a, u) for _ in range(3)]
    want = [layer_by_layer(lambda: step(b, v)) for _ in range(3)]
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        got.append(step(a, u))
    torch.cuda.current_stream().wait_stream(stream)
    want.append(layer_by_layer(lambda: step(b, v)))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        last = step(a, u)
    for _ in range(4):
        graph.replay()
        got.append([[o.clone() for o in part] for part in last])
        want.append(layer_by_layer(lambda: step(b, v)))
    for (same, near), (same_b, near_b) in zip(got, want):
        assert all(torch.equal(p, q) for p, q in zip(same, same_b)) and len(same) == len(same_b)
        assert all(rel(p.cpu().numpy(), q.cpu().numpy()) < 1e-5 for p, q in zip(near, near_b)) and len(near) == len(near_b)
