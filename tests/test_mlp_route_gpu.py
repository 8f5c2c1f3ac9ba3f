"""When the whole-net calls (csrc/mlp.cu) stand in for the layers: never where the layers would do something else."""
import pytest
import torch

from gpu_util import rel
from test_mlp_gpu import nets

pytestmark = pytest.mark.gpu


def by_layers(fn):
    """fn() without the whole-net calls: layer by layer, as at sizes where they do not apply."""
    from sortnet_b200 import norm_dist_cuda as C
    keep, C.MlpPlan.applies = C.MlpPlan.applies, lambda self, *a: False
    try:
        return fn()
    finally:
        C.MlpPlan.applies = keep


def batch(B=70, dims=(3, 17, 17), classes=10, seed=3):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.rand(B, *dims, device="cuda", generator=g), torch.randint(0, classes, (B,), device="cuda", generator=g)


def step(net, x, t, **kw):
    torch.manual_seed(7)
    loss = net.mixture_loss(x, t, 0.05, **kw)
    loss.backward()
    return loss.detach()


def same_step(a, b, x, t, **kw):
    """Loss, gradients and running means of a step with the whole-net calls allowed and without them."""
    la, lb = step(a, x, t, **kw), by_layers(lambda: step(b, x, t, **kw))
    assert abs(float(la) - float(lb)) <= 2e-6 * max(1.0, abs(float(lb)))
    for p, q in zip(a.parameters(), b.parameters()):
        assert (p.grad is None) == (q.grad is None)
        assert p.grad is None or rel(p.grad.cpu().numpy(), q.grad.cpu().numpy()) < 1e-5
    for u, v in zip(a.buffers(), b.buffers()):
        assert torch.equal(u, v)


@pytest.mark.parametrize("keep", [0.8, 1.0])
def test_layer_in_evaluation_mode_during_training(keep):
    """A layer with frozen statistics subtracts its running mean and leaves it alone, whatever the batch size."""
    a, b = nets(4, 700, (3, 17, 17), 10, keep)
    for net in (a, b):
        net.train()
        net.fc_dist[1].mean_shift.running_mean.fill_(2.0)
        net.fc_dist[1].eval()
    same_step(a, b, *batch())
    assert bool((a.fc_dist[1].mean_shift.running_mean == 2.0).all())


def test_model_in_training_mode_with_layers_in_evaluation_mode():
    """Sub-sampling follows the model's own flag: masks are drawn although every layer evaluates."""
    a, b = nets(4, 700, (3, 17, 17), 10, 0.8)
    x, _ = batch()
    for net in (a, b):
        net.requires_grad_(False).train()
        for l in net.fc_dist:
            l.eval()
    torch.manual_seed(7)
    got = a(x)
    torch.manual_seed(7)
    assert torch.equal(got, by_layers(lambda: b(x)))


def evaluating(keep=0.8, scalar=False):
    a, _ = nets(4, 700, (3, 17, 17), 10, keep, scalar=scalar)
    return a.eval()


def test_labels_out_of_range_give_nan_margins():
    """As the last row and inside: no other row's bounds are read for them."""
    a, (x, t) = evaluating(), batch()
    with torch.no_grad():
        score, margin = a(x, t, 0.02, up=1.0, down=0.0)
        for row, label in ((0, -1), (5, 10), (69, 2 ** 40), (31, -(2 ** 62))):
            t[row] = label
        s2, m2 = a(x, t, 0.02, up=1.0, down=0.0)
    bad = torch.tensor([0, 5, 31, 69], device="cuda")
    good = torch.ones(70, dtype=torch.bool, device="cuda").index_fill_(0, bad, False)
    assert torch.equal(score, s2) and torch.equal(margin[good], m2[good]) and bool(m2[bad].isnan().all())


def test_targets_of_another_kind():
    """Other types, devices, counts and shapes: what torch.gather makes of them, as at sizes where the layers run."""
    a, (x, t) = evaluating(), batch()

    def outcome(targets):
        try:
            return a(x, targets, 0.02, up=1.0, down=0.0)[1]
        except (RuntimeError, IndexError) as exc:
            return type(exc)
    with torch.no_grad():
        for other in (t.int(), t.cpu(), t[:60], t.view(-1, 1), t.repeat_interleave(2)[::2]):
            got, want = outcome(other), by_layers(lambda: outcome(other))
            assert got is want or rel(got.cpu().numpy(), want.cpu().numpy()) < 1e-6      # a quotient or a product by 1 / (2 eps)
    a.train()
    for bad in (t.int(), t[:60]):
        with pytest.raises(RuntimeError):
            a.mixture_loss(x, bad, 0.02)


@pytest.mark.parametrize("keep", [0.8, 1.0])
@pytest.mark.parametrize("limits", ["numbers", "pixels"])
@pytest.mark.parametrize("eps", ["row", "one", "zero-dim"])
def test_eps_as_a_tensor(keep, limits, eps):
    a, (x, t) = evaluating(keep), batch()
    eps = {"row": 0.05 * torch.rand(70, 1, device="cuda") + 0.01, "one": torch.full((1,), 0.02, device="cuda"),
           "zero-dim": torch.tensor(0.02)}[eps]
    box = (1.0, 0.0) if limits == "numbers" else (torch.ones(867, device="cuda"), torch.zeros(867, device="cuda"))
    with torch.no_grad():
        got, want = (run(lambda: a(x, t, eps, up=box[0], down=box[1])) for run in (lambda f: f(), by_layers))
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])


def test_masks_of_the_caller(monkeypatch):
    """Entries outside the layer keep nothing and are written nowhere; with index checks on they are refused, as
    lists in another order are; lists of another shape go to the layers, which refuse them."""
    from sortnet_b200 import norm_dist_cuda as C
    a, b = nets(4, 700, (3, 17, 17), 10, 0.8)
    x, t = batch()
    masks = a.draw_masks(70, "cuda")
    shorter = [m[..., :-1].contiguous() for m in masks]
    for m in masks:
        m[0, 0, -1], m[1, 0, -1], m[2, 0, -1] = 700, 2 ** 30, -1
    out = [net.mixture_loss(x, t, 0.05, masks=m).detach() for net, m in ((a, masks), (b, shorter))]
    assert torch.equal(*out)
    good = a.draw_masks(70, "cuda")
    monkeypatch.setattr(C, "DEBUG_INDEX_CHECKS", True)
    a.mixture_loss(x, t, 0.05, masks=good)
    for bad in (masks, [m.flip(-1).contiguous() for m in good]):
        with pytest.raises(RuntimeError):
            a.mixture_loss(x, t, 0.05, masks=bad)


def test_hooks_of_layers_are_called():
    a, (x, t) = nets(4, 700, (3, 17, 17), 10, 0.8)[0], batch()
    seen = []
    for k, l in enumerate(a.fc_dist):
        l.register_forward_hook(lambda m, i, o, k=k: seen.append(k))
    a.mixture_loss(x, t, 0.05).backward()
    a.eval()
    with torch.no_grad():
        a(x, t, 0.02, up=1.0, down=0.0)
        a.certified_margin(x, t, 0.02, 1.0, 0.0)
    assert seen == 3 * [0, 1, 2, 3]


def test_gradients_arrive_layer_by_layer_for_post_accumulate_hooks(monkeypatch):
    """What dist.GradientAllReduce overlaps its exchange with: when the hook of a layer fires, the backward of the layer
    before it has not been queued yet."""
    from sortnet_b200 import norm_dist_cuda as C
    a, b = nets(4, 700, (3, 17, 17), 10, 0.8)
    x, t = batch()
    log, call = [], C._layer_call
    monkeypatch.setattr(C, "_layer_call", lambda entry, *args: (log.append(entry), call(entry, *args)))
    for k, l in enumerate(a.fc_dist):
        l.weight.register_post_accumulate_grad_hook(lambda p, k=k: log.append(k))
    step(a, x, t)
    events = [e for e in log if not isinstance(e, str) or "backward" in e]
    assert events == [e for k in (3, 2, 1, 0) for e in ("snb_layer_backward_ws", k)]
    by_layers(lambda: step(b, x, t))
    for p, q in zip(a.parameters(), b.parameters()):
        assert rel(p.grad.cpu().numpy(), q.grad.cpu().numpy()) < 1e-5


def test_head_wider_than_shared_memory():
    """The backward's shared memory follows the layers' inputs; 60 000 classes are no more than 60 000 rows."""
    a, b = nets(4, 512, (1, 16, 16), 60000, 0.8)
    same_step(a, b, *batch(33, (1, 16, 16), 60000))
