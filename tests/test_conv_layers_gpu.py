"""NormDistConv (grouped, spatial) and the mean shift over [B, C, HW] on the GPU against fixtures
recorded from the reference's own NormDistConv / MeanShiftDropout layers (PyTorch branches)."""
import numpy as np
import pytest
import torch

from gpu_util import dev, rel

pytestmark = pytest.mark.gpu


def build_stack(g):
    from sortnet_b200.layers import NormDistConv
    p, q, G = float(g["p"]), float(g["q"]), int(g["G"])
    drop = None if q == 1.0 else q
    layers = [NormDistConv(4, 12, 3, stride=1, groups=G, bias=False, mean_shift=True, p=p),
              NormDistConv(12, 12, 1, groups=G, bias=True, mean_shift=True, dropout=drop, p=p),
              NormDistConv(12, 8, 1, groups=G, bias=True, mean_shift=False, dropout=drop, p=p)]
    for i, l in enumerate(layers):
        l.load_state_dict({k: torch.from_numpy(g["state0.%d.%s" % (i, k)]) for k in l.state_dict()})
        l.cuda()
    return layers


@pytest.mark.parametrize("name", ["conv_stack_masked_inf", "conv_stack_masked_p8", "conv_stack_plain_inf"])
def test_conv_stack_training_step(golden, name):
    g = golden(name)
    layers = build_stack(g)
    masked = "mask0" in g
    masks = [dev(g["mask0"], torch.int32), dev(g["mask1"], torch.int32)] if masked else [None, None]
    x = dev(g["x"]).requires_grad_()
    for l in layers:
        l.train()
    z = layers[0](x, mask_out=masks[0])
    z = layers[1](z[0], mask_in=masks[0], mask_out=masks[1])
    z = layers[2](z[0], mask_in=masks[1])
    y = z[0]
    tol = 1e-5
    assert rel(y.detach().cpu().numpy(), g["y"]) < tol
    y.backward(dev(g["gy"]))
    assert rel(x.grad.cpu().numpy(), g["gx"]) < tol
    for i, l in enumerate(layers):
        for k, prm in l.named_parameters():
            assert rel(prm.grad.cpu().numpy(), g["grad.%d.%s" % (i, k)]) < tol, (i, k)
        if l.mean_shift is not None:
            assert rel(l.mean_shift.running_mean.cpu().numpy(), g["state1.%d.mean_shift.running_mean" % i]) < tol


@pytest.mark.parametrize("name", ["conv_stack_masked_inf", "conv_stack_plain_inf"])
def test_conv_stack_evaluation(golden, name):
    g = golden(name)
    layers = build_stack(g)
    for i, l in enumerate(layers):
        if l.mean_shift is not None:
            l.mean_shift.running_mean.copy_(dev(g["state1.%d.mean_shift.running_mean" % i]))
        l.eval()
    x = dev(g["x"])
    with torch.no_grad():
        if "eval_lower" in g:
            z = (x, (x - 0.05).clamp(0, 1), (x + 0.05).clamp(0, 1))
            for l in layers:
                z = l(*z)
            assert rel(z[0].cpu().numpy(), g["eval_y"]) < 1e-6
            assert rel(z[1].cpu().numpy(), g["eval_lower"]) < 1e-6
            assert rel(z[2].cpu().numpy(), g["eval_upper"]) < 1e-6
            assert bool((z[1] <= z[0]).all()) and bool((z[0] <= z[2]).all())
        else:
            z = (x, None, None)
            for l in layers:
                z = l(*z, sort_eval=True)
            assert rel(z[0].cpu().numpy(), g["eval_y"]) < 1e-5
            # interval bounds of the sort neurons enclose the point value
            lo, up = (x - 0.02).clamp(0, 1), (x + 0.02).clamp(0, 1)
            zb = (x, lo, up)
            for l in layers:
                zb = l(*zb, sort_eval=True)
            assert bool((zb[1] <= zb[0] + 1e-5).all()) and bool((zb[0] <= zb[2] + 1e-5).all())


def test_mean_shift_plane_matches_per_channel_mean():
    from sortnet_b200.layers import MeanShiftDropout
    torch.manual_seed(0)
    m = MeanShiftDropout(6, affine=True).cuda()
    with torch.no_grad():
        m.bias.normal_()
    x = torch.randn(45, 6, 7, device="cuda", requires_grad=True)
    m.train()
    y, _, _ = m(x)
    mean = x.detach().mean(dim=(0, 2))
    want = x.detach() - mean.view(1, -1, 1) + m.bias.detach().view(1, -1, 1)
    assert rel(y.detach().cpu().numpy(), want.cpu().numpy()) < 1e-5
    assert rel(m.running_mean.cpu().numpy(), (0.1 * mean).cpu().numpy()) < 1e-5
    gy = torch.randn_like(y)
    y.backward(gy)
    assert rel(x.grad.cpu().numpy(), (gy - gy.mean(dim=(0, 2), keepdim=True)).cpu().numpy()) < 1e-5


@pytest.mark.parametrize("B,G,C,kept,hw", [(1, 1, 5, 5, 1), (33, 1, 9, 4, 4), (70, 3, 30, 7, 9)])
def test_native_glue_is_the_python_one(B, G, C, kept, hw):
    """Mean shift and per-channel add in native code: values and gradients of the Python functions, second order of the add included."""
    from sortnet_b200 import layers, _lib
    gen = torch.Generator(device="cuda").manual_seed(B)
    S, per = (B + 31) // 32, C // G
    index = None if kept == per else torch.rand(S, G, per, device="cuda", generator=gen).argsort(-1)[..., :kept].sort(-1)[0].int().contiguous()
    x = torch.randn(hw, G * kept, B, device="cuda", generator=gen).permute(2, 1, 0).requires_grad_()       # not contiguous
    v = torch.randn(C, device="cuda", generator=gen).requires_grad_()
    g = torch.randn(B, G * kept, hw, device="cuda", generator=gen)
    got = []
    for shift, add in ((_lib.ops().mean_shift, _lib.ops().add_per_channel), (layers._MeanShiftPlaneF.apply, layers._PlaneAddF.apply)):
        run = torch.ones(C, device="cuda")
        y, mean = shift(x, index, run, 0.1)
        z = add(y, v, index)
        gx, gv = torch.autograd.grad(z, (x, v), g)
        second, = torch.autograd.grad(torch.autograd.grad((add(x, v, index) ** 3).sum(), v, create_graph=True)[0].sum(), v)
        assert not mean.requires_grad
        got.append((y, mean, run, z, gx, gv, second))
    assert all(torch.equal(a, b) for a, b in zip(*got))
    rows = torch.arange(B, device="cuda") // 32
    chan = torch.arange(C, device="cuda").expand(B, C) if index is None else layers._global_index(index, C)[rows]
    terms = 6 * (x + v[chan].unsqueeze(-1)).double()
    want, size = (torch.zeros(C, dtype=torch.float64, device="cuda").index_add_(0, chan.reshape(-1), t.sum(-1).reshape(-1)) for t in (terms, terms.abs()))
    assert ((got[0][-1].double() - want).abs() <= 2 ** -20 * size).all()          # a dozen roundings of 2^-24 per term, sums in 64 bits


@pytest.mark.parametrize("S,G,channel,q", [(1, 1, 7, 0.5), (4, 1, 1024, 0.75), (3, 3, 341, 0.9), (2, 1, 40, 0.0)])
def test_sample_mask_draws_what_it_did(S, G, channel, q):
    """The lists of the seeds and counts that the host generator gives, one kernel call as before."""
    from sortnet_b200 import layers, norm_dist_cuda as C
    torch.manual_seed(7)
    got, after = layers.sample_mask(S, G, channel, q, "cuda"), torch.rand(1)
    torch.manual_seed(7)
    count = min(max(int((torch.rand(channel) < q).sum()), 1), channel)
    seed = int(torch.randint(0, 2 ** 62, (1,)))
    want = torch.empty(S, G, count, dtype=torch.int32, device="cuda")
    C.sample_mask_into(want, channel, seed)
    assert torch.equal(got, want) and got.is_contiguous() and torch.equal(after, torch.rand(1))


@pytest.mark.parametrize("G,repeat", [(1, False), (1, True), (3, False), (3, True)])
def test_bias_gradient_of_lists_in_any_order(G, repeat):
    """Output masks that do not ascend and, with `repeat`, name a channel twice: values, bias, input and weight gradients of a layer without mean shift against
    the same in PyTorch's indexing and 64 bits."""
    from sortnet_b200.layers import NormDistConv
    B, ci, co, side, kept = 70, 12, 30, 3, 7
    S, per = (B + 31) // 32, co // G
    gen = torch.Generator(device="cuda").manual_seed(G)
    lists = torch.rand(S, G, per, device="cuda", generator=gen).argsort(-1)[..., :kept].int()
    if repeat:
        lists[:, :, 3], lists[1, :, 5] = lists[:, :, 0], lists[1, :, 0]
    lists = lists.contiguous()
    layer = NormDistConv(ci, co, 1, groups=G, bias=True, mean_shift=False, dropout=0.5).cuda().train()
    with torch.no_grad():
        layer.bias.normal_(generator=gen)
    x = torch.rand(B, ci, side, side, device="cuda", generator=gen).requires_grad_()
    y = layer(x, mask_out=lists)[0]
    gy = torch.randn(y.shape, device="cuda", generator=gen) + 1
    gx, gw, gb = torch.autograd.grad(y, (x, layer.weight, layer.bias), gy)
    xo, wo, bo = (t.detach().double().requires_grad_() for t in (x, layer.weight, layer.bias))
    chan = (lists.long() + torch.arange(G, device="cuda").view(1, G, 1) * per)[torch.arange(B, device="cuda") // 32]          # [B, G, kept]
    dist = (xo.view(B, G, 1, ci // G, -1) - wo[chan].unsqueeze(-1)).abs().amax(3) + bo[chan].unsqueeze(-1)
    want = torch.autograd.grad(dist.reshape(y.shape), (xo, wo, bo), gy.double())
    assert rel(y.detach().cpu().numpy(), dist.reshape(y.shape).detach().cpu().numpy()) < 1e-6
    for got, exact, tol in zip((gx, gw, gb), want, (1e-5, 1e-5, 1e-6)):  # the bias sums in 64 bits up to a few additions of 2^-24
        assert rel(got.cpu().numpy(), exact.cpu().numpy()) < tol


@pytest.mark.parametrize("entry", [-1, 10])
def test_lists_that_name_no_channel(entry, monkeypatch):
    """Validated where that is asked for, by mean shift and bias alike; otherwise such an entry adds NaN and reads nothing."""
    from sortnet_b200 import layers, norm_dist_cuda as C
    index = torch.arange(7, device="cuda", dtype=torch.int32).repeat(3, 3, 1)
    index[1, 2, 4] = entry
    x, bias = torch.randn(70, 21, 4, device="cuda"), torch.randn(30, device="cuda", requires_grad=True)
    y = layers._add_per_channel(x, bias, index)
    bad = torch.zeros_like(x, dtype=torch.bool)
    bad[32:64, 18] = True
    assert torch.equal(y.isnan(), bad)
    y.sum().backward()                                       # leaves the entry out
    rows = 70.0 * 4 * torch.ones(3, 7, device="cuda")
    rows[2, 4] -= 32 * 4
    assert torch.equal(bias.grad.view(3, 10)[:, :7], rows) and not bias.grad.view(3, 10)[:, 7:].any()
    monkeypatch.setattr(C, "DEBUG_INDEX_CHECKS", True)
    shift = layers.MeanShiftDropout(30, affine=False).cuda().train()
    for call in (lambda: layers._add_per_channel(x, bias, index), lambda: shift(x, index=index)):
        with pytest.raises(RuntimeError, match="outside"):
            call()
    index[1, 2, 4] = 4
    assert torch.isfinite(layers._add_per_channel(x, bias, index)).all() and torch.isfinite(shift(x, index=index)[0]).all()


@pytest.mark.parametrize("kind", ["double", "strided"])
def test_running_mean_of_another_layout(kind):
    """A running mean that the kernel cannot update is updated in PyTorch."""
    from sortnet_b200.layers import MeanShiftDropout
    x = torch.randn(40, 6, 9, device="cuda")
    want, got = (MeanShiftDropout(6, affine=False).cuda().train() for _ in range(2))
    got.running_mean = torch.zeros(6, device="cuda", dtype=torch.float64) if kind == "double" else torch.zeros(12, device="cuda")[::2]
    for _ in range(2):
        y, z = want(x)[0], got(x)[0]
        assert torch.equal(y, z) and torch.allclose(want.running_mean.double(), got.running_mean.double(), rtol=1e-6, atol=1e-8)
    assert got.running_mean.dtype == (torch.float64 if kind == "double" else torch.float32)
