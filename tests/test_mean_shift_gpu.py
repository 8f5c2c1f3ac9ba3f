"""GPU parity of the mean-shift kernels against the numpy restatement and the fixtures."""
import numpy as np
import pytest
import torch

import oracle
from gpu_util import col3, dev, host, idx3, make_masks, rel

pytestmark = pytest.mark.gpu


def run_center(x, index, C_full, running=None, momentum=0.1):
    from sortnet_b200 import norm_dist_cuda as C
    X = col3(x)
    mean = torch.full((C_full,), float("nan"), device="cuda")
    rm = None if running is None else dev(running)
    C.mean_shift_stats(X, idx3(index), mean, rm, momentum)
    y = torch.empty_like(X)
    C.mean_shift_apply(X, mean, idx3(index), y)
    return host(y), mean.cpu().numpy(), None if rm is None else rm.cpu().numpy()


@pytest.mark.parametrize("name", ["mean_shift_masked", "mean_shift_plain"])
def test_golden(golden, name):
    g = golden(name)
    index = g.get("index")
    C_full = g["running_mean0"].shape[0]
    y, mean, rm = run_center(g["x"], index, C_full, g["running_mean0"])
    assert rel(y, g["y"]) < 1e-5 and rel(rm, g["running_mean1"]) < 1e-5
    gx, _, _ = run_center(g["gy"], index, C_full)          # backward = the same centring of grad
    assert rel(gx, g["gx"]) < 1e-5


@pytest.mark.parametrize("B,C_full,keep", [(70, 40, 0.8), (512, 5120, 0.9), (33, 300, 0.5), (64, 128, None),
                                           (100, 77, None)])
def test_vs_oracle(B, C_full, keep):
    rng = np.random.default_rng(B + C_full)
    index = make_masks(rng, B, C_full, keep) if keep is not None else None
    C = index.shape[1] if index is not None else C_full
    x = rng.standard_normal((B, C)).astype(np.float32)
    y_o, mean_o = oracle.mean_shift_train(x, index, C_full)
    y, mean, _ = run_center(x, index, C_full)
    assert rel(y, y_o) < 1e-5 and rel(mean, mean_o) < 1e-5
    a = run_center(x, index, C_full)
    assert np.array_equal(a[0], y) and np.array_equal(a[1], mean)   # deterministic


def test_in_place_apply_and_eval():
    from sortnet_b200 import norm_dist_cuda as C
    rng = np.random.default_rng(1)
    x = rng.standard_normal((45, 24)).astype(np.float32)
    rm = rng.standard_normal(24).astype(np.float32)
    X = col3(x)
    C.mean_shift_apply(X, dev(rm), None, X)
    assert rel(host(X), x - rm[None]) < 1e-6


@pytest.mark.parametrize("B,G,C,kept,hw", [(1, 1, 8, 8, 1), (33, 1, 9, 5, 4), (70, 3, 30, 7, 9), (64, 2, 1000, 400, 1), (1100, 1, 40, 30, 2),
                                           (31, 1, 7, 7, 33)])
def test_plane_shift(B, G, C, kept, hw):
    """Mean shift, per-channel add and per-channel sums over rows and positions against float64."""
    from sortnet_b200 import norm_dist_cuda as NC
    gen = torch.Generator(device="cuda").manual_seed(B + hw)
    S, per, masked = (B + 31) // 32, C // G, kept * G < C
    index = None
    if masked:
        index = torch.rand(S, G, per, device="cuda", generator=gen).argsort(-1)[..., :kept].sort(-1)[0].int().contiguous()
        glob = (index.long() + torch.arange(G, device="cuda").view(1, G, 1) * per).reshape(S, -1)
    else:
        kept, glob = per, torch.arange(C, device="cuda").expand(S, C)
    chan = glob[torch.arange(B, device="cuda") // 32]
    x = torch.randn(B, G * kept, hw, device="cuda", generator=gen) + 3
    sums = torch.zeros(C, dtype=torch.float64, device="cuda").index_add_(0, chan.reshape(-1), x.double().sum(-1).reshape(-1))
    rows = torch.zeros(C, dtype=torch.float64, device="cuda").index_add_(0, chan.reshape(-1), torch.full((chan.numel(),), float(hw), dtype=torch.float64, device="cuda"))
    mean_o = torch.where(rows > 0, sums / rows.clamp(min=1), 0.0)
    mean, y, run = torch.empty(C, device="cuda"), torch.empty_like(x), torch.ones(C, device="cuda")
    NC.plane_shift(x, index, C, mean, y, run, 0.1)
    # sums in 64 bits: the mean has its own rounding and that of the quotient's operands, the running mean those of two products and a sum more
    assert ((mean.double() - mean_o).abs() <= 2 ** -23 * mean_o.abs()).all() and torch.equal(y, x - mean[chan].unsqueeze(-1))
    assert (run.double() - (0.9 + 0.1 * mean_o)).abs().max() <= 2e-6
    assert ((NC.plane_sum(x, index, C).double() - sums).abs() <= 2 ** -23 * sums.abs()).all()
    v = torch.randn(C, device="cuda", generator=gen)
    assert torch.equal(NC.plane_add(x, index, v), x + v[chan].unsqueeze(-1))


@pytest.mark.parametrize("B,G,per,kept,hw", [(70, 3, 10, 7, 9), (33, 1, 40, 40, 4), (1100, 1, 12, 5, 2)])
def test_plane_shift_writes_every_element(B, G, per, kept, hw):
    """Lists are to ascend; those that do not, or name a channel twice, leave no element of y unwritten: each is x minus the mean that its channel got."""
    from sortnet_b200 import norm_dist_cuda as NC
    gen = torch.Generator(device="cuda").manual_seed(B)
    S, C = (B + 31) // 32, G * per
    index = torch.rand(S, G, per, device="cuda", generator=gen).argsort(-1)[..., :kept].int()
    index[1:, :, 3] = index[1:, :, 0]
    index = index.contiguous()
    chan = (index.long() + torch.arange(G, device="cuda").view(1, G, 1) * per).reshape(S, -1)[torch.arange(B, device="cuda") // 32]
    x = torch.randn(B, G * kept, hw, device="cuda", generator=gen)
    mean, y = torch.empty(C, device="cuda"), torch.full_like(x, float("nan"))
    NC.plane_shift(x, index, C, mean, y)
    assert torch.equal(y, x - mean[chan].unsqueeze(-1))


# a warp per channel (with more than 32 sub-batches too), one CTA, clusters of 2, 4 and 8; more sub-batches than a CTA has threads; positions by four and by one
@pytest.mark.parametrize("B,G,C,kept,hw", [(1100, 1, 2000, 1500, 1), (40, 1, 600, 500, 4), (40, 1, 64, 48, 32), (70, 3, 30, 7, 49), (200, 1, 64, 64, 100), (200, 1, 64, 48, 33),
                                           (130, 1, 40, 30, 225), (128, 1, 16, 16, 1024), (128, 3, 15, 4, 1024), (8300, 2, 4, 1, 1), (300, 1, 3, 3, 401)])
@pytest.mark.parametrize("lists", ["ascending", "any order", "misaligned"])
def test_plane_kernels_of_every_form(B, G, C, kept, hw, lists):
    """Mean shift, sums and add against float64; lists in any order and with repeated channels as far as they are taken."""
    from sortnet_b200 import norm_dist_cuda as NC
    gen = torch.Generator(device="cuda").manual_seed(B + hw)
    S, per = (B + 31) // 32, C // G
    index, chan = None, torch.arange(C, device="cuda").expand(B, C)
    if kept * G < C:
        index = torch.rand(S, G, per, device="cuda", generator=gen).argsort(-1)[..., :kept].int()
        if lists == "any order":
            index[::2, :, -1] = index[::2, :, 0]
        else:
            index = index.sort(-1)[0]
        index = index.contiguous()
        chan = (index.long() + torch.arange(G, device="cuda").view(1, G, 1) * per).reshape(S, -1)[torch.arange(B, device="cuda") // 32]
    off = 1 if lists == "misaligned" else 0
    def buffer():
        return torch.full((off + chan.numel() * hw + 8,), 7.0, device="cuda")
    def view(t):
        return t[off:off + chan.numel() * hw].view(*chan.shape, hw)
    x = view(buffer())
    x.copy_(torch.randn(x.shape, device="cuda", generator=gen) + 1000)
    rows = torch.zeros(C, dtype=torch.float64, device="cuda").index_add_(0, chan.reshape(-1), torch.full((chan.numel(),), float(hw), dtype=torch.float64, device="cuda"))
    sums = torch.zeros(C, dtype=torch.float64, device="cuda").index_add_(0, chan.reshape(-1), x.double().sum(-1).reshape(-1))
    y_all, mean, run = buffer(), torch.empty(C, device="cuda"), torch.ones(C, device="cuda")
    y = view(y_all)
    NC.plane_shift(x, index, C, mean, y, run, 0.1)
    assert torch.equal(y, x - mean[chan].unsqueeze(-1)) and (y_all[off + y.numel():] == 7).all() and (y_all[:off] == 7).all()
    if lists != "any order" or index is None:
        want = torch.where(rows > 0, sums / rows.clamp(min=1), 0.0)
        assert ((mean.double() - want).abs() <= 2 ** -23 * want.abs()).all()         # 64-bit sums: the result's rounding and a last digit
        assert ((run.double() - (0.9 + 0.1 * want)).abs() <= 2 ** -22 * (0.9 + 0.1 * want.abs())).all()
    # in any order up to three additions of parts per sub-batch
    bound = 2 ** -23 if lists != "any order" else 2 ** -23 * (2 + 3 * S)
    assert ((NC.plane_sum(x, index, C).double() - sums).abs() <= bound * sums.abs()).all()
    v = torch.randn(C, device="cuda", generator=gen)
    assert torch.equal(NC.plane_add(x, index, v), x + v[chan].unsqueeze(-1))


@pytest.mark.parametrize("lists", [False, True])
def test_plane_kernels_past_31_bits(lists):
    """More than 2^31 elements in all."""
    from sortnet_b200 import norm_dist_cuda as NC
    B, G, kept, hw = 33, 2, 2, (1 << 31) // (33 * 4) + 5
    C = G * (3 if lists else 2)
    index = torch.tensor([[[0, 2], [1, 2]], [[1, 2], [0, 1]]], dtype=torch.int32, device="cuda") if lists else None
    chan = torch.tensor([[0, 2, 4, 5]] * 32 + [[1, 2, 3, 4]] if lists else [[0, 1, 2, 3]] * B, device="cuda")
    x = torch.empty(B, G * kept, hw, device="cuda").uniform_(generator=torch.Generator(device="cuda").manual_seed(0))
    sums = torch.zeros(C, dtype=torch.float64, device="cuda").index_add_(0, chan.reshape(-1), x.sum(-1, dtype=torch.float64).reshape(-1))
    rows = torch.zeros(C, dtype=torch.float64, device="cuda").index_add_(0, chan.reshape(-1), torch.ones(chan.numel(), dtype=torch.float64, device="cuda"))
    assert ((NC.plane_sum(x, index, C).double() - sums).abs() <= 2 ** -23 * sums).all()
    v = torch.randn(C, device="cuda")
    y = NC.plane_add(x, index, v)
    assert all(torch.equal(y[b, j], x[b, j] + v[chan[b, j]]) for b in range(B) for j in range(G * kept))
    mean = torch.empty(C, device="cuda")
    NC.plane_shift(x, index, C, mean, y.fill_(7.0))
    assert ((mean.double() - sums / (rows * hw)).abs() <= 2 ** -23).all()
    assert all(torch.equal(y[b, j], x[b, j] - mean[chan[b, j]]) for b in range(B) for j in range(G * kept))
