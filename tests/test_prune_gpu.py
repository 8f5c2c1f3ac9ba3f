"""Pruned evaluation of the max-type operators (csrc/prune.cu) against the CPU oracle: bit-exact values,
positions and bound words, whatever the data.  Every shape here is large enough for it
(snb_prune_scratch_bytes > 0)."""
import numpy as np
import pytest
import torch

import oracle
from gpu_util import col3, dev, host, idx3, make_masks, rel

pytestmark = pytest.mark.gpu
EPS = np.float32(1e-10)


def operands(kind, rng, B, CI, CO):
    if kind == "normal":                 # what the layers hold: a handful of columns per row survive
        return rng.random((B, CI), dtype=np.float32), rng.standard_normal((CO, CI)).astype(np.float32)
    if kind == "ties":                   # quantised: many columns share the maximum
        return ((rng.integers(0, 4, (B, CI)) / 4).astype(np.float32),
                (rng.standard_normal((CO, CI)) * 2).round().astype(np.float32) / 2)
    if kind == "flat":                   # nothing can be pruned: every output is left to the dense kernel
        return ((rng.random((B, CI)) * 2 - 1).astype(np.float32), (0.01 * rng.random((CO, CI))).astype(np.float32))
    assert kind == "mixed"               # some rows of W flat, NaN and infinities among the rest
    x, w = rng.standard_normal((B, CI)).astype(np.float32), rng.standard_normal((CO, CI)).astype(np.float32)
    w[::7] *= 0.001
    x[3, 5], x[1, 9], w[2, 4], w[8, 11], w[11] = np.nan, np.inf, np.nan, -np.inf, np.nan
    return x, w


def uses_pruning(tensors, K, words, B, CO, CI, W_CO, W_CI, lists):
    from sortnet_b200 import _lib
    return _lib.load().snb_prune_scratch_bytes(tensors, K, words, B, CO, CI, W_CO, W_CI, lists) > 0


# widths: one step of the filter up to its widest row, odd ones, tile edges; ragged rows and outputs
SHAPES = [(70, 1024, 1000), (33, 1025, 1101), (128, 784, 520), (32, 5120, 257), (40, 6147, 200), (31, 12288, 130),
          (300, 130, 1033), (5, 8192, 1024)]


@pytest.mark.parametrize("B,CI,CO", SHAPES)
@pytest.mark.parametrize("kind", ["normal", "ties", "flat", "mixed"])
def test_distance_and_words(B, CI, CO, kind):
    from sortnet_b200 import norm_dist_cuda as C
    assert uses_pruning(1, 1, 1, B, CO, CI, CO, CI, 0)
    x, w = operands(kind, np.random.default_rng(B + CI), B, CI, CO)
    y_o, pos_o = oracle.inf_dist_forward(x, w)
    y, pos = torch.full((B, CO, 1), 7.0, device="cuda"), torch.full((B, CO, 1), 7, device="cuda", dtype=torch.int32)
    C.inf_dist_forward(col3(x), dev(w), y, pos, 1)
    assert np.array_equal(host(y), y_o) and np.array_equal(host(pos), pos_o)
    yn = torch.full((B, CO, 1), 7.0, device="cuda")
    C.inf_dist_forward_nograd(col3(x), dev(w), yn, 1)
    assert np.array_equal(host(yn), y_o)


# widths on both sides of the filter's forms, copied by fours and by ones; fewer rows than CTAs, and many steps per CTA
@pytest.mark.parametrize("B,CI,CO", [(32, 2048, 200), (33, 2050, 200), (31, 3072, 150), (31, 3073, 150), (32, 4096, 120), (32, 4097, 120),
                                     (32, 5501, 100), (32, 6144, 90), (32, 8193, 60), (32, 300, 4001), (32, 132, 9001)])
@pytest.mark.parametrize("kind", ["normal", "ties", "mixed"])
def test_filter_forms(B, CI, CO, kind):
    from sortnet_b200 import norm_dist_cuda as C
    assert uses_pruning(1, 1, 1, B, CO, CI, CO, CI, 0)
    x, w = operands(kind, np.random.default_rng(CI), B, CI, CO)
    y_o, pos_o = oracle.inf_dist_forward(x, w)
    y, pos = torch.full((B, CO, 1), 7.0, device="cuda"), torch.full((B, CO, 1), 7, device="cuda", dtype=torch.int32)
    C.inf_dist_forward(col3(x), dev(w), y, pos, 1)
    assert np.array_equal(host(y), y_o) and np.array_equal(host(pos), pos_o)


@pytest.mark.parametrize("B,CI,CO,keep", [(70, 1024, 1100, 0.9), (160, 1030, 460, 0.7), (33, 2049, 1900, 0.5),
                                          (96, 5120, 200, 0.95)])
@pytest.mark.parametrize("which", ["both", "ci", "co"])
@pytest.mark.parametrize("kind", ["normal", "ties", "flat"])
@pytest.mark.parametrize("ascending", [True, False])
def test_masked_distance(B, CI, CO, keep, which, kind, ascending):
    from sortnet_b200 import norm_dist_cuda as C
    rng = np.random.default_rng(B + CI + CO)
    ci = make_masks(rng, B, CI, keep) if which in ("both", "ci") else None
    co = make_masks(rng, B, CO, keep) if which in ("both", "co") else None
    if not ascending:
        ci, co = (None if m is None else rng.permuted(m, axis=1) for m in (ci, co))
    x, w = operands(kind, rng, B, CI, CO)
    x = np.ascontiguousarray(x[:, :ci.shape[1]]) if ci is not None else x
    n_out = co.shape[1] if co is not None else CO
    assert uses_pruning(1, 1, 1, B, n_out, x.shape[1], CO, CI, int(ci is not None))
    y_o, pos_o = oracle.inf_dist_forward(x, w, ci, co)
    y = torch.empty(B, n_out, 1, device="cuda")
    pos = torch.empty(B, n_out, 1, device="cuda", dtype=torch.int32)
    entry = C.inf_dist_forward_sorted if ascending else lambda a, b, c, d, i, o: C.inf_dist_forward(a, b, c, d, 1, i, o)
    entry(col3(x), dev(w), y, pos, idx3(ci), idx3(co))
    assert np.array_equal(host(y), y_o) and np.array_equal(host(pos), pos_o)


def test_lists_that_miss_the_largest_weights():
    """The kept columns are those with the smallest weights: every output is found wanting and redone."""
    from sortnet_b200 import norm_dist_cuda as C
    rng = np.random.default_rng(5)
    B, CI, CO = 64, 1024, 600
    x, w = operands("normal", rng, B, CI, CO)
    w[:, CI // 2:] *= 100
    ci = np.tile(np.arange(CI // 2, dtype=np.int32), (2, 1))
    x = np.ascontiguousarray(x[:, :CI // 2])
    y_o, pos_o = oracle.inf_dist_forward(x, w, ci, None)
    y, pos = torch.empty(B, CO, 1, device="cuda"), torch.empty(B, CO, 1, device="cuda", dtype=torch.int32)
    C.inf_dist_forward_sorted(col3(x), dev(w), y, pos, idx3(ci), None)
    assert np.array_equal(host(y), y_o) and np.array_equal(host(pos), pos_o)


@pytest.mark.parametrize("B,CI,CO", SHAPES[:6])
@pytest.mark.parametrize("kind", ["normal", "ties", "flat", "mixed"])
def test_interval_bounds(B, CI, CO, kind):
    from sortnet_b200 import norm_dist_cuda as C
    rng = np.random.default_rng(B * 3 + CI)
    assert uses_pruning(2, 1, 1, B, CO, CI, CO, CI, 0) and uses_pruning(3, 1, 0, B, CO, CI, CO, CI, 0)
    x, w = operands(kind, rng, B, CI, CO)
    half = np.float32(0.25) if kind == "ties" else np.float32(0.03)
    xl, xu = (x - half).astype(np.float32), (x + half).astype(np.float32)
    flip = rng.random((B, CI)) < 0.01                       # inverted intervals are repaired to their midpoint
    xl[flip], xu[flip] = xu[flip], xl[flip]
    yl_o, yu_o, pl_o, pu_o = oracle.bound_inf_dist_forward(xl, xu, w)
    XL, XU, W = col3(xl), col3(xu), dev(w)
    yl, yu = torch.empty(B, CO, 1, device="cuda"), torch.empty(B, CO, 1, device="cuda")
    C.bound_inf_dist_forward_nograd(XL, XU, W, yl, yu, 1)
    assert np.array_equal(host(yl), yl_o) and np.array_equal(host(yu), yu_o)
    pl, pu = torch.empty_like(yl, dtype=torch.int32), torch.empty_like(yl, dtype=torch.int32)
    yl.fill_(7), yu.fill_(7)
    C.bound_inf_dist_forward(XL, XU, W, yl, yu, pl, pu, 1)
    assert np.array_equal(host(yl), yl_o) and np.array_equal(host(yu), yu_o)
    assert np.array_equal(host(pl), pl_o) and np.array_equal(host(pu), pu_o)
    # point value and box in one pass; the point may lie outside the box
    y3 = [torch.empty(B, CO, device="cuda") for _ in range(3)]
    xp = (x + np.float32(0.1)).astype(np.float32)
    C.layer_bound_forward(dev(xp), XL.squeeze(-1), XU.squeeze(-1), W, None, None, *y3)
    y_o, _ = oracle.inf_dist_forward(xp, w)
    assert all(np.array_equal(a.cpu().numpy(), b) for a, b in zip(y3, (y_o, yl_o, yu_o)))


@pytest.mark.parametrize("B,CI,CO", [(70, 1024, 1000), (33, 1025, 1101), (32, 5120, 257)])
@pytest.mark.parametrize("q,K", [(0.75, 10), (0.5, 4), (0.85, 25), (0.6, 17)])
@pytest.mark.parametrize("kind", ["normal", "ties", "flat"])
def test_sort_neuron(B, CI, CO, q, K, kind):
    from sortnet_b200 import norm_dist_cuda as C
    assert uses_pruning(1, K, 1, B, CO, CI, CO, CI, 0)
    x, w = operands(kind, np.random.default_rng(B + CI), B, CI, CO)
    y_o, pos_o = oracle.sort_forward(x, w, q, K)
    X, W = col3(x), dev(w)
    y = torch.empty(B, CO, 1, device="cuda")
    C.sort_neuron_forward_nograd(X, W, y, 1, q, K)
    assert rel(host(y), y_o) < 2e-6
    y2, pos = torch.empty_like(y), torch.empty(K, B, CO, 1, device="cuda", dtype=torch.int32)
    C.sort_neuron_forward(X, W, y2, pos, 1, q, K)
    assert np.array_equal(host(y2), host(y)) and np.array_equal(pos.squeeze(-1).cpu().numpy(), pos_o)
    xl, xu = (x - np.float32(0.03)).astype(np.float32), (x + np.float32(0.03)).astype(np.float32)
    yl_o, yu_o = oracle.sort_bound_forward(xl, xu, w, q, K)
    yl, yu = torch.empty_like(y), torch.empty_like(y)
    C.bound_sort_neuron_forward(col3(xl), col3(xu), W, yl, yu, 1, q, K)
    assert rel(host(yl), yl_o) < 2e-6 and rel(host(yu), yu_o) < 2e-6


def half_prunable(kind, rng, B, CI, CO):
    """Rows of W whose list overflows: single ones (below the share at which the layer is evaluated as a whole), a block
    of neighbours, and all of them, on inputs as wide as the weights and with NaN, infinities and ties."""
    x, w = rng.random((B, CI), dtype=np.float32), rng.standard_normal((CO, CI)).astype(np.float32)
    if kind == "single":
        w[::64] *= 0.001
    elif kind == "block":
        w[40:40 + CO // 40] *= 0.001
    else:
        x = (0.5 * rng.standard_normal((B, CI))).astype(np.float32)
        if kind == "wide ties":
            x, w = (x * 4).round() / 4, (w * 2).round() / 2
        else:
            x[3, 5], x[1, 9], x[0], w[2, 4], w[8, 11], w[11] = np.nan, np.inf, 0.25, np.nan, -np.inf, 0.25
    return x.astype(np.float32), w


@pytest.mark.parametrize("off", [-1, 0])
@pytest.mark.parametrize("kind", ["normal", "ties"])
@pytest.mark.parametrize("q,K", [(0.75, 10), (0.5, 4)])
def test_sort_neuron_around_the_split_of_outputs(off, kind, q, K):
    """Eight outputs per CTA below twelve CTAs of 32 per SM, 32 from there on: both give what 32 rows by themselves give
    (those are held against the oracle above)."""
    from sortnet_b200 import norm_dist_cuda as C
    B, CI = 310, 140
    tiles = -(-12 * torch.cuda.get_device_properties(0).multi_processor_count // 10) + off
    CO = 32 * tiles - 27
    x, w = operands(kind, np.random.default_rng(CO), B, CI, CO)
    X, W = col3(x), dev(w)

    def run(rows):
        part, n = X[rows].contiguous(), rows.stop - rows.start
        y, v = (torch.empty(n, CO, 1, device="cuda") for _ in range(2))
        pos = torch.empty(K, n, CO, 1, device="cuda", dtype=torch.int32)
        C.sort_neuron_forward(part, W, y, pos, 1, q, K)
        C.sort_neuron_forward_nograd(part, W, v, 1, q, K)
        return torch.stack((y, v)), pos

    Y, P = run(slice(0, B))
    assert torch.equal(Y[0], Y[1])
    for b in range(0, B, 32):
        rows = slice(b, min(b + 32, B))
        y, p = run(rows)
        assert torch.equal(y, Y[:, rows]) and torch.equal(p, P[:, rows])


@pytest.mark.parametrize("off", [-1, 0])
@pytest.mark.parametrize("kind", ["normal", "ties"])
@pytest.mark.parametrize("K", [11, 21, 22, 25])
def test_sort_neuron_of_many_values_around_the_split_of_outputs(off, kind, K):
    """The same above ten values: eight outputs per CTA below six CTAs of 32 per SM, and always past K = 21."""
    from sortnet_b200 import _lib, norm_dist_cuda as C
    B, CI, q = 100, 200, 0.8
    CO = 32 * (-(-6 * torch.cuda.get_device_properties(0).multi_processor_count // 4) + off) - 27
    x, w = operands(kind, np.random.default_rng(CO), B, CI, CO)
    X, W = col3(x), dev(w)
    y, v, z = (torch.empty(B, CO, 1, device="cuda") for _ in range(3))
    pos, want = (torch.empty(K, B, CO, 1, device="cuda", dtype=torch.int32) for _ in range(2))
    C.sort_neuron_forward(X, W, y, pos, 1, q, K)
    C.sort_neuron_forward_nograd(X, W, v, 1, q, K)
    _lib.check(_lib.load().snb_sort_neuron_forward(X.data_ptr(), W.data_ptr(), B, CO, CI, 1, 1, z.data_ptr(), want.data_ptr(), q, K,
                                                   torch.cuda.current_stream().cuda_stream), "sort_neuron_forward")
    assert torch.equal(pos, want) and torch.equal(y, v) and rel(host(y), host(z)) < 2e-6


@pytest.mark.parametrize("K", [2, 8, 9, 10, 11, 25])
@pytest.mark.parametrize("kind", ["rising", "few", "few and NaN"])
def test_sort_neuron_queues(K, kind):
    """Rows whose values rise along the list, so that every entry enters and is merged in its turn (the log of positions runs over), and
    lists around the entries that start a row's list (8) and a step (4).  Values, positions and bounds against the dense kernels."""
    from sortnet_b200 import _lib, norm_dist_cuda as C
    B, CI, CO, q = 70, 140, 1100, 0.8
    rng = np.random.default_rng(K)
    x, w = rng.random((B, CI), dtype=np.float32), rng.standard_normal((CO, CI)).astype(np.float32)
    if kind == "rising":
        # every column spans [0, 1]; its largest bound is 4 - c / 1000, while rows 2, 34 and 66 see 3 + c / 1000
        x[:] = 0.0
        x[1::32] = 1.0
        x[2::32] = 0.002 * np.arange(CI)
        w[:] = -3.0 + 0.001 * np.arange(CI) + 1e-5 * rng.random((CO, CI))
    else:
        # a handful of columns with far weights, K and more of them in turn
        x *= 0.01
        w *= 0.01
        for j in range(CO):
            w[j, rng.permutation(CI)[:K + j % 7]] += 5.0
        if kind == "few and NaN":
            x[40, 3], w[5, 100], x[7] = np.nan, np.nan, np.nan
    X, W = col3(x.astype(np.float32)), dev(w.astype(np.float32))
    st = torch.cuda.current_stream().cuda_stream
    y, v, z = (torch.empty(B, CO, 1, device="cuda") for _ in range(3))
    pos, want = (torch.empty(K, B, CO, 1, device="cuda", dtype=torch.int32) for _ in range(2))
    C.sort_neuron_forward(X, W, y, pos, 1, q, K)
    C.sort_neuron_forward_nograd(X, W, v, 1, q, K)
    _lib.check(_lib.load().snb_sort_neuron_forward(X.data_ptr(), W.data_ptr(), B, CO, CI, 1, 1, z.data_ptr(), want.data_ptr(), q, K, st), "sort")
    assert torch.equal(pos, want) and torch.equal(y, v) and torch.allclose(y, z, rtol=2e-6, atol=0)
    if "NaN" in kind:
        return                                              # dense bounds move their lists on NaN
    XL, XU = X - 0.03, X + 0.03
    yl, yu, zl, zu = (torch.empty_like(y) for _ in range(4))
    C.bound_sort_neuron_forward(XL, XU, W, yl, yu, 1, q, K)
    _lib.check(_lib.load().snb_bound_sort_neuron_forward(XL.data_ptr(), XU.data_ptr(), W.data_ptr(), B, CO, CI, 1, 1, zl.data_ptr(), zu.data_ptr(),
                                                         q, K, st), "bounds")
    assert torch.allclose(yl, zl, rtol=2e-6, atol=0) and torch.allclose(yu, zu, rtol=2e-6, atol=0)


def test_positions_of_25_values_where_some_lists_overflow():
    """Outputs that the walk leaves to prune_redo, among others that it does not: the positions of all are the dense kernel's."""
    from sortnet_b200 import _lib, norm_dist_cuda as C
    B, CI, CO, q, K = 70, 5120, 700, 0.75, 25
    x, w = operands("normal", np.random.default_rng(3), B, CI, CO)
    X, W = col3(x), dev(w)
    y, z = (torch.empty(B, CO, 1, device="cuda") for _ in range(2))
    pos, want = (torch.full((K, B, CO, 1), -1, device="cuda", dtype=torch.int32) for _ in range(2))
    C.sort_neuron_forward(X, W, y, pos, 1, q, K)
    _lib.check(_lib.load().snb_sort_neuron_forward(X.data_ptr(), W.data_ptr(), B, CO, CI, 1, 1, z.data_ptr(), want.data_ptr(), q, K,
                                                   torch.cuda.current_stream().cuda_stream), "sort_neuron_forward")
    assert torch.equal(pos, want) and rel(host(y), host(z)) < 2e-6


# columns around the tiles' steps (32) and the rows' alignment (4), outputs around their tiles (64, 128, 256), one and more sub-batches
@pytest.mark.parametrize("B,CI,CO", [(33, 1024, 1100), (64, 1028, 1000), (70, 1025, 1000), (31, 1503, 1281), (100, 4100, 321)])
@pytest.mark.parametrize("kind", ["single", "block", "wide", "wide ties"])
def test_lists_that_overflow(B, CI, CO, kind):
    from sortnet_b200 import norm_dist_cuda as C
    assert uses_pruning(1, 1, 1, B, CO, CI, CO, CI, 0) and uses_pruning(1, 10, 1, B, CO, CI, CO, CI, 0)
    x, w = half_prunable(kind, np.random.default_rng(B + CI), B, CI, CO)
    y_o, pos_o = oracle.inf_dist_forward(x, w)
    X, W = col3(x), dev(w)
    y, pos = torch.full((B, CO, 1), 7.0, device="cuda"), torch.full((B, CO, 1), 7, device="cuda", dtype=torch.int32)
    C.inf_dist_forward(X, W, y, pos, 1)
    assert np.array_equal(host(y), y_o) and np.array_equal(host(pos), pos_o)
    C.inf_dist_forward_nograd(X, W, y.fill_(7), 1)
    assert np.array_equal(host(y), y_o)
    xl, xu = (x - np.float32(0.05)).astype(np.float32), (x + np.float32(0.05)).astype(np.float32)
    yl_o, yu_o, pl_o, pu_o = oracle.bound_inf_dist_forward(xl, xu, w)
    XL, XU = col3(xl), col3(xu)
    yl, yu, pl, pu = (torch.empty_like(y), torch.empty_like(y), torch.empty_like(pos), torch.empty_like(pos))
    C.bound_inf_dist_forward(XL, XU, W, yl, yu, pl, pu, 1)
    assert all(np.array_equal(host(a), b) for a, b in zip((yl, yu, pl, pu), (yl_o, yu_o, pl_o, pu_o)))
    y3 = [torch.empty(B, CO, device="cuda") for _ in range(3)]
    C.layer_bound_forward(X.squeeze(-1), XL.squeeze(-1), XU.squeeze(-1), W, None, None, *y3)
    assert all(np.array_equal(a.cpu().numpy(), b) for a, b in zip(y3, (y_o, yl_o, yu_o)))
    if kind == "wide":
        return                                              # the oracle's sort is not defined on NaN
    ys, ps = torch.empty_like(y), torch.empty(10, B, CO, 1, device="cuda", dtype=torch.int32)
    ys_o, ps_o = oracle.sort_forward(x, w, 0.75, 10)
    C.sort_neuron_forward(X, W, ys, ps, 1, 0.75, 10)
    assert rel(host(ys), ys_o) < 2e-6 and np.array_equal(ps.squeeze(-1).cpu().numpy(), ps_o)
    C.sort_neuron_forward_nograd(X, W, ys.fill_(7), 1, 0.75, 10)
    assert rel(host(ys), ys_o) < 2e-6
    yl_o, yu_o = oracle.sort_bound_forward(xl, xu, w, 0.75, 10)
    C.bound_sort_neuron_forward(XL, XU, W, yl, yu, 1, 0.75, 10)
    assert rel(host(yl), yl_o) < 2e-6 and rel(host(yu), yu_o) < 2e-6


@pytest.mark.parametrize("which", ["both", "ci"])
@pytest.mark.parametrize("kind", ["wide", "wide ties", "single"])
@pytest.mark.parametrize("ascending", [True, False])
def test_masked_lists_that_overflow(which, kind, ascending):
    from sortnet_b200 import norm_dist_cuda as C
    rng = np.random.default_rng(4)
    B, CI, CO = 97, 1030, 700
    ci, co = make_masks(rng, B, CI, 0.8), make_masks(rng, B, CO, 0.8) if which == "both" else None
    ci = ci if ascending else rng.permuted(ci, axis=1)
    x, w = half_prunable(kind, rng, B, CI, CO)
    x = np.ascontiguousarray(x[:, :ci.shape[1]])
    n_out = CO if co is None else co.shape[1]
    y_o, pos_o = oracle.inf_dist_forward(x, w, ci, co)
    entries = [lambda a, b, c, d, i, o: C.inf_dist_forward(a, b, c, d, 1, i, o)] + ([C.inf_dist_forward_sorted] if ascending else [])
    for entry in entries:
        y, pos = torch.empty(B, n_out, 1, device="cuda"), torch.empty(B, n_out, 1, device="cuda", dtype=torch.int32)
        entry(col3(x), dev(w), y, pos, idx3(ci), idx3(co))
        assert np.array_equal(host(y), y_o) and np.array_equal(host(pos), pos_o)


@pytest.mark.parametrize("kind", ["normal", "ties", "flat"])
def test_columns_that_come_twice(kind):
    """A list may name a column more than once, each with inputs of its own."""
    from sortnet_b200 import norm_dist_cuda as C
    rng = np.random.default_rng(6)
    B, CI, CO = 70, 1024, 1000
    x, w = operands(kind, rng, B, CI, CO)
    ci = rng.integers(0, CI, (3, 900)).astype(np.int32)
    ci[1] = np.sort(rng.permutation(CI)[:900])              # one of the sub-batches has a list like any other
    x = np.ascontiguousarray(x[:, :900])
    assert uses_pruning(1, 1, 1, B, CO, 900, CO, CI, 1)
    y_o, pos_o = oracle.inf_dist_forward(x, w, ci, None)
    y, pos = torch.empty(B, CO, 1, device="cuda"), torch.empty(B, CO, 1, device="cuda", dtype=torch.int32)
    C.inf_dist_forward(col3(x), dev(w), y, pos, 1, idx3(ci), None)
    assert np.array_equal(host(y), y_o) and np.array_equal(host(pos), pos_o)
