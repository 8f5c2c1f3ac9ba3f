"""The sparse form of the l-p kernels (large p, csrc/lp_skip.cu) against float64 and against the dense kernels.

Sizes sit at the edges of its slabs (1344 columns in the forward, 704 outputs in the backward), of a scan step
(256) and of a sub-batch (32 rows).  Forward: every element to 1e-5 like the dense kernels (the left-out terms are below 2^-27 of a
sum whose p-th root is taken).  Backward: max-abs error over max-abs value <= 1e-5."""
import numpy as np
import pytest
import torch

from gpu_util import make_masks

pytestmark = pytest.mark.gpu

TOL = 1e-5


def inputs(B, CI, CO, keep, seed, spread=1.0):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    W_CI, W_CO = CI, CO
    ci = co = None
    if keep < 1.0:
        rng = np.random.default_rng(seed)
        lists = [torch.from_numpy(make_masks(rng, B, n, keep)).cuda() for n in (W_CI, W_CO)]
        ci, co = lists[0], lists[1].flip(-1).contiguous()           # the order of a list is free
        CI, CO = ci.size(1), co.size(1)
    x = spread * torch.rand(B, CI, device="cuda", generator=gen)
    w = torch.randn(W_CO, W_CI, device="cuda", generator=gen)
    g = torch.randn(B, CO, device="cuda", generator=gen)
    return x, w, g, ci, co


def calls(x, w, g, ci, co, p, y=None, weight=True, sparse=True):
    """(y, gx, gw) through the library, with the scratch of the sparse form or with that of the dense kernels."""
    from sortnet_b200 import _lib
    lib = _lib.load()
    B, CI = x.shape
    CO = g.size(1)
    ptr = lambda t: None if t is None else t.data_ptr()
    dims, stream = (B, CO, CI, 1, 1), torch.cuda.current_stream().cuda_stream
    tail = (ptr(ci), ptr(co), w.size(0), w.size(1))
    need = [lib.snb_norm_dist_scratch_bytes(k, B, CO, CI, w.size(0), w.size(1), p, int(ci is not None)) for k in (0, 1)]
    assert need[1] > 0 and need[0] > 4 * B * (CO + CI)              # the sizes of this file take the sparse form
    if not sparse:
        need = [4 * B * CO, 0]
    ws = [torch.full((n + 16,), 0xff, dtype=torch.uint8, device="cuda") for n in need]   # scratch holds anything
    if y is None:
        y = torch.full((B, CO), float("nan"), device="cuda")
        _lib.check(lib.snb_norm_dist_forward_ws(ptr(x), ptr(w), *dims, ptr(y), p, *tail, ptr(ws[0]), need[0], stream), "forward")
    gx = torch.full((B, CI), float("nan"), device="cuda")
    gw = torch.full(w.shape, float("nan"), device="cuda") if weight else None
    _lib.check(lib.snb_norm_dist_backward_ws(ptr(g), ptr(x), ptr(w), ptr(y), *dims, ptr(gx), ptr(gw), p, *tail,
                                             ptr(ws[1]) if need[1] else None, need[1], stream), "backward")
    return y, gx, gw


def reference(x, w, g, ci, co, p, y):
    """float64 from the fp32 difference t = x - w on, which is part of the operators' definition (its rounding, taken
    to the power 999, alone would be 3e-5); the backward at the given y."""
    out = torch.zeros(g.shape, dtype=torch.float64, device="cuda")
    gx = torch.zeros(x.shape, dtype=torch.float64, device="cuda")
    gw = torch.zeros(w.shape, dtype=torch.float64, device="cuda")
    for s in range((x.size(0) + 31) // 32):
        rows = slice(32 * s, min(32 * s + 32, x.size(0)))
        cols = ci[s].long() if ci is not None else torch.arange(w.size(1), device="cuda")
        outs = co[s].long() if co is not None else torch.arange(w.size(0), device="cuda")
        sub = w[outs][:, cols]
        for b in range(rows.start, rows.stop):
            t = (x[b][None, :] - sub).double()
            a = t.abs()
            m = a.amax(1).clamp(min=1e-10)
            out[b] = m * ((a / m[:, None]).pow(p).sum(1) + (1e-10 / m).pow(p)).pow(1 / p)
            term = g[b].double()[:, None] * t.sign() * (a / y[b].double()[:, None]).pow(p - 1)
            gx[b] = term.sum(0)
            gw.index_put_((outs[:, None].expand_as(term), cols[None, :].expand_as(term)), -term, accumulate=True)
    return out, gx, gw


def near(a, b):
    return float((a.double() - b.double()).abs().max() / b.double().abs().max())


@pytest.mark.parametrize("B,CI,CO,keep", [(32, 1344, 1600, 1.0), (33, 1345, 1600, 1.0), (64, 1500, 704, 1.0), (31, 3100, 705, 1.0),
                                          (70, 3073, 320, 1.0), (1100, 257, 257, 1.0), (97, 1800, 1000, 0.7), (64, 2300, 1600, 0.75)])
@pytest.mark.parametrize("p", [10.5, 31.6, 41.5, 1000.0])
def test_against_float64(B, CI, CO, keep, p):
    x, w, g, ci, co = inputs(B, CI, CO, keep, B + CI)
    y, gx, gw = calls(x, w, g, ci, co, p)
    y_o, gx_o, gw_o = reference(x, w, g, ci, co, p, y)
    assert float(((y.double() - y_o).abs() / y_o).max()) < TOL
    assert near(gx, gx_o) < TOL and near(gw, gw_o) < TOL
    _, gx2, _ = calls(x, w, g, ci, co, p, y=y, weight=False)
    assert near(gx2, gx) < 1e-6                                     # sums in another order


# two, ten and three sub-batches on both sides of the 32 M weights that are not read again; slabs of one and more chunks
@pytest.mark.parametrize("B,CI,CO,keep", [(33, 5900, 5800, 1.0), (33, 5700, 5800, 1.0), (290, 2003, 1900, 1.0), (1100, 1003, 1100, 1.0), (96, 5120, 4600, 0.9), (96, 4700, 4200, 0.9)])
@pytest.mark.parametrize("kind", ["plain", "no numbers", "wide"])
@pytest.mark.parametrize("p", [31.6, 1000.0])
def test_maxima_of_many_sub_batches(B, CI, CO, keep, kind, p):
    """The forward where the maxima come from the pruned evaluation: values of the first, a middle and the last row against float64."""
    x, w, g, ci, co = inputs(B, CI, CO, keep, B + CI, spread=30.0 if kind == "wide" else 1.0)
    if kind == "wide":
        w *= 0.01                                                   # no list holds the columns that matter
    if kind == "no numbers":
        x[1, 17], x[B - 2, 5], w[7, 100], w[8, 101] = float("nan"), float("inf"), float("nan"), -float("inf")
    y, _, _ = calls(x, w, g, ci, co, p)
    dense, _, _ = calls(x, w, g, ci, co, p, sparse=False)
    # from p = 48 on the dense kernel passes over whole batches of terms, NaN among them
    assert torch.equal(dense.isfinite(), y.isfinite()) if p < 48 else bool((dense.isfinite() | ~y.isfinite()).all())
    ok = dense.isfinite() & y.isfinite()
    assert torch.allclose(dense[ok], y[ok], rtol=TOL, atol=0)
    for b in (0, B // 2, B - 1):
        cols = ci[b // 32].long() if ci is not None else slice(None)
        outs = co[b // 32].long() if co is not None else slice(None)
        a = (x[b][None, :] - w[outs][:, cols]).abs().double()
        m = a.amax(1).clamp(min=1e-10)
        y_o = m * ((a / m[:, None]).pow(p).sum(1) + (1e-10 / m).pow(p)).pow(1 / p)
        ok = y_o.isfinite() & y[b].isfinite()
        assert float(((y[b].double() - y_o).abs() / y_o)[ok].max()) < TOL


def test_data_that_cannot_be_skipped():
    """Inputs spread far wider than the weights: nearly every pair passes the test."""
    x, w, g, ci, co = inputs(64, 1400, 800, 1.0, 5, spread=50.0)
    y, gx, gw = calls(x, 0.01 * w, g, ci, co, 20.0)
    y_o, gx_o, gw_o = reference(x, 0.01 * w, g, ci, co, 20.0, y)
    assert float(((y.double() - y_o).abs() / y_o).max()) < TOL
    assert near(gx, gx_o) < TOL and near(gw, gw_o) < TOL


@pytest.mark.parametrize("p", [20.0, 60.0])
def test_values_that_are_no_numbers(p):
    """NaN and infinities reach the same outputs as through the dense kernels; zero distances and zero y too."""
    x, w, g, ci, co = inputs(64, 1400, 800, 1.0, 9)
    x[3, 17] = float("nan")
    x[40, 5] = float("inf")
    w[7, 100] = float("nan")
    w[8, 101] = -float("inf")
    x[33], w[9] = 0.25, 0.25                                        # distance 0
    dense = calls(x, w, g, ci, co, p, sparse=False)
    sparse = calls(x, w, g, ci, co, p)
    assert torch.equal(dense[0].isfinite(), sparse[0].isfinite())
    ok = dense[0].isfinite()
    assert torch.allclose(dense[0][ok], sparse[0][ok], rtol=TOL, atol=0)
    y = dense[0]
    y[50, 60], y[51, 61], g[52, 62], g[53, 63] = 0.0, -1.0, float("inf"), float("nan")
    dense = calls(x, w, g, ci, co, p, y=y, sparse=False)
    sparse = calls(x, w, g, ci, co, p, y=y)
    for a, b in zip(dense[1:], sparse[1:]):
        # from p = 49 on the dense backward passes over whole batches of terms, NaN among them
        assert torch.equal(a.isnan(), b.isnan()) if p < 49 else bool((b.isnan() | ~a.isnan()).all())
        ok = a.isfinite() & b.isfinite()
        assert p >= 49 or torch.equal(a.isfinite(), b.isfinite())
        assert not ok.any() or near(b[ok], a[ok]) < TOL


def test_host_threads_with_different_sizes():
    """Launches of the same kernel with more and with less shared memory from several threads."""
    import threading
    jobs = [(inputs(32, CI, CO, 1.0, CI), 60.0) for CI, CO in ((1344, 1600), (400, 1100), (3100, 705), (257, 1700))]
    want = [calls(*args, p)[0] for args, p in jobs]
    failures = []

    def work(args, p, y_o):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(100):
                    y, _, _ = calls(*args, p)
                    torch.cuda.current_stream().synchronize()
                    if near(y, y_o) > 1e-6:                         # sums in another order
                        failures.append("values")
        except Exception as exc:
            failures.append(repr(exc))
    torch.cuda.synchronize()
    threads = [threading.Thread(target=work, args=(args, p, y)) for (args, p), y in zip(jobs, want)]
    [t.start() for t in threads], [t.join() for t in threads]
    assert not failures, failures[:3]


@pytest.mark.parametrize("p", [1e6, 1e8, 3e8])
@pytest.mark.parametrize("shape", [(64, 1400, 800), (512, 300, 300)])
@pytest.mark.parametrize("narrow", [False, True])
def test_huge_finite_p(p, shape, narrow):
    """y is the maximum up to CI^(1/p), of which nothing is left in fp32.  At p = 3e8 the rounding of |t| / M and of
    its logarithm (2^-22, to the power p above 2^-126) leaves a sum that is not zero, in the dense kernel as here.  narrow: rows that hardly
    differ, so that the range of a column is no wider than the rounding of the test."""
    x, w, g, ci, co = inputs(*shape, 1.0, 11)
    if narrow:
        x = x[:1] + 2e-7 * x
    y, _, _ = calls(x, w, g, ci, co, p)
    dense, _, _ = calls(x, w, g, ci, co, p, sparse=False)
    top = (x[:, None, :] - w[None]).abs().amax(-1)
    assert near(y, dense) < 1e-6 and float(((y - top).abs() / top).max()) < 1e-5


def test_forward_with_scratch_between_the_forms():
    """Scratch for the sparse form but not for pruned maxima, as it was asked for before there were such: the scan's maxima, which are the same
    numbers, and so the same result; a byte less and the dense kernels run."""
    from sortnet_b200 import _lib
    lib = _lib.load()
    B, CI, CO, p = 1100, 1003, 1100, 200.0                          # one chunk of columns: sums in a fixed order
    x, w, _, _, _ = inputs(B, CI, CO, 1.0, 3)
    up256 = lambda n: (n + 255) // 256 * 256
    S = (B + 31) // 32
    least, full = up256(S * CI * 128) + up256(S * CI * 8) + 2 * up256(S * CO * 128), lib.snb_norm_dist_scratch_bytes(0, B, CO, CI, CO, CI, p, 0)
    assert full > least
    ys = []
    for nbytes in (full, full - 1, least, least - 1):
        ws = torch.full((nbytes + 16,), 0xff, dtype=torch.uint8, device="cuda")
        y = torch.full((B, CO), float("nan"), device="cuda")
        _lib.check(lib.snb_norm_dist_forward_ws(x.data_ptr(), w.data_ptr(), B, CO, CI, 1, 1, y.data_ptr(), p, None, None, CO, CI, ws.data_ptr(), nbytes,
                                                torch.cuda.current_stream().cuda_stream), "forward")
        assert (ws[nbytes:] == 0xff).all()
        ys.append(y)
    assert torch.equal(ys[0], ys[1]) and torch.equal(ys[0], ys[2])
    assert not torch.equal(ys[0], ys[3]) and torch.allclose(ys[0], ys[3], rtol=TOL, atol=0)
