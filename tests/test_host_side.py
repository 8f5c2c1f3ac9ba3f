"""CPU-only checks of the host side: the C-ABI library exports what the header declares, the
tensor-level module offers the reference extension's names, and argument validation works
without touching a GPU."""
import ctypes
import os
import re

import pytest
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def declared_symbols():
    text = open(os.path.join(ROOT, "include", "sortnet_b200.h")).read()
    return sorted(set(re.findall(r"\b(snb_[a-z0-9_]+)\s*\(", text)))


@pytest.fixture(scope="module")
def built_lib():
    from sortnet_b200 import build
    return ctypes.CDLL(build.build())


def test_library_exports_every_declared_symbol(built_lib):
    names = declared_symbols()
    assert len(names) >= 16
    for n in names:
        assert hasattr(built_lib, n), n


def test_loader_signatures_cover_the_header(built_lib):
    from sortnet_b200 import _lib
    utility = {"snb_status_string", "snb_last_cuda_error", "snb_version", "snb_inf_dist_forward_workspace_bytes",
               "snb_inf_dist_forward_noalloc_max_outputs", "snb_device_wait_failed", "snb_trim_scratch",
               "snb_norm_dist_forward_workspace_bytes", "snb_inf_dist_forward_sorted_workspace_bytes"}
    assert set(_lib.SIGNATURES) | utility == set(declared_symbols())
    lib = _lib.load()
    assert lib.snb_version() >= 100
    assert lib.snb_status_string(0) == b"ok" and b"null" in lib.snb_status_string(1)
    assert lib.snb_inf_dist_forward_workspace_bytes(512, 5120) == 8 * 512 * 5120
    # merge keys + full-width input + one inverse list per 32-row sub-batch
    assert lib.snb_inf_dist_forward_sorted_workspace_bytes(512, 4600, 5120) == 8 * 512 * 4600 + 4 * 512 * 5120 + 4 * 16 * 5120
    assert lib.snb_inf_dist_forward_sorted_workspace_bytes(33, 3, 8) == 800 + 4 * 33 * 8 + 4 * 2 * 8   # 792 rounded up to 16


def test_operator_module_follows_the_installed_torch(built_lib, monkeypatch):
    """_ops.so is rebuilt for another PyTorch, whatever the modification times say."""
    import subprocess
    from sortnet_b200 import build
    calls = []

    def compiler(cmd, **kw):
        calls.append(cmd[0])
        return subprocess.CompletedProcess(cmd, 0, "", "")
    monkeypatch.setattr(build.subprocess, "run", compiler)
    build.build_ops()
    assert calls == []
    stamp = os.path.join(build.OBJ, "ops_built_for")
    was = open(stamp).read()
    try:
        monkeypatch.setattr(torch, "__version__", "0.0.0")
        build.build_ops()
        assert calls == ["g++"]
    finally:
        with open(stamp, "w") as f:
            f.write(was)


def test_status_codes_without_gpu(built_lib):
    # argument checks run before any CUDA call
    from sortnet_b200 import _lib
    lib = _lib.load()
    assert lib.snb_inf_dist_forward_nograd(None, None, 1, 1, 1, 1, 1, None, None) == 1
    one = ctypes.c_void_p(16)
    assert lib.snb_inf_dist_forward_nograd(one, one, 1, 1, 1, 2, 1, one, None) == 2      # 1 channel, 2 groups
    assert lib.snb_inf_dist_forward_noalloc(one, one, 2, 2, 2, 2, 1, one, one, None) == 3   # groups need scratch
    assert lib.snb_inf_dist_forward_nograd(one, one, 0, 1, 1, 1, 1, one, None) == 2      # empty batch
    assert lib.snb_inf_dist_forward(one, one, 4, 4, 4, 1, 1, one, one, None, None, 5, 4, None) == 2
    assert lib.snb_norm_dist_forward(one, one, 4, 4, 4, 1, 1, one, ctypes.c_float(-1.0), None, None, 4, 4, None) == 3
    assert lib.snb_bound_inf_dist_forward_nograd(one, one, one, 70000, 70000, 4, 1, 1, one, one, None) == 4
    with pytest.raises(_lib.SortnetB200Error):
        _lib.check(2, "probe")


REFERENCE_NAMES = [
    "norm_dist_forward", "norm_dist_forward_with_max", "norm_dist_backward_input",
    "norm_dist_backward_input_weight", "inf_dist_forward", "inf_dist_forward_nograd",
    "inf_dist_backward_input", "inf_dist_backward_input_weight", "bound_inf_dist_forward",
    "bound_inf_dist_forward_nograd", "bound_inf_dist_backward_input", "bound_inf_dist_backward_input_weight",
    "sort_neuron_forward", "bound_sort_neuron_forward", "sort_neuron_forward_nograd",
    "sort_neuron_backward_input", "sort_neuron_backward_input_weight",
]


FAILED_LAUNCH = """
#include "launch.h"
// the runtime keeps the error of a failed call until somebody takes it
static cudaError_t held = cudaSuccess;
extern "C" cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t*, const void*, void**) { return held = cudaErrorInvalidConfiguration; }
extern "C" cudaError_t cudaGetLastError() {
    const cudaError_t e = held;
    held = cudaSuccess;
    return e;
}
cudaError_t snb::launched(int) { return cudaGetLastError(); }
static void kernel(int) {}
int main() { return snb::launch_next(kernel, 1, 1, 0, nullptr, 0) != cudaErrorInvalidConfiguration ? 1 : held != cudaSuccess ? 2 : 0; }
"""


def test_failed_launch_is_reported_once(tmp_path):
    """The next call, which works, must not be refused for it."""
    import subprocess
    from sortnet_b200 import build
    source, program = tmp_path / "failed_launch.cpp", tmp_path / "failed_launch"
    source.write_text(FAILED_LAUNCH)
    subprocess.run(["g++", "-std=c++17", "-I", build.CSRC, "-I", os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include"),
                    str(source), "-o", str(program)], check=True)
    assert subprocess.run([str(program)]).returncode == 0


def test_tensor_level_module_has_the_reference_names():
    from sortnet_b200 import norm_dist_cuda as C
    for n in REFERENCE_NAMES:
        assert callable(getattr(C, n)), n


def test_tensor_checks_raise_on_cpu_tensors():
    from sortnet_b200 import norm_dist_cuda as C
    x = torch.rand(4, 8, 1)
    w = torch.rand(3, 8)
    y = torch.empty(4, 3, 1)
    with pytest.raises(RuntimeError, match="CUDA tensor"):
        C.inf_dist_forward_nograd(x, w, y, 1)
    with pytest.raises(RuntimeError, match="CUDA tensor"):
        C.bound_inf_dist_forward_nograd(x, x, w, y, y, 1)


def test_whole_net_calls_refuse_other_targets():
    """Labels are read as int64 on the device: nothing else gets as far as a launch."""
    from sortnet_b200 import norm_dist_cuda as C
    x = torch.rand(4, 8)
    C._check_targets(torch.tensor([0, 1, 2, 3]), x)
    for bad in (torch.zeros(4, dtype=torch.int32), torch.zeros(3, dtype=torch.int64), torch.zeros(8, dtype=torch.int64)[::2],
                torch.zeros(4, dtype=torch.int64, device="meta"), torch.zeros(4)):
        for call in (lambda: C.mlp_train_forward(None, x, bad, 0.1, 1.0, 0.1, 1.0), lambda: C.mlp_eval_forward(None, x, None, bad)):
            with pytest.raises(RuntimeError, match="targets"):
                call()


def test_whole_net_calls_take_numbers_as_float_takes_them():
    from fractions import Fraction
    from sortnet_b200 import norm_dist_cuda as C
    plan = C.MlpPlan([[torch.rand(3, 8), torch.zeros(3), None, 0.0, None, 1, 0.0]])
    x, t = torch.rand(4, 8), torch.tensor([0, 1, 2, 0])
    for eps in (0.1, 1, "0.1", Fraction(1, 10), torch.tensor(0.1), torch.tensor([0.1])):
        with pytest.raises(RuntimeError, match="(?i)cuda"):  # gets as far as the device, which is none
            C.mlp_train_forward(plan, x, t, eps, 1.0, 0.1, 1.0)
    with pytest.raises(ValueError, match="one element"):
        C.mlp_train_forward(plan, x, t, torch.rand(2), 1.0, 0.1, 1.0)


def test_whole_net_plan_takes_only_what_the_kernels_read():
    """Anything else is left to the layers, which refuse it or know what to do with it."""
    from sortnet_b200 import norm_dist_cuda as C
    x = torch.rand(40, 12)

    def rows():
        lists = torch.zeros(2, 1, 5, dtype=torch.int32)
        return [[torch.rand(8, 12), None, torch.zeros(8), 0.1, lists, 1, 0.0], [torch.rand(3, 8), torch.zeros(3), None, 0.0, None, 1, 0.0]]

    assert C.MlpPlan(rows()).takes(x)
    assert not C.MlpPlan(rows()).takes(x[:, :11]) and not C.MlpPlan(rows()).takes(torch.rand(70, 12))
    for layer, field, bad in ((0, 0, torch.rand(8, 12).double()), (0, 0, torch.rand(12, 8).t()), (0, 0, torch.rand(8, 11)),
                              (1, 0, torch.rand(3, 9)), (0, 2, torch.zeros(7)), (1, 1, torch.zeros(3).half()),
                              (0, 4, torch.zeros(1, 1, 5, dtype=torch.int32)), (0, 4, torch.zeros(2, 2, 5, dtype=torch.int32)),
                              (0, 4, torch.zeros(2, 1, 5, dtype=torch.int64)), (0, 4, torch.zeros(2, 5, dtype=torch.int32))):
        table = rows()
        table[layer][field] = bad
        assert not C.MlpPlan(table).takes(x), (layer, field)
    assert C.box_fits((x, x), x)
    for bad in (x.double(), x[:, :11], x.unsqueeze(0)):
        assert not C.box_fits((x, bad), x)
        with pytest.raises(RuntimeError, match="box"):
            C.mlp_eval_forward(C.MlpPlan(rows()), x, (x, bad))


def test_hooks_and_overrides_keep_the_layers():
    """No whole-net plan for a net whose layers somebody wants called."""
    from sortnet_b200 import layers

    def net(p=float("inf")):
        m = layers.SortMLPModel(depth=3, width=16, input_dim=(1, 3, 3), num_classes=3, dropout=0.9)
        m.set_p(p)
        return m

    class Loud(layers.NormDist):
        def forward(self, *args, **kw):
            return super().forward(*args, **kw)

    class Other(layers.SortMLPModel):
        def _distances(self, *args, **kw):
            return super()._distances(*args, **kw)

    assert net()._plan() is not None and net(8.0)._plan() is None
    for register in ("register_forward_hook", "register_forward_pre_hook", "register_full_backward_hook",
                     "register_full_backward_pre_hook"):
        for pick in (lambda m: m.fc_dist[1], lambda m: m.fc_dist[2], lambda m: m.fc_dist[0].mean_shift):
            m = net()
            handle = getattr(pick(m), register)(lambda *a: None)
            assert m._plan() is None, register
            handle.remove()
            assert m._plan() is not None
    handle = torch.nn.modules.module.register_module_forward_hook(lambda *a: None)
    assert net()._plan() is None
    handle.remove()
    m = net()
    m.fc_dist[1].__class__ = Loud
    assert m._plan() is None
    m = net()
    m.fc_dist[1].forward = m.fc_dist[1].forward
    assert m._plan() is None
    assert Other(depth=3, width=16, input_dim=(1, 3, 3), num_classes=3)._plan() is None


class CudaWeight:
    """As far as ops._native looks at a weight."""
    is_cuda = True


def test_native_operators_stand_back_while_tracing():
    from sortnet_b200 import ops
    seen = []

    def f(x):
        seen.append(ops._native(CudaWeight()))
        return x + 1
    f(torch.ones(1))
    torch.jit.trace(f, (torch.ones(1),), check_trace=False)
    assert seen == [True, False]


def test_native_operators_stand_back_in_forward_mode():
    from torch.autograd import forward_ad
    from sortnet_b200 import ops
    assert ops._native(CudaWeight())
    with forward_ad.dual_level():
        assert not ops._native(CudaWeight())
    assert ops._native(CudaWeight())


def test_forms_with_scratch_stay_within_their_limits(built_lib):
    """Millions of outputs: no sparse form beyond its grids, no pruned form whose lists outgrow the card."""
    from sortnet_b200 import _lib
    lib = _lib.load()
    for outputs, sparse in ((4_000_000, True), (5_000_000, False)):
        assert (lib.snb_norm_dist_scratch_bytes(1, 32, outputs, 128, outputs, 128, 100.0, 0) > 0) == sparse
        dense = lib.snb_norm_dist_forward_workspace_bytes(32, outputs, 100.0)
        assert (lib.snb_norm_dist_scratch_bytes(0, 32, outputs, 128, outputs, 128, 100.0, 0) > dense) == sparse
    for outputs, pruned in ((1_000_000, True), (10_000_000, False)):
        assert (lib.snb_prune_scratch_bytes(1, 1, 1, 32, outputs, 128, outputs, 128, 0) > 0) == pruned
    assert lib.snb_prune_scratch_bytes(3, 10, 0, 512, 5120, 5120, 5120, 5120, 0) > 0


def test_operator_layer_signatures_match_the_reference():
    import inspect
    from sortnet_b200 import ops
    want = {
        "norm_dist": ["input", "weight", "p", "groups", "use_custom_cuda_func", "tag"],
        "norm_dist_dropout": ["input", "weight", "w_index_ci", "w_index_co", "p", "groups",
                              "use_custom_cuda_func", "tag"],
        "sort_neuron": ["input", "weight", "groups", "q", "truncate", "use_custom_cuda_func", "tag"],
        "bound_sort_neuron": ["x_lower", "x_upper", "weight", "groups", "q", "truncate", "tag"],
        "bound_inf_dist": ["x_lower", "x_upper", "weight", "groups", "use_custom_cuda_func", "tag"],
    }
    for name, params in want.items():
        assert list(inspect.signature(getattr(ops, name)).parameters) == params, name
    for cls in ("NormDistF", "NormDistDropoutF", "SortNeuronF", "BoundInfDistF"):
        assert issubclass(getattr(ops, cls), torch.autograd.Function)


def test_sample_mask_format():
    from sortnet_b200.layers import sample_mask
    torch.manual_seed(0)
    m = sample_mask(3, 1, 50, 0.8, device="cpu")
    assert m.dtype == torch.int32 and m.dim() == 3 and m.size(0) == 3 and m.size(1) == 1
    assert bool((m[..., 1:] > m[..., :-1]).all()) and int(m.max()) < 50 and int(m.min()) >= 0


def test_model_state_dict_keys_match_the_reference_layout():
    from sortnet_b200.layers import SortMLPModel
    model = SortMLPModel(depth=4, width=16, input_dim=(1, 2, 2), num_classes=3, dropout=0.9)
    keys = set(model.state_dict().keys())
    assert keys == {"fc_dist.0.weight", "fc_dist.0.mean_shift.running_mean", "fc_dist.1.weight",
                    "fc_dist.1.mean_shift.running_mean", "fc_dist.2.weight",
                    "fc_dist.2.mean_shift.running_mean", "fc_dist.3.weight", "fc_dist.3.bias"}


def test_shard_bounds_tile_the_flat_buffer():
    from sortnet_b200.optim import shard_bounds
    for numel in (4, 8, 120, 4096, 120644 // 4 * 4):
        for world in (1, 2, 3, 4, 8):
            edges = [shard_bounds(numel, world, r) for r in range(world)]
            assert edges[0][0] == 0 and edges[-1][1] == numel
            for (lo, hi), (lo2, _) in zip(edges, edges[1:]):
                assert hi == lo2 and lo <= hi
            assert all(lo % 4 == 0 and hi % 4 == 0 for lo, hi in edges)


def up256(n):
    return (n + 255) // 256 * 256


def sparse_forward_bytes(B, CO, CI):
    """Scratch of the sparse l-p forward itself: transposed inputs and their ranges, maxima and sums."""
    S = (B + 31) // 32
    return up256(S * CI * 128) + up256(S * CI * 8) + 2 * up256(S * CO * 128)


# sub-batches read W again often enough, and the pruned form does not read much more of it than they do
@pytest.mark.parametrize("B,CO,CI,W_CO,W_CI,pruned", [(512, 5120, 5120, 5120, 5120, True), (64, 5120, 5120, 5120, 5120, False), (96, 5120, 5120, 5120, 5120, True),
                                                      (512, 3840, 3840, 5120, 5120, True), (512, 512, 5120, 5120, 5120, True), (256, 4096, 4096, 8192, 8192, True),
                                                      (128, 4096, 4096, 8192, 8192, False), (512, 1000, 3300, 8192, 8192, False), (128, 2000, 6000, 12288, 12288, False),
                                                      (512, 2000, 6000, 12288, 12288, False)])
def test_maxima_of_the_sparse_forward_by_pruning(built_lib, B, CO, CI, W_CO, W_CI, pruned):
    from sortnet_b200 import _lib
    need = _lib.load().snb_norm_dist_scratch_bytes(0, B, CO, CI, W_CO, W_CI, 1000.0, int(CI < W_CI))
    own = sparse_forward_bytes(B, CO, CI)
    assert need > own if pruned else need == own


@pytest.mark.parametrize("B,CO,CI,W_CO,W_CI", [(512, 5120, 5120, 5120, 5120), (1024, 3840, 3840, 5120, 5120), (4096, 1500, 1001, 1500, 1001)])
def test_scratch_of_pruned_maxima(built_lib, B, CO, CI, W_CO, W_CI):
    """What the pruned form of this layer takes, without what only an evaluation as a whole needs: rows side by side, partial results, counters of tiles."""
    from sortnet_b200 import _lib
    lib = _lib.load()
    S, lists = (B + 31) // 32, int(CI < W_CI)
    whole = lib.snb_prune_scratch_bytes(1, 1, 0, B, CO, CI, W_CO, W_CI, lists)
    unused = up256(4 * S * 32 * ((W_CI + 3) // 4 * 4)) + up256(4 * S * CO * 32) + up256(4 * S * ((CO + 127) // 128))
    assert lib.snb_norm_dist_scratch_bytes(0, B, CO, CI, W_CO, W_CI, 1000.0, lists) == sparse_forward_bytes(B, CO, CI) + up256(whole - unused)
