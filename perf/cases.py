"""What a user of this framework has it do, as cases that can be timed: single norm-distance layers,
SortNet-MLP training steps over the p schedule, certification and attack passes, a convolutional
stack, and the optimiser update.

listed()          the fixed cases
draw(rng)         one more case of the same ranges
prepare(case, s)  inputs, weights and model on the GPU, made from the seed s alone
run(state)        one pass through the public entry points, and its outputs
work(case)        bytes and operations that a pass cannot do without
tolerance(case)   how far another correct implementation at the same precision may be off

A case is a dict of plain values.  `p` is a text: "inf" or a number.  Image sizes are channels x side
x side.  The weights are N(0, 1) as the layers initialise them and images are smooth, with pixel noise
and a brightness of their own, in [0, 1]."""
import math

import torch
import torch.nn.functional as F

from sortnet_b200 import layers, ops
from sortnet_b200.optim import FlatAdamW

DEV = "cuda"


def _model(kind, rows, channels, side, classes, depth, width, keep, p, eps, **more):
    return dict(kind=kind, rows=rows, channels=channels, side=side, classes=classes, depth=depth, width=width,
                keep=keep, p=p, eps=eps, **more)


def listed():
    return [
        # the smallest call: one layer of odd sizes, distance and bounds with gradients; launches and host time count
        dict(name="layer_9x97x33", kind="layer", rows=9, inputs=97, outputs=33, p="inf", eps=0.1, bound_grad=True),
        # one l-inf layer of an MNIST net: forward, backward and interval bounds
        dict(name="layer_128x784x5120", kind="layer", rows=128, inputs=784, outputs=5120, p="inf", eps=0.3,
             bound_grad=False),
        # SortNet-MLP on CIFAR-10 in the last phase of its p schedule: masked forward, loss, sparse backward
        dict(name="train_cifar_inf", **_model("train", 512, 3, 32, 10, 6, 5120, 0.9, "inf", 8 / 255)),
        # the same on TinyImageNet: the widest first layer and a head of 200 classes
        dict(name="train_tiny_inf", **_model("train", 512, 3, 64, 200, 6, 5120, 0.9, "inf", 1 / 255)),
        # MNIST net on a ragged share of a batch, as one of several GPUs gets it: per-layer costs count
        dict(name="train_mnist_inf_67", **_model("train", 67, 1, 28, 10, 5, 5120, 0.7, "inf", 0.1)),
        # first phase of the schedule (p = 8): dense forward and backward
        dict(name="train_cifar_p8", **_model("train", 512, 3, 32, 10, 6, 5120, 0.75, "8", 2 / 255)),
        # middle of the schedule (p between 8 and infinity), where most epochs are spent
        dict(name="train_mnist_p31.6", **_model("train", 512, 1, 28, 10, 5, 5120, 0.75, "31.6", 0.3)),
        # certification of a pure l-inf-distance net: values and interval bounds, no gradients
        dict(name="certify_cifar_linf", **_model("certify", 512, 3, 32, 10, 7, 5120, 1.0, "inf", 2 / 255)),
        # certification of a SortNet: sort neurons and their bounds in every layer after the first
        dict(name="certify_cifar_sort", **_model("certify", 512, 3, 32, 10, 6, 5120, 0.75, "inf", 2 / 255)),
        # one step of a gradient attack on a SortNet, built from the operators: logits and the gradient of the image
        dict(name="attack_cifar_sort", **_model("attack", 128, 3, 32, 10, 6, 5120, 0.85, "inf", 8 / 255)),
        # patch convolution and a masked 1 x 1 layer, four positions each: forward and backward
        dict(name="conv_128x4x1024", kind="conv", rows=128, side=16, kernel=8, width=1024, groups=1, keep=0.75, p="inf"),
        # optimiser update of the CIFAR-10 net, 120.6 M parameters
        dict(name="update_cifar", **_model("update", 0, 3, 32, 10, 6, 5120, 0.9, "inf", 0.0)),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _width(rng, lo, hi):
    """Mostly round, as users choose them; odd now and then."""
    n = _log_int(rng, lo, hi)
    return n if rng.random() < 0.35 else max(64, n // 64 * 64)


def _draw_p(rng, whole):
    """infinity, one of the whole numbers, or a value on the way from 8 to 1000 (the schedules' range)."""
    pick = rng.random()
    if pick < 0.5:
        return "inf"
    if pick < 0.7:
        return str(rng.choice(whole))
    return "%.4g" % math.exp(rng.uniform(math.log(8.5), math.log(1000)))


def draw(rng):
    case = _draw_any(rng)
    most = max(work(c)["flops"] for c in listed())
    while work(case)["flops"] > most:
        case["rows"] = case["rows"] * 2 // 3
    return case


def _draw_any(rng):
    kind = rng.choice(["layer", "train", "train", "train", "certify", "certify", "attack", "conv", "update"])
    if kind == "layer":
        p = _draw_p(rng, [2, 3, 5, 8])
        return dict(kind=kind, rows=_log_int(rng, 4, 512), inputs=_width(rng, 64, 5120), outputs=_width(rng, 64, 5120),
                    p=p, eps=round(rng.uniform(0.01, 0.3), 3), bound_grad=rng.random() < 0.5)
    if kind == "conv":
        groups = rng.choice([1, 1, 3])
        kernel = rng.choice([3, 4, 5, 8])
        return dict(kind=kind, rows=_log_int(rng, 16, 192), side=kernel * rng.choice([1, 2, 3]), kernel=kernel,
                    width=_log_int(rng, 100, 1000) // groups * groups, groups=groups, keep=round(rng.uniform(0.6, 0.95), 2),
                    p=rng.choice(["inf", "8"]))
    channels, side = rng.choice([(1, 28), (3, 32), (3, 32), (3, 64), (1, rng.randint(9, 40)), (3, rng.randint(9, 40))])
    rows = _log_int(rng, 24, 512)
    keep = 1.0 if rng.random() < 0.2 else round(rng.uniform(0.65, 0.95), 3)
    p = _draw_p(rng, [8]) if kind == "train" else "inf"
    if kind == "update":
        rows = 0
    return _model(kind, rows, channels, side, rng.choice([10, 10, 100, 200]), rng.randint(4, 6), _width(rng, 500, 5120),
                  keep, p, round(rng.choice([1 / 255, 2 / 255, 8 / 255, 0.1]), 5))


# ---- inputs -------------------------------------------------------------------------------------


def _images(gen, rows, channels, side):
    coarse = torch.rand(rows, channels, 4, 4, device=DEV, generator=gen)
    x = F.interpolate(coarse, size=(side, side), mode="bilinear", align_corners=False)
    light = 0.6 * torch.rand(rows, 1, 1, 1, device=DEV, generator=gen) - 0.3
    noise = 0.2 * torch.rand(rows, channels, side, side, device=DEV, generator=gen) - 0.1
    return (x + light + noise).clamp_(0, 1)


def _build_model(case):
    with torch.device(DEV):
        model = layers.SortMLPModel(depth=case["depth"], width=case["width"],
                                    input_dim=(case["channels"], case["side"], case["side"]), num_classes=case["classes"],
                                    dropout=case["keep"])
    model.set_p(float(case["p"]))
    return model


def _settle_means(model, x):
    """Running means as training leaves them: those of one pass over the batch."""
    layers.update_running_means(model, [x])


def prepare(case, seed):
    torch.manual_seed(seed)
    gen = torch.Generator(device=DEV).manual_seed(seed + 1)
    kind = case["kind"]
    if kind == "layer":
        rows, inputs, outputs = case["rows"], case["inputs"], case["outputs"]
        x = torch.rand(rows, inputs, 1, device=DEV, generator=gen)
        w = torch.randn(outputs, inputs, device=DEV, generator=gen)
        lower, upper = (x - case["eps"]).clamp(0, 1), (x + case["eps"]).clamp(0, 1)
        grads = [torch.randn(rows, outputs, 1, device=DEV, generator=gen) for _ in range(3)]
        for t in (x, w) + ((lower, upper) if case["bound_grad"] else ()):
            t.requires_grad_()
        return dict(kind=kind, p=float(case["p"]), bound_grad=case["bound_grad"], x=x, w=w, lower=lower, upper=upper,
                    grads=grads)
    if kind == "conv":
        k, width, groups, p = case["kernel"], case["width"], case["groups"], float(case["p"])
        with torch.device(DEV):
            first = layers.NormDistConv(3, width, k, stride=k, groups=groups, bias=False, p=p)
            second = layers.NormDistConv(width, width, 1, groups=groups, bias=True, dropout=case["keep"], p=p)
        x = _images(gen, case["rows"], 3, case["side"])
        grad = torch.randn(case["rows"], width, case["side"] // k, case["side"] // k, device=DEV, generator=gen)
        return dict(kind=kind, x=x, grad=grad, first=first, second=second, width=width, groups=groups, keep=case["keep"],
                    mask_seed=seed)
    model = _build_model(case)
    state = dict(kind=kind, model=model, eps=case["eps"], mask_seed=seed)
    if kind == "update":
        state["opt"] = FlatAdamW(model, lr=0.02, betas=(0.9, 0.99), eps=1e-10)
        # gradients of a p = inf step: a few entries per row of a weight matrix, zeros elsewhere
        grad = state["opt"].flat_grad
        grad.normal_(std=1e-3, generator=gen)
        grad.mul_(torch.rand(grad.shape, device=DEV, generator=gen) < 0.1)
        return state
    x = _images(gen, case["rows"], case["channels"], case["side"])
    state["targets"] = torch.randint(0, case["classes"], (case["rows"],), device=DEV, generator=gen)
    if kind == "train":
        model.train()
        state["opt"] = FlatAdamW(model, lr=0.02, betas=(0.9, 0.99), eps=1e-10)
    else:
        _settle_means(model, x)
        model.eval()
    if kind == "attack":
        model.requires_grad_(False)        # only the image moves
        x.requires_grad_()
    state["x"] = x
    return state


# ---- one pass -----------------------------------------------------------------------------------


def _run_layer(s):
    y = ops.norm_dist(s["x"], s["w"], s["p"])
    out = [y, *torch.autograd.grad(y, (s["x"], s["w"]), s["grads"][0])]
    if s["bound_grad"]:
        yl, yu = ops.bound_inf_dist(s["lower"], s["upper"], s["w"])
        return out + [yl, yu, *torch.autograd.grad((yl, yu), (s["lower"], s["upper"], s["w"]), s["grads"][1:])]
    with torch.no_grad():
        return out + list(ops.bound_inf_dist(s["lower"], s["upper"], s["w"]))


def _run_conv(s):
    torch.manual_seed(s["mask_seed"])
    sub = (s["x"].size(0) + layers.SUB_BATCH - 1) // layers.SUB_BATCH
    mask = layers.sample_mask(sub, s["groups"], s["width"] // s["groups"], s["keep"], DEV)
    hidden = s["first"](s["x"], mask_out=mask)[0]
    y = s["second"](hidden, mask_in=mask)[0]
    weights = (s["first"].weight, s["second"].weight, s["second"].bias)
    return [y, *torch.autograd.grad(y, weights, s["grad"])]


def _run_train(s):
    torch.manual_seed(s["mask_seed"])      # the masks of the pass
    opt = s["opt"]
    loss = s["model"].mixture_loss(s["x"], s["targets"], s["eps"])
    opt.zero_grad()
    loss.backward()
    opt.gather_grads()
    return [loss, opt.flat_grad] + [m.running_mean for m in s["model"].modules() if isinstance(m, layers.MeanShiftDropout)]


def _run_certify(s):
    with torch.no_grad():
        return s["model"](s["x"], s["targets"], s["eps"], up=1.0, down=0.0)


def _run_attack(s):
    z = s["x"].flatten(1).unsqueeze(-1)
    for layer in s["model"].fc_dist:
        z = ops.sort_neuron(z, layer.weight, q=layer.dropout)
        if layer.mean_shift is not None:
            z = z - layer.mean_shift.running_mean.view(1, -1, 1)
        if layer.bias is not None:
            z = z + layer.bias.view(1, -1, 1)
    logits = -z.squeeze(-1)
    loss = F.cross_entropy(logits, s["targets"])
    return [logits, *torch.autograd.grad(loss, s["x"])]


def _run_update(s):
    opt = s["opt"]
    opt.set_flat_grad()                    # the gradients in the flat buffer are this step's
    opt.step()
    return [opt.flat_param, opt.exp_avg, opt.exp_avg_sq]


_RUN = dict(layer=_run_layer, conv=_run_conv, train=_run_train, certify=_run_certify, attack=_run_attack,
            update=_run_update)


def run(state):
    return _RUN[state["kind"]](state)


# ---- work and tolerance -------------------------------------------------------------------------


def _ops(p):
    """Operations of one (row, output, input) term of the forward, and of the dense backward."""
    if math.isinf(p):
        return 2, 0
    if p == int(p) and p <= 8:
        return 2 + int(p).bit_length(), 4 + int(p).bit_length()
    return 5, 7


def _mlp_shapes(case):
    pixels = case["channels"] * case["side"] * case["side"]
    dims = [pixels] + [case["width"]] * (case["depth"] - 1) + [case["classes"]]
    return [(dims[k], dims[k + 1]) for k in range(case["depth"])]


def work(case):
    kind, rows, p = case["kind"], case["rows"], float(case["p"])
    fwd, bwd = _ops(p)
    if kind == "layer":
        ci, co = case["inputs"], case["outputs"]
        bound_words = 5 * rows * ci + 4 * rows * co + co * ci if case["bound_grad"] else 2 * rows * ci + 2 * rows * co
        words = 2 * (rows * ci + co * ci) + 2 * rows * co + bound_words
        return dict(bytes=4 * words, flops=(fwd + bwd + 6) * rows * ci * co)
    if kind == "conv":
        places = (case["side"] // case["kernel"]) ** 2
        width, groups, keep = case["width"], case["groups"], case["keep"]
        fan = 3 // groups * case["kernel"] ** 2
        weights = width * fan + width * width // groups
        terms = rows * places * keep * weights
        return dict(bytes=4 * (2 * weights + rows * (3 * case["side"] ** 2 + 2 * width * places)), flops=(fwd + bwd) * terms)
    shapes = _mlp_shapes(case)
    params = sum(ci * co for ci, co in shapes) + case["classes"]
    if kind == "update":
        return dict(bytes=28 * params, flops=12 * params)
    keep = case["keep"]
    image = rows * shapes[0][0]
    terms = kept = 0.0
    for k, (ci, co) in enumerate(shapes):
        part = (1 if k == 0 else keep) * (1 if k == len(shapes) - 1 else keep)
        kept += rows * part * ci * co
        terms += rows * ci * co
    if kind == "train":
        return dict(bytes=4 * (2 * params + image), flops=(fwd + bwd) * kept)
    if kind == "certify":
        return dict(bytes=4 * (params + image + 2 * rows * case["classes"]), flops=8 * terms)
    return dict(bytes=4 * (params + 2 * image + rows * case["classes"]), flops=2 * terms)


def tolerance(case):
    p = float(case["p"])
    if math.isinf(p):
        return {"rel": 1e-5, "max": 2e-3}  # fp32 sums in another order; maxima and their places are exact
    # the backward raises fp32 ratios to the power p - 1, layer after layer; where large gradients cancel
    # the rounding of their sum shows against a small result
    return {"rel": 2e-5 if p <= 8 else 1e-4, "max": 1e-2}
