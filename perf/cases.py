"""The calls that a training or inference program makes of this library, with sizes, as measurable cases.

A case is a dict of plain values.  `prepare` builds what such a program has in hand before the call (network, optimizer,
input tensors on the device), `run` makes one pass through the nc_* C API and returns views of everything the pass
produced, `work` says what the pass cannot do without, `tolerance` how far two correct implementations may be apart.

Kinds:
  train  one full step (zero_grad, forward, loss, backward, optimizer step) of one of the four trainable networks of
         nocta_b200.configs
  eval   the same networks' forward pass in evaluation mode with gradients off, then the row argmax
  conv   nc_conv2d forward and nc_backward of one layer whose input needs a gradient, operands in dense (N, C, H, W)
         order as a caller hands them over
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from nocta_b200 import capi, configs

# nc_cuda_set_math_mode values that programs select: the default, and the one for tighter accuracy
MODES = {"tf32": 0, "3xtf32": 2}


def listed():
    return [
        # a hand-written digit at a time through the small network: the shortest call there is
        {"name": "lenet_eval_b1", "kind": "eval", "net": "lenet", "batch": 1, "mode": "tf32"},
        # LeNet-style CNN of the MNIST example, batch 64, SGD with momentum: many very short kernels
        {"name": "lenet_train_b64", "kind": "train", "net": "lenet", "batch": 64, "mode": "tf32"},
        # conv-BatchNorm CNN on 32 x 32 images, batch 128, AdamW
        {"name": "convbn_train_b128", "kind": "train", "net": "convbn", "batch": 128, "mode": "tf32"},
        # VGG-style CNN on 64 x 64 images at the batch it is benchmarked at
        {"name": "vgg_train_b256", "kind": "train", "net": "vgg", "batch": 256, "size": 64, "base": 64, "classes": 100, "mode": "tf32"},
        # the same family where nothing is a power of two: an image size that pools down to odd extents, widths of 48 / 96 / 192
        # and the odd batch that ends an epoch
        {"name": "vgg_train_ragged", "kind": "train", "net": "vgg", "batch": 37, "size": 44, "base": 48, "classes": 257, "mode": "tf32"},
        # the accuracy option: three TF32 products per contraction
        {"name": "vgg_train_3xtf32_b64", "kind": "train", "net": "vgg", "batch": 64, "size": 64, "base": 64, "classes": 100, "mode": "3xtf32"},
        # validation pass over a batch of images
        {"name": "vgg_eval_b200", "kind": "eval", "net": "vgg", "batch": 200, "size": 64, "base": 64, "classes": 100, "mode": "tf32"},
        # residual MLP stack (1024 -> 4096 -> 1024, four blocks), batch 4096, Adam: the largest matrices
        {"name": "mlp_train_b4096", "kind": "train", "net": "mlp", "batch": 4096, "width": 1024, "hidden": 4096, "blocks": 4, "mode": "tf32"},
        # tabular data: a feature count that is no multiple of four, and a batch that is no multiple of anything
        {"name": "mlp_train_ragged", "kind": "train", "net": "mlp", "batch": 1001, "width": 310, "hidden": 1250, "blocks": 2, "mode": "tf32"},
        # serving the MLP stack to a handful of requests
        {"name": "mlp_eval_b16", "kind": "eval", "net": "mlp", "batch": 16, "width": 1024, "hidden": 4096, "blocks": 4, "mode": "tf32"},
        # the isolated 3 x 3 convolution layer, forward and all three gradients
        {"name": "conv_3x3_b256", "kind": "conv", "batch": 256, "cin": 64, "cout": 64, "size": 56, "k": 3, "stride": 1, "pad": 1, "mode": "tf32"},
        # a strided 3 x 3 layer, as used between the stages of a network
        {"name": "conv_3x3_stride2_b32", "kind": "conv", "batch": 32, "cin": 64, "cout": 128, "size": 56, "k": 3, "stride": 2, "pad": 1, "mode": "tf32"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choice(["lenet_train", "lenet_eval", "convbn_train", "vgg_train", "vgg_train_3x", "vgg_eval", "mlp_train", "mlp_train_3x",
                       "mlp_eval", "conv", "conv_strided"])
    if what == "lenet_eval":
        return {"kind": "eval", "net": "lenet", "batch": _log_int(rng, 3, 768), "mode": "tf32"}
    if what == "lenet_train":
        return {"kind": "train", "net": "lenet", "batch": _log_int(rng, 4, 768), "mode": "tf32"}
    if what == "convbn_train":
        return {"kind": "train", "net": "convbn", "batch": _log_int(rng, 8, 512), "mode": "tf32"}
    if what in ("vgg_train", "vgg_train_3x", "vgg_eval"):
        three = what == "vgg_train_3x"
        base = rng.choice([32, 48, 64])
        top = 64 if three else 192
        if base == 48:
            top //= 4
        return {"kind": "eval" if what == "vgg_eval" else "train", "net": "vgg", "batch": _log_int(rng, 4, top), "size": rng.randint(16, 64),
                "base": base, "classes": _log_int(rng, 10, 1000), "mode": "3xtf32" if three else "tf32"}
    if what in ("mlp_train", "mlp_train_3x"):
        three = what == "mlp_train_3x"
        even = rng.random() < 0.6   # most programs pick widths that are multiples of a small power of two
        width, hidden = _log_int(rng, 64, 1024), _log_int(rng, 256, 4096)
        if even:
            width, hidden = (width + 7) // 8 * 8, (hidden + 7) // 8 * 8
        batch, blocks = _log_int(rng, 64, 4096), rng.randint(1, 4)
        most = 2.0e11 if three else (6.0e11 if even else 3.0e10)   # FLOPs of a step
        batch = max(48, min(batch, int(most / (12.0 * width * hidden * blocks))))
        return {"kind": "train", "net": "mlp", "batch": batch, "width": width, "hidden": hidden, "blocks": blocks,
                "mode": "3xtf32" if three else "tf32"}
    if what == "mlp_eval":
        return {"kind": "eval", "net": "mlp", "batch": _log_int(rng, 1, 256), "width": (_log_int(rng, 64, 1024) + 3) // 4 * 4,
                "hidden": (_log_int(rng, 256, 4096) + 3) // 4 * 4, "blocks": rng.randint(1, 4), "mode": "tf32"}
    stride = 2 if what == "conv_strided" else 1
    k = rng.choice([1, 3, 3, 3, 5])
    cin, cout, size = rng.choice([32, 48, 64, 96, 128, 256]), rng.choice([32, 64, 96, 128, 256]), rng.randint(14, 64)
    out = (size + 2 * (k // 2) - k) // stride + 1
    # the strided layer costs more for its size: keep it below the largest listed case
    most = (1.2e11 if stride == 1 else 8.0e9) / (6.0 * out * out * cin * cout * k * k)
    batch = max(1, min(_log_int(rng, 2, 256), int(most)))
    return {"kind": "conv", "batch": batch, "cin": cin, "cout": cout, "size": size, "k": k, "stride": stride, "pad": k // 2, "mode": "tf32"}


# ----------------------------------------------------------------------------------------------
# state
# ----------------------------------------------------------------------------------------------
_api = None
_runner = None


def _library():
    global _api, _runner
    if _runner is None:
        _api = configs.load_library()
        _runner = configs.Runner(_api, on_device=True)
        _api.lib.nc_cuda_set_math_mode.restype = C.c_int
        _api.lib.nc_cuda_set_math_mode.argtypes = [C.c_int]
    return _api, _runner


_TYPES = {capi.NC_F32: ("<f4", 4), capi.NC_I64: ("<i8", 8)}


class _Memory:
    def __init__(self, pointer, shape, strides, kind):
        self.__cuda_array_interface__ = {"data": (pointer, False), "shape": shape, "strides": strides, "typestr": kind, "version": 2}


class State:
    """A network (or one layer) with its inputs, and the torch views of library tensors it has handed out."""

    def __init__(self, case):
        self.case = case
        self.views = {}
        self.net = self.forward = self.loss_kind = self.tensors = None
        self.params = []      # every parameter, running statistics among them
        self.trained = []     # those that get a gradient
        self.param_views = []
        self.tensors_to_free = []
        self.step = []        # outputs of the last pass, kept until the next one
        self.layer = self.x = self.grad_output = None

    def view(self, t):
        """The device tensor `t` as a torch tensor on the same memory (made once for each place)."""
        tt = t.contents
        kind, size = _TYPES[tt.dtype]
        pointer = tt.storage.contents.cuda_data + tt.offset * size
        v = self.views.get((pointer, tt.numel))
        if v is None:
            shape = tuple(tt.shape[i] for i in range(tt.ndim))
            strides = tuple(tt.strides[i] * size for i in range(tt.ndim))
            v = torch.as_tensor(_Memory(pointer, shape, strides, kind), device="cuda")
            if len(self.views) < 512:
                self.views[(pointer, tt.numel)] = v
        elif tuple(v.shape) != tuple(tt.shape[i] for i in range(tt.ndim)):
            v = v.as_strided(tuple(tt.shape[i] for i in range(tt.ndim)), tuple(tt.strides[i] for i in range(tt.ndim)))
        return v

    def release_step(self):
        for t in self.step:
            _api.nc_tensor_free(t)
        self.step = []

    def __del__(self):
        if _api is None or torch is None:
            return
        if self.net is not None:
            self.net.free_step_tensors()
        self.release_step()
        if self.net is not None:
            if self.net.optimizer:
                _api.nc_optimizer_free(self.net.optimizer)
            for m in self.net.modules.values():
                _api.nc_module_free(m)
        if self.layer is not None:
            _api.nc_module_free(self.layer)
        for t in self.tensors_to_free:
            _api.nc_tensor_free(t)


def _build(case, seed):
    api, r = _library()
    net = case["net"]
    if net == "lenet":
        built = configs.build_lenet(r, seed=seed)
    elif net == "convbn":
        built = configs.build_convbn(r, seed=seed, batch=case["batch"])
    elif net == "vgg":
        b = case["base"]
        built = configs.build_vgg(r, seed=seed, batch=case["batch"], classes=case["classes"], size=case["size"], widths=(b, 2 * b, 4 * b))
    else:
        built = configs.build_mlp(r, seed=seed, batch=case["batch"], width=case["width"], hidden=case["hidden"], blocks=case["blocks"])
    net_, forward, loss_kind, data = built
    if net == "lenet":   # its builder makes 64 images
        rng = np.random.default_rng(seed + 1)
        data = (rng.random((case["batch"], 1, 28, 28), dtype=np.float32), rng.integers(0, 10, case["batch"]).astype(np.int64))
    # normalisation layers as they are in the middle of training, not at their initial ones and zeros
    rng = np.random.default_rng(seed + 2)
    for m in net_.modules.values():
        named = dict(api.module_params(m))
        vector = lambda t, lo, hi: r.load(t, rng.uniform(lo, hi, t.contents.numel).astype(np.float32))  # noqa: E731
        if named["weight"].contents.ndim == 1:
            vector(named["weight"], 0.7, 1.3)
            vector(named["bias"], -0.3, 0.3)
            if "running_mean" in named:
                vector(named["running_mean"], -0.2, 0.2)
                vector(named["running_var"], 0.5, 1.5)
    return net_, forward, loss_kind, data


def prepare(case, seed):
    api, r = _library()
    api.lib.nc_cuda_set_math_mode(MODES[case["mode"]])
    seed = seed & 0x7FFFFFFF
    s = State(case)
    if case["kind"] == "conv":
        g = torch.Generator(device="cuda").manual_seed(seed)
        size, k, stride, pad = case["size"], case["k"], case["stride"], case["pad"]
        out = (size + 2 * pad - k) // stride + 1

        def tensor(shape):
            t = api.nc_tensor_empty(capi.shape_arr(shape), len(shape), capi.NC_F32)
            s.view(t).copy_(torch.randn(shape, generator=g, device="cuda"))
            s.tensors_to_free.append(t)
            return t

        s.x = tensor((case["batch"], case["cin"], size, size))
        s.grad_output = tensor((case["batch"], case["cout"], out, out))
        api.nc_tensor_requires_grad_(s.x, True)
        s.layer = api.nc_conv2d(case["cin"], case["cout"], k, stride, pad, True)
        named = dict(api.module_params(s.layer))
        scale = math.sqrt(2.0 / (case["cin"] * k * k))
        s.view(named["weight"]).copy_(torch.randn((case["cout"], case["cin"], k, k), generator=g, device="cuda") * scale)
        s.view(named["bias"]).copy_(torch.randn((case["cout"],), generator=g, device="cuda") * 0.1)
        s.trained = [named["weight"], named["bias"]]
        return s
    s.net, s.forward, s.loss_kind, data = _build(case, seed)
    for m in s.net.modules.values():
        for name, p in api.module_params(m):
            s.params.append(p)
            s.param_views.append(s.view(p))
            if not name.startswith("running"):
                s.trained.append(p)
    if case["kind"] == "train":
        s.tensors = configs.upload(r, s.loss_kind, data)
    else:
        for m in s.net.modules.values():
            api.nc_module_train(m, False)
        # dropout is off in evaluation: its mask is all ones
        s.tensors = [r.tensor(data[0])] + ([[r.tensor(np.ones_like(m)) for m in data[2]]] if s.loss_kind == "mse" else [])
    for t in s.tensors:
        s.tensors_to_free += t if isinstance(t, list) else [t]
    return s


# ----------------------------------------------------------------------------------------------
# one pass
# ----------------------------------------------------------------------------------------------
def run(s):
    api, r = _api, _runner
    if s.case["kind"] == "train":
        s.net.free_step_tensors()
        loss = configs.train_step(r, s.net, s.forward, s.loss_kind, s.tensors)
        out = [s.view(loss)] + s.param_views
        if s.case["net"] in ("lenet", "mlp"):
            # The gradients that reach the first layers through several BatchNorm and ReLU layers are not reproducible to better
            # than a few percent between two correct orders of summation, in TF32 mode: sums with heavy cancellation over
            # entries that a turned ReLU switches on or off.  Of those networks the pass hands out what it leaves behind: the
            # updated parameters and running statistics.
            out += [s.view(p.contents.grad) for p in s.trained]
        return out
    if s.case["kind"] == "eval":
        s.net.free_step_tensors()
        api.nc_set_grad_enabled(0)
        logits = s.forward(s.net, *s.tensors)
        best = api.nc_argmax(logits, 1, False)
        api.nc_set_grad_enabled(1)
        s.net.keep.append(best)
        return [s.view(logits), s.view(best)]
    s.release_step()
    api.nc_tensor_zero_grad_(s.x)
    api.nc_module_zero_grad(s.layer)
    y = api.nc_module_forward(s.layer, s.x)
    s.step.append(y)
    if api.nc_backward(y, s.grad_output) != 0:
        raise RuntimeError("nc_backward failed")
    return [s.view(y), s.view(s.x.contents.grad)] + [s.view(p.contents.grad) for p in s.trained]


# ----------------------------------------------------------------------------------------------
# what a pass cannot do without
# ----------------------------------------------------------------------------------------------
def _network(case):
    """(multiply-adds of the forward pass, of those without an input gradient, parameters, input values, output values)"""
    n, net = case["batch"], case["net"]
    if net == "lenet":
        first = 6 * 25 * 24 * 24
        return n * (first + 16 * 150 * 64 + 256 * 120 + 120 * 84 + 840), n * first, 44426, n * 784, n * 10
    if net == "convbn":
        first = 64 * 27 * 1024
        return n * (first + 128 * 576 * 256 + 81920), n * first, 64 * 27 + 128 * 576 + 4 * 192 + 81930, n * 3072, n * 10
    if net == "vgg":
        macs = first = params = 0
        cin, size = 3, case["size"]
        for width in (case["base"], 2 * case["base"], 4 * case["base"]):
            for _ in range(2):
                m = n * size * size * cin * width * 9
                first = first or m
                macs += m
                params += cin * width * 9 + 2 * width
                cin = width
            size //= 2
        features = cin * size * size
        return (macs + n * features * case["classes"], first, params + (features + 1) * case["classes"], n * 3 * case["size"] ** 2,
                n * case["classes"])
    w, h, b = case["width"], case["hidden"], case["blocks"]
    # every block also has a mask, and a training step a regression target
    return n * 2 * w * h * b, 0, b * (2 * w * h + h + 3 * w), n * w * (b + 1 + (case["kind"] == "train")), n * w


def work(case):
    if case["kind"] == "conv":
        out = (case["size"] + 2 * case["pad"] - case["k"]) // case["stride"] + 1
        macs = case["batch"] * out * out * case["cin"] * case["cout"] * case["k"] ** 2
        nx, ny = case["batch"] * case["cin"] * case["size"] ** 2, case["batch"] * case["cout"] * out * out
        nw = case["cin"] * case["cout"] * case["k"] ** 2 + case["cout"]
        # x, dy, w read; y, dx, dw, db written
        return {"bytes": 4 * (2 * nx + 2 * ny + 2 * nw), "flops": 6 * macs}
    macs, first, params, inputs, outputs = _network(case)
    if case["kind"] == "eval":
        return {"bytes": 4 * (inputs + params + outputs) + 8 * case["batch"], "flops": 2 * macs}
    # the input, the parameters and the optimizer's moments (SGD: one, Adam: two) read, the parameters, the moments and the
    # gradients written; a layer without an input gradient saves a third of its products
    moments = 2 if case["net"] in ("convbn", "mlp") else 1
    return {"bytes": 4 * inputs + 4 * params * (3 + 2 * moments), "flops": 6 * macs - 2 * first}


def tolerance(case):
    """TF32 keeps 11 significant bits of each operand, 3xTF32 about 21; sums are f32 or wider in both.  Two orders of summation
    differ by 1e-7 at first, but in TF32 mode activations are rounded to 11 bits where they are stored, and such a difference
    turns the rounding of a few of them; behind a ReLU or a max-pool it turns a few decisions.  The figures are a small multiple
    of what perturbing the input by that much does."""
    three = case["mode"] == "3xtf32"
    if case["kind"] == "conv":
        return {"rel": 1e-3}
    if case["kind"] == "eval":
        return {"rel": 2e-3, "differ": 0.01}
    if case["net"] == "mlp":
        # max: Adam's first step is lr times the sign of the gradient, whatever its size
        return {"rel": 1e-4, "max": 0.1} if three else {"rel": 3e-3, "max": 0.12}
    if case["net"] == "lenet":
        return {"rel": 5e-3}      # one pooling decision in 55 000 already moves a gradient by 2e-3
    if case["net"] == "convbn":
        return {"rel": 5e-3, "max": 0.8}    # AdamW, as above
    return {"rel": 3e-4} if three else {"rel": 1.5e-3}
