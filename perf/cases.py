"""The work that users of this package have it do, as cases that can be timed and compared.

A case is a dict of plain values.  ``listed()`` names the ones that are always looked at, ``draw(rng)`` gives
another one of the same ranges, ``prepare`` makes what a program holds before the call, ``run`` is one pass
through the public entry points, ``work`` is what a pass cannot do without and ``tolerance`` how far two correct
implementations at the same precision may lie apart.

Images are the package's synthetic stand-ins for MNIST (28x28, strokes on a zero canvas, uint8 / 255); the widened
net gets 56x56 images of the same sparsity.  Parameters are drawn as the reference draws them (uniform in
[-0.5, 0.5]); the widened net's 10,816-term output layer is scaled so that its sigmoids do not saturate.
"""
import math

import numpy as np
import torch

import __graft_entry__ as entry

pkg = entry.load_package()

DT = 0.1                        # the reference's step size
WIDE_H, WIDE_F = 56, 64         # the widened net of benchmark configuration 5
N_PARAMS = pkg.N_PARAMS
CONV = {"fp32": 0, "tf32": 1, "3xtf32": 2}


def listed():
    return [
        # one image, as the reference's classify() takes it: launch latency and nothing else
        {"name": "forward_1", "call": "forward", "n": 1, "pixels": "fp32", "precision": "default"},
        # the 2,000-image test set of benchmark configuration 1 (a serving batch of ordinary size)
        {"name": "forward_2000", "call": "forward", "n": 2000, "pixels": "fp32", "precision": "default"},
        # bulk inference, benchmark configuration 2
        {"name": "forward_65536", "call": "forward", "n": 65536, "pixels": "fp32", "precision": "default"},
        # bulk inference on pixels as the IDX files store them, already on the GPU, a ragged count
        {"name": "forward_u8_30011", "call": "forward", "n": 30011, "pixels": "uint8", "precision": "default"},
        # bulk inference in the reduced precision that a caller can ask for
        {"name": "forward_reduced_65536", "call": "forward", "n": 65536, "pixels": "fp32", "precision": "reduced"},
        # the reference's test(): 10,000 images straight from the file in ordinary host memory, results on the host
        {"name": "forward_host_10000", "call": "forward_host", "n": 10000, "pixels": "uint8", "pinned": False},
        # one gradient step of a caller's own training loop at the batch of benchmark configuration 4
        {"name": "step_256", "call": "step", "n": 256},
        # one full-batch gradient step over an MNIST-sized training set
        {"name": "step_60000", "call": "step", "n": 60000},
        # one epoch of minibatch SGD, benchmark configuration 4
        {"name": "minibatch_60000", "call": "minibatch", "n": 60000, "batch": 256},
        # one epoch of the reference's own per-sample SGD, benchmark configuration 1
        {"name": "persample_10000", "call": "persample", "n": 10000},
        # the widened net: inference as it comes (fp32 convolution), a ragged batch of ordinary size
        {"name": "wide_forward_333", "call": "wide_forward", "n": 333, "conv": "fp32"},
        # the widened net: forward and backward on the tensor cores, benchmark configuration 5
        {"name": "wide_grad_1024", "call": "wide_grad", "n": 1024, "conv": "3xtf32"},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    call = rng.choice(["forward", "forward", "forward", "forward_host", "step", "step", "minibatch", "persample",
                       "wide_forward", "wide_grad"])
    if call == "forward":
        pixels = rng.choice(["fp32", "fp32", "uint8"])
        return {"call": call, "n": _log_int(rng, 1, 65536), "pixels": pixels,
                "precision": rng.choice(["default", "default", "reduced"]) if pixels == "fp32" else "default"}
    if call == "forward_host":
        return {"call": call, "n": _log_int(rng, 100, 20000), "pixels": rng.choice(["uint8", "fp32"]),
                "pinned": rng.random() < 0.5}
    if call == "step":
        return {"call": call, "n": _log_int(rng, 1, 60000)}
    if call == "minibatch":
        batch = _log_int(rng, 16, 1024)
        return {"call": call, "n": min(60000, batch * rng.randint(8, 235) + rng.randrange(batch)), "batch": batch}
    if call == "persample":
        return {"call": call, "n": _log_int(rng, 500, 10000)}
    conv = rng.choice(["fp32", "tf32", "3xtf32"])
    return {"call": call, "n": _log_int(rng, 1, 320 if conv == "fp32" else 1024), "conv": conv}


class _DeviceView:
    """The net's own parameter arena as something that torch can look at without a copy.  The tensor keeps this
    object, and with it the net that owns the memory."""

    def __init__(self, net):
        self.net = net
        self.__cuda_array_interface__ = {"shape": (N_PARAMS,), "typestr": "<f4", "version": 3,
                                         "data": (net.params_device_ptr(), False)}


def _params_of(net):
    return torch.as_tensor(_DeviceView(net), device="cuda")


def _images(seed, n):
    images = torch.empty((n, 28, 28), dtype=torch.float32, device="cuda")
    labels = torch.empty(n, dtype=torch.int32, device="cuda")
    pkg.synth_images_device(seed, 0, n, images, labels)
    return images, labels


def _wide_params(net, gen):
    p = torch.rand(net.n_params, device="cuda", generator=gen) - 0.5
    first = WIDE_F * 26 + 17
    fc = net.n_params - first - 10
    p[first:first + fc] *= 6.0 / math.sqrt(fc / 10)
    return p.cpu().numpy()


def prepare(case, seed):
    call, n = case["call"], case["n"]
    st = {"call": call, "n": n}
    if call.startswith("wide"):
        gen = torch.Generator("cuda").manual_seed(seed)
        shape = (n, WIDE_H, WIDE_H)
        st["images"] = (torch.rand(shape, device="cuda", generator=gen)
                        * (torch.rand(shape, device="cuda", generator=gen) < 0.2)).contiguous()
        st["labels"] = torch.randint(0, 10, (n,), dtype=torch.int32, device="cuda", generator=gen)
        net = pkg.WideNet(WIDE_H, WIDE_F)
        net.set_params(_wide_params(net, gen))
        net.set_option("conv", CONV[case["conv"]])
        st["grad"] = torch.empty(net.n_padded, dtype=torch.float32, device="cuda")
    else:
        st["images"], st["labels"] = _images(seed, n)
        net = pkg.Net(seed)
        st["params"] = _params_of(net)
        st["grad"] = torch.empty(pkg.N_PARAMS_PADDED, dtype=torch.float32, device="cuda")
    st["net"] = net
    if "forward" in call:
        if case.get("pixels") == "uint8":
            st["images"] = (st["images"] * 255.0).round().to(torch.uint8)
        st["out"] = torch.empty((n, 10), dtype=torch.float32, device="cuda")
        st["argmax"] = torch.empty(n, dtype=torch.int32, device="cuda")
    if call == "forward":
        if case["precision"] == "reduced":
            net.set_option("forward_path", 2)
        st["fn"] = net.forward_u8 if case["pixels"] == "uint8" else net.forward
    elif call == "forward_host":
        host = [st[k].cpu() for k in ("images", "out", "argmax")]
        if case["pinned"]:
            host = [t.pin_memory() for t in host]
        st["keep"] = host
        st["images"], st["out"], st["argmax"] = (t.numpy() for t in host)
        st["fn"] = net.forward_u8_host if case["pixels"] == "uint8" else net.forward_host
    elif call == "minibatch":
        st["batch"] = case["batch"]
        st["mean_err"] = torch.empty(1, dtype=torch.float32, device="cuda")
    return st


def run(st):
    net, call, n = st["net"], st["call"], st["n"]
    if call in ("forward", "forward_host"):
        st["fn"](st["images"], n, st["out"], st["argmax"])
        return st["out"], st["argmax"]
    if call == "step":
        net.grad_batch(st["images"], st["labels"], n, st["grad"])
        net.apply_update(st["grad"], DT / n)
        return st["grad"], st["params"]
    if call == "minibatch":
        net.train_minibatch(st["images"], st["labels"], n, st["batch"], 1, DT, st["mean_err"])
        return st["params"], st["mean_err"]
    if call == "persample":
        _, mean_err = net.train_sgd_persample(st["images"], st["labels"], n, 1, DT)
        return st["params"], np.array(mean_err)
    if call == "wide_forward":
        net.forward(st["images"], n, st["out"], st["argmax"])
        return st["out"], st["argmax"]
    net.grad_batch(st["images"], st["labels"], n, st["grad"])
    return st["grad"]


def work(case):
    n = case["n"]
    if case["call"].startswith("wide"):
        conv = WIDE_H - 4
        windows = WIDE_F * (conv // 4) ** 2
        params = WIDE_F * 26 + 17 + 10 * windows + 10
        macs = conv * conv * WIDE_F * 25 + 16 * windows + 10 * windows       # convolution, subsample, output layer
        if case["call"] == "wide_forward":
            return {"bytes": n * (4 * WIDE_H * WIDE_H + 44) + 4 * params, "flops": n * 2 * macs}
        return {"bytes": n * (4 * WIDE_H * WIDE_H + 4) + 8 * params, "flops": n * 18992896}
    if case["call"].startswith("forward"):
        pixel = 1 if case["pixels"] == "uint8" else 4
        return {"bytes": n * (784 * pixel + 44) + 4 * N_PARAMS, "flops": n * 184032}
    return {"bytes": n * 3140 + 8 * N_PARAMS, "flops": n * 379296}


def tolerance(case):
    call = case["call"]
    if call.startswith("wide"):
        if case["conv"] == "tf32":      # operands of ten mantissa bits; sums over images partly cancel in a gradient
            return {"rel": 1e-2, "differ": 1e-2} if call == "wide_grad" else {"rel": 2e-3, "differ": 1e-2}
        return {"rel": 2e-5, "differ": 3e-3}
    if call.startswith("forward"):
        if case.get("precision") == "reduced":      # ten mantissa bits and an approximate sigmoid
            return {"rel": 1e-3, "differ": 3e-3}
        return {"rel": 1e-5, "differ": 1e-3}
    if call == "step":
        return {"rel": 1e-5}
    return {"rel": 2e-5}        # rounding compounds along a chain of steps
