"""The workloads that this framework's speed is judged on, each one pass through its public entry points.

Five kinds of work, as users of the registries and of the operator layer have it done:

  classify   zoo.load(model, "b200").model(images) -> fp32 logits
  features   backbones.build(model, "b200").fn(images) -> fp32 feature map
  classmap   seg.build(model, "b200").predict(images) -> int32 class map at the image's size
  scores     seg.build(model, "b200").logits(images) -> fp32 class scores at an eighth of the image's size
  conv       ops.conv_fused(x, w, bias, residual, ...) -> fp16 activations: one operator on its own

The models are held for the life of the process and have run once at a shape before it is used (a serving program loads a
model and warms it up before it takes traffic); images are new for every state. Weights are the registries' seeded ones
(there is no network for checkpoints), with ConvNeXt's LayerScale drawn from U(0.1, 1) as training leaves it, not at its
initial 1e-6, which would switch the residual branches off.
"""
from __future__ import annotations

import math

import torch

from fast_vision_models_b200 import backbones, ops, seg, zoo

_HANDLES = {}       # (kind of registry, model) -> loaded model
_WARM = set()       # (handle, image shape, dtype) that have run once
_FLOPS = {}         # (model, height, width) -> (operations, weights) of one image


def listed():
    return [
        # Operators on their own: the two ends of the fused-convolution sweep (3x3 over 256 channels with residual and
        # ReLU, bound by the tensor unit; 1x1 over 64 channels on a large map, bound by memory).
        dict(name="conv3x3_256_14_b64", kind="conv", n=64, c=256, h=14, w=14, k=3, res=True),
        dict(name="conv1x1_64_56_b64", kind="conv", n=64, c=64, h=56, w=56, k=1, res=True),
        # One image at a time: interactive use, where latency and launches count.
        dict(name="resnet50_b1", kind="classify", model="resnet50", n=1, h=224, w=224, half=False),
        dict(name="efficientnet_b0_b1", kind="classify", model="efficientnet_b0", n=1, h=224, w=224, half=False),
        # A small batch in fp16: a server that batches what has arrived.
        dict(name="convnext_tiny_b8_fp16", kind="classify", model="convnext_tiny", n=8, h=224, w=224, half=True),
        # A ragged batch of images that keep their aspect ratio, from a host that decodes to fp16.
        dict(name="resnet50_b13_200x264", kind="classify", model="resnet50", n=13, h=200, w=264, half=True),
        # Throughput: the benchmark's batch of 64 at each family's own resolution.
        dict(name="resnet50_b64", kind="classify", model="resnet50", n=64, h=224, w=224, half=False),
        dict(name="convnext_tiny_b64", kind="classify", model="convnext_tiny", n=64, h=224, w=224, half=False),
        dict(name="efficientnet_b4_b64", kind="classify", model="efficientnet_b4", n=64, h=380, w=380, half=False),
        # Dense features of mid-sized images.
        dict(name="features_resnet50_b4", kind="features", model="tv-resnet50", n=4, h=448, w=640, half=False),
        # Segmentation of street scenes: one frame's class scores, and a batch's class maps.
        dict(name="deeplab_scores_b1", kind="scores", model="deeplabv3-r50", n=1, h=512, w=1024, half=False),
        dict(name="deeplab_classmap_b8", kind="classmap", model="deeplabv3-r50", n=8, h=512, w=1024, half=False),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """One more case of the same ranges. Batches are spread over their logarithm; heights and widths differ and are often
    odd multiples; the largest batches and sizes are cut so that no case costs more than the largest listed one."""
    kind = rng.choices(["conv", "classify", "features", "classmap", "scores"], [5, 9, 3, 2, 2])[0]
    if kind == "conv":
        c = rng.choice([64, 128, 256, 512, 8 * _log_int(rng, 3, 64)])
        h = _log_int(rng, 7, 56)
        return dict(kind=kind, n=_log_int(rng, 1, 64), c=c, h=h, w=rng.choice([h, h, _log_int(rng, 7, 56)]),
                    k=rng.choice([1, 3]), res=rng.random() < 0.6)
    half = rng.random() < 0.4
    if kind == "classify":
        # (model, smallest side, largest side, most images x pixels)
        model, lo, hi, most = rng.choice([
            ("resnet18", 128, 288, 64 * 288 * 288), ("resnet50", 128, 288, 64 * 256 * 256), ("resnet50", 128, 288, 64 * 256 * 256),
            ("resnet101", 128, 288, 64 * 224 * 224), ("efficientnet_b0", 160, 288, 64 * 256 * 256),
            ("efficientnet_b4", 224, 380, 64 * 340 * 340), ("convnext_tiny", 160, 288, 64 * 224 * 224),
            ("convnext_small", 160, 288, 48 * 224 * 224)])
        h = rng.randint(lo, hi)
        w = h if rng.random() < 0.5 else rng.randint(lo, hi)
        n = min(_log_int(rng, 1, 64), max(1, most // (h * w)))
        return dict(kind=kind, model=model, n=n, h=h, w=w, half=half)
    if kind == "features":
        return dict(kind=kind, model=rng.choice(["tv-resnet50", "tv-resnet18", "tv-convnext_tiny"]), n=_log_int(rng, 1, 12),
                    h=32 * rng.randint(7, 16), w=32 * rng.randint(7, 20), half=half)
    return dict(kind=kind, model="deeplabv3-r50", n=_log_int(rng, 1, 7), h=8 * rng.randint(32, 64), w=8 * rng.randint(48, 128),
                half=half)


def _handle(case):
    kind, model = case["kind"], case["model"]
    key = ("seg" if kind in ("classmap", "scores") else kind, model)
    if key not in _HANDLES:
        if kind == "classify":
            _HANDLES[key] = zoo.load(model, "b200", layer_scale="uniform" if model.startswith("convnext") else None)
        elif kind == "features":
            _HANDLES[key] = backbones.build(model, "b200")
        else:
            _HANDLES[key] = seg.build(model, "b200")
    h = _HANDLES[key]
    return {"classify": lambda: h.model, "features": lambda: h.fn, "classmap": lambda: h.predict, "scores": lambda: h.logits}[kind]()


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    if case["kind"] == "conv":
        n, c, h, w, k = (case[a] for a in ("n", "c", "h", "w", "k"))

        def nhwc(*shape, std=1.0):
            return (torch.randn(shape, generator=g, device="cuda") * std).half().contiguous(memory_format=torch.channels_last)
        return dict(case=case, x=nhwc(n, c, h, w), wt=nhwc(c, c, k, k, std=0.02),
                    bias=(torch.randn(c, generator=g, device="cuda") * 0.1).half(),
                    res=nhwc(n, c, h, w) if case["res"] else None, pad=(k // 2, k // 2))
    x = torch.randn((case["n"], 3, case["h"], case["w"]), generator=g, device="cuda")
    x = x.half() if case["half"] else x
    fn = _handle(case)
    key = (case["kind"], case["model"], tuple(x.shape), x.dtype)
    if key not in _WARM:
        fn(x)
        _WARM.add(key)
    return dict(case=case, fn=fn, x=x)


def run(state):
    if state["case"]["kind"] == "conv":
        return ops.conv_fused(state["x"], state["wt"], state["bias"], state["res"], state["pad"], (1, 1), ops.ACT_RELU)
    return state["fn"](state["x"])


def _network(model, h, w):
    """Multiply-add operations (two each) and weights of the convolutions and linear layers for one image."""
    if (model, h, w) not in _FLOPS:
        import torchvision
        name = model.removeprefix("tv-")
        with torch.device("meta"):
            if name == "deeplabv3-r50":
                net = torchvision.models.segmentation.deeplabv3_resnet50(weights=None, weights_backbone=None, num_classes=19, aux_loss=False)
            else:
                net = torchvision.models.get_model(name, weights=None)
        total = [0]

        def count(m, args, out):
            total[0] += 2 * out.numel() * m.weight.numel() // m.weight.shape[0]
        layers = [m for m in net.modules() if isinstance(m, (torch.nn.Conv2d, torch.nn.Linear))]
        for m in layers:
            m.register_forward_hook(count)
        net.eval()(torch.empty((1, 3, h, w), device="meta"))
        _FLOPS[(model, h, w)] = (total[0], sum(m.weight.numel() for m in layers))
    return _FLOPS[(model, h, w)]


def work(case):
    """What one pass cannot do without: images (or activations), fp16 weights and results once each, and the operations
    of the convolutions and linear layers."""
    n, h, w = case["n"], case["h"], case["w"]
    if case["kind"] == "conv":
        c, k = case["c"], case["k"]
        act = n * c * h * w
        return dict(bytes=2 * (act * (3 if case["res"] else 2) + c * c * k * k + c), flops=2 * act * c * k * k)
    ops_1, weights = _network(case["model"], h, w)
    out = {"classify": 4 * 1000, "classmap": 4 * h * w, "scores": 4 * 19 * ((h + 7) // 8) * ((w + 7) // 8),
           "features": 4 * {"tv-resnet50": 2048, "tv-resnet18": 512}.get(case.get("model"), 768) * ((h + 31) // 32) * ((w + 31) // 32)
           }[case["kind"]]
    return dict(bytes=n * (3 * h * w * (2 if case["half"] else 4) + out) + 2 * weights, flops=n * ops_1)


def tolerance(case):
    """About four times the largest difference measured on a B200 between the fp16 path and the same network (or operator)
    in fp32 and between it and plain fp16 PyTorch with cuDNN's order of the sums: an fp16 convolution 2e-4 to 3.4e-4 (2e-3 at
    the worst element), logits of ResNets 5e-4 to 7e-4, of ConvNeXt 9e-4, of EfficientNet-B0 6e-4 and -B4 1.9e-3, feature
    maps 8e-4 to 1.9e-3 (1.7e-2 at the worst element), DeepLabV3's scores 1.3e-3 to 1.7e-3 and 4.3e-4 of its class map's
    pixels (where two classes tie)."""
    kind, model = case["kind"], case.get("model", "")
    if kind == "conv":
        return {"rel": 1.4e-3, "max": 8e-3}
    if kind == "classmap":
        return {"rel": 0.0, "differ": 1.7e-3}
    if kind == "features":
        return {"rel": 7e-3, "max": 7e-2}
    if kind == "scores":
        return {"rel": 6e-3, "max": 4e-2}
    return {"rel": {"efficientnet_b4": 7e-3, "efficientnet_b0": 2.5e-3, "convnext_tiny": 3.7e-3, "convnext_small": 3.7e-3}.get(model, 2.8e-3),
            "max": 4e-2 if model == "efficientnet_b4" else 1.5e-2}
