"""Performance cases of the framework: the calls that a user's program makes, over the sizes it makes them at.

A case is a dict of plain values.  `prepare` makes what the program has in hand before the call, `run` makes the call.
Kinds of case:

  deform     DeformConv3d on predicted offsets and modulation mask (training step or inference)
  field      DeformConv3d driven by a dilation field (training step or inference)
  depthwise  DepthwiseConv3d of a channel-separated backbone block (training step)
  conv1d     DeformConv1d on a sequence (training step)
  decoder    the segmentation decoder on one clip's feature pyramid (inference)

A training step is the forward and the gradients of every input and parameter.
"""
import math

import torch

import d2conv3d_b200
from d2conv3d_b200 import dconv_native, fast_depthwise_conv3d
from d2conv3d_b200.decoder import Decoder, pyramid_shapes

_FIELD_CHANNELS = {"x": 1, "xy": 2, "xxz": 2, "xyz": 3}


def _deform(name, mode, step, b, cin, cout, dims, g, pad=1, stride=1):
    return dict(name=name, kind="deform", mode=mode, step=step, b=b, cin=cin, cout=cout, d=dims[0], h=dims[1], w=dims[2],
                g=g, pad=pad, stride=stride)


def listed():
    return [
        # one small layer on a small crop, the size at which the op is tried out and unit-tested: launches and host time
        _deform("small_train", "auto", "train", 1, 64, 64, (4, 16, 16), 1),
        # one layer of a running model on the coarsest pyramid level of a 480 x 854 clip (stride 32), latency counts
        _deform("coarse_infer", "auto", "infer", 1, 256, 256, (8, 15, 27), 1),
        # the reference's own benchmark program: narrow layer, many small clips (CUDA-core kernels)
        _deform("narrow_train", "auto", "train", 8, 16, 32, (9, 9, 9), 1, pad=0),
        # a fine-tuning run that asks for plain fp32 arithmetic (CUDA-core kernels at a middling size)
        _deform("exact_train", "fp32", "train", 1, 128, 128, (8, 30, 54), 4),
        # the modulated deformable layer of a stage-4 backbone block, two clips per GPU, default arithmetic
        _deform("stage4_train", "auto", "train", 2, 512, 512, (8, 30, 54), 8),
        # the same layer where the user chose single-pass bf16 operands
        _deform("stage4_train_bf16", "bf16", "train", 2, 512, 512, (8, 30, 54), 8),
        # the wide modulated layer that follows a bottleneck, serving one clip with bf16 operands
        _deform("wide_infer_bf16", "bf16", "infer", 1, 1024, 256, (8, 30, 54), 8),
        # a refine block's dynamic-dilated layer at stride 8 (odd width), the batch that the training scripts use
        dict(name="field_train", kind="field", mode="auto", step="train", field="xyz", b=2, cin=256, cout=256, d=8, h=60, w=107,
             g=1),
        # the depthwise convolution of a backbone stage, fp32
        dict(name="depthwise_train", kind="depthwise", dtype="float32", b=8, c=1024, d=8, h=30, w=54, stride=1),
        # the same under autocast on an earlier stage (odd width)
        dict(name="depthwise_half_train", kind="depthwise", dtype="float16", b=4, c=256, d=8, h=60, w=107, stride=1),
        # a deformable layer over sequences
        dict(name="conv1d_train", kind="conv1d", b=8, cin=64, cout=64, length=2048, k=3, g=1),
        # the whole decoder on one clip of 8 frames at 480 x 854
        dict(name="decoder_infer", kind="decoder", mode="auto", frames=8, height=480, width=854),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _volume(rng, most):
    """Clip sizes D, H, W of at most `most` voxels: up to 16 frames, up to the stride-4 level of a 480 x 854 clip."""
    while True:
        d, h, w = _log(rng, 2, 16), _log(rng, 6, 120), _log(rng, 8, 214)
        if d * h * w <= most:
            return d, h, w


def draw(rng):
    kind = rng.choice(["deform", "deform", "deform", "field", "field", "narrow", "exact", "depthwise", "depthwise", "conv1d",
                       "decoder"])
    if kind in ("deform", "field"):
        # network widths; the largest column matrix is about that of the widest listed layer at a few clips
        cin, cout = rng.choice([64, 128, 256, 512, 1024]), rng.choice([64, 128, 256, 512])
        g = rng.choice([1, 1, 2, 4, 8])
        g = min(g, cin // 32)
        b = _log(rng, 1, 8)
        d, h, w = _volume(rng, int(min(1.0e9 / (27 * b * cin), 1.5e12 / (54.0 * b * cin * cout))))
        mode, step = rng.choice(["auto", "auto", "bf16"]), rng.choice(["train", "train", "infer"])
        c = dict(kind=kind, mode=mode, step=step, b=b, cin=cin, cout=cout, d=d, h=h, w=w, g=g)
        if kind == "field":
            c["field"] = rng.choice(["x", "xy", "xyz"])
        else:
            c.update(pad=1, stride=1)
        return c
    if kind in ("narrow", "exact"):
        # layers that run on the CUDA-core kernels: few or unusual channel counts, or plain fp32 asked for
        step_c = 8 if kind == "narrow" else 32
        cin = step_c * rng.randint(1, 6 if kind == "narrow" else 8)
        cout = step_c * rng.randint(1, 6 if kind == "narrow" else 8)
        b = _log(rng, 1, 8)
        d, h, w = _volume(rng, int(2.0e10 / (54.0 * b * cin * cout)))
        return dict(kind="deform", mode="fp32" if kind == "exact" else "auto", step="train", b=b, cin=cin, cout=cout, d=d,
                    h=h, w=w, g=rng.choice([1, 2, 4]), pad=1, stride=rng.choice([1, 1, 2]))
    if kind == "depthwise":
        c, b = 64 * rng.choice([1, 2, 4, 8, 16]), _log(rng, 1, 8)
        d, h, w = _volume(rng, int(1.06e8 / (b * c)))
        return dict(kind=kind, dtype=rng.choice(["float32", "float16"]), b=b, c=c, d=d, h=h, w=w, stride=rng.choice([1, 1, 1, 2]))
    if kind == "conv1d":
        return dict(kind=kind, b=_log(rng, 1, 16), cin=16 * rng.randint(1, 8), cout=16 * rng.randint(1, 8),
                    length=_log(rng, 64, 8192), k=rng.choice([3, 5, 7]), g=rng.choice([1, 2]))
    return dict(kind="decoder", mode=rng.choice(["auto", "bf16"]), frames=rng.randint(2, 8), height=_log(rng, 128, 480),
                width=_log(rng, 128, 854))


def _out(n, pad, stride, k=3):
    return (n + 2 * pad - k) // stride + 1


def _out_dims(case):
    pad, stride = case.get("pad", 1), case.get("stride", 1)
    return tuple(_out(case[n], pad, stride) for n in "dhw")


def prepare(case, seed):
    gen = torch.Generator("cuda").manual_seed(1000 + seed)
    rand = lambda *shape: torch.randn(shape, generator=gen, device="cuda")  # noqa: E731
    kind, train = case["kind"], case.get("step", "train") == "train" and case["kind"] != "decoder"
    state = dict(case=case, train=train)
    if kind in ("deform", "field"):
        b, g, out = case["b"], case["g"], _out_dims(case)
        with torch.device("cuda"):
            layer = dconv_native.DeformConv3d(case["cin"], case["cout"], 3, case.get("stride", 1), case.get("pad", 1),
                                              offset_groups=g)
        x = rand(b, case["cin"], case["d"], case["h"], case["w"])
        mask = torch.sigmoid(rand(b, 27 * g, *out))
        if kind == "deform":
            geo = 2.0 * rand(b, 81 * g, *out)                     # offsets of a couple of voxels
        else:
            geo = 1 + torch.nn.functional.softplus(rand(b, _FIELD_CHANNELS[case["field"]], *out))
        state.update(layer=layer, inputs=[x, geo, mask], params=[layer.weight, layer.bias],
                     grad=rand(b, case["cout"], *out) if train else None)
    elif kind == "conv1d":
        b, g, n, k = case["b"], case["g"], case["length"], case["k"]
        with torch.device("cuda"):
            layer = dconv_native.DeformConv1d(case["cin"], case["cout"], k, padding=k // 2, offset_groups=g)
        x, geo, mask = rand(b, case["cin"], n), 2.0 * rand(b, k * g, n), torch.sigmoid(rand(b, k * g, n))
        state.update(layer=layer, inputs=[x, geo, mask], params=[layer.weight, layer.bias], grad=rand(b, case["cout"], n))
    elif kind == "depthwise":
        dtype, c, stride = getattr(torch, case["dtype"]), case["c"], case["stride"]
        with torch.device("cuda"):
            layer = fast_depthwise_conv3d.DepthwiseConv3d(c, c, 3, (1, stride, stride), 1, bias=False)
        x = rand(case["b"], c, case["d"], case["h"], case["w"]).to(dtype)
        out = (case["d"],) + tuple(_out(case[n], 1, stride) for n in "hw")
        state.update(layer=layer, inputs=[x], params=[layer.weight], grad=rand(case["b"], c, *out).to(dtype))
    else:
        with torch.device("cuda"):
            net = Decoder()
        # a trained predictor: dilation and modulation vary from voxel to voxel
        for name, p in net.named_parameters():
            if name.endswith("deform_params.weight"):
                p.data = rand(*p.shape) * (0.5 / math.sqrt(p[0].numel()))
        shapes = pyramid_shapes(1, case["frames"], case["height"], case["width"])
        state.update(layer=net.eval(), inputs=[torch.relu(rand(*s)) for s in shapes])
    if "params" in state:
        for p in state["params"]:
            bound = 1 / math.sqrt(state["params"][0][0].numel())
            p.data = rand(*p.shape) * bound
    elif kind == "decoder":
        for name, p in net.named_parameters():
            if not name.endswith("deform_params.weight") and p.dim() == 5:
                p.data = rand(*p.shape) * math.sqrt(1.0 / p[0].numel())
            elif name.endswith("bias"):
                p.data = 0.1 * rand(*p.shape)
    if train:
        for t in state["inputs"]:
            t.requires_grad_()
    return state


def _forward(state):
    case, layer = state["case"], state["layer"]
    if case["kind"] == "field":
        return layer.forward_field(*state["inputs"], case["field"])
    return layer(*state["inputs"])


def run(state):
    if "mode" in state["case"]:
        d2conv3d_b200.set_math_mode(state["case"]["mode"])
    if not state["train"]:
        with torch.no_grad():
            return _forward(state)
    y = _forward(state)
    return [y.detach()] + list(torch.autograd.grad(y, state["inputs"] + state["params"], state["grad"]))


def _decoder_work(case):
    """Features read, weights read, logits written; the multiply-adds of every convolution."""
    shapes = pyramid_shapes(1, case["frames"], case["height"], case["width"])
    vox = [s[2] * s[3] * s[4] for s in shapes]
    wid = [s[1] for s in shapes]
    ch, predictor = 256, 3 + 8 * 27
    macs = weights = 0
    for level in (2, 1, 0):
        for cin in (wid[level], ch, ch, ch, ch):                  # predictor and deformable convolution of a unit
            weights += 27 * cin * (ch + predictor)
            macs += 27 * cin * (ch + predictor) * vox[level]
    bridge = 2 * 7 * (wid[3] * ch + ch * ch) + 2 * 27 * ch * ch
    weights += bridge + 27 * ch * 2
    macs += bridge * vox[3] + 27 * ch * 2 * vox[0]
    out = 2 * case["frames"] * 16 * shapes[0][3] * shapes[0][4]
    return {"bytes": 4 * (sum(v * w for v, w in zip(vox, wid)) + weights + out), "flops": 2 * macs}


def work(case):
    kind = case["kind"]
    if kind == "decoder":
        return _decoder_work(case)
    if kind == "conv1d":
        b, cin, cout, n, k, g = (case[v] for v in ("b", "cin", "cout", "length", "k", "g"))
        x, y, w, geo = b * cin * n, b * cout * n, cout * cin * k, 2 * b * k * g * n
        return {"bytes": 4 * (2 * (x + w + geo + cout) + 2 * y), "flops": 3 * 2 * b * n * cin * cout * k}
    if kind == "depthwise":
        size, s = (4 if case["dtype"] == "float32" else 2), case["stride"]
        x = case["b"] * case["c"] * case["d"] * case["h"] * case["w"]
        y = case["b"] * case["c"] * case["d"] * _out(case["h"], 1, s) * _out(case["w"], 1, s)
        return {"bytes": size * (2 * x + 2 * y) + 4 * 2 * 27 * case["c"], "flops": 3 * 2 * 27 * y}
    out = _out_dims(case)
    v = case["b"] * out[0] * out[1] * out[2]
    x = case["b"] * case["cin"] * case["d"] * case["h"] * case["w"]
    geo = v * (27 * case["g"] + (81 * case["g"] if kind == "deform" else _FIELD_CHANNELS[case["field"]]))
    w, y, f = 27 * case["cin"] * case["cout"] + case["cout"], v * case["cout"], 2 * v * case["cin"] * case["cout"] * 27
    if case["step"] == "train":
        return {"bytes": 4 * (2 * (x + geo + w) + 2 * y), "flops": 3 * f}
    return {"bytes": 4 * (x + geo + w + y), "flops": f}


def tolerance(case):
    if case["kind"] == "decoder":
        # fifteen deformable layers and the library's TF32 convolutions between them
        return {"rel": 1e-3 if case["mode"] == "auto" else 1e-2}
    if case["kind"] == "depthwise":
        return {"rel": 1e-5} if case["dtype"] == "float32" else {"rel": 1e-3}
    if case["kind"] == "conv1d" or case["mode"] == "fp32" or (case["cin"] // case["g"]) % 32 or case["cout"] % 64:
        return {"rel": 1e-5}                                      # fp32 sums
    # split operands keep 16 significand bits; single-pass operands keep 8
    return {"rel": 3e-5} if case["mode"] == "auto" else {"rel": 1e-2}
