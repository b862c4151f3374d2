"""Stand-in for the reference's compiled module `dconv_native._ops`
(ops/dconv-native/csrc/ops/dconv.cpp:6-12): `deform_conv3d`, `deform_conv1d`
and the `config` sub-namespace, with the same positional signatures.  The work is
done by libd2conv3d.so; checks, allocations and the autograd nodes (the counterparts of
DeformConv3dFunction, csrc/ops/dconv3d.h:70-186, and DeformConv1dFunction,
csrc/ops/dconv1d.h:69-156) are native too (csrc/torch_ops.cpp).
"""
import ctypes
import threading
import types

import torch

from .. import _lib


_ready_lock = threading.Lock()
_ready = None


def params_ready_event():
    """The torch.cuda.Event that the most recent `deform_conv3d` / `dyn_dilated_conv3d` backward of this process
    recorded as soon as its parameter gradients (grad_weight, grad_bias) were final -- on the tensor-core tier
    before the data-side gradients are computed.  A data-parallel trainer makes a side stream wait for it and
    all-reduces the parameter gradients there (d2conv3d_b200.sharding.all_reduce_param_grads_overlapped), which
    hides the collective under the rest of the backward.  No later backward records it again.  None before the first
    backward."""
    global _ready
    with _ready_lock:
        _ready = _lib.native().take_params_ready_event() or _ready
        return _ready


def _will_differentiate(*tensors):
    """Whether autograd is recording this call (an evaluation pass under no_grad over trainable weights is not)."""
    return torch.is_grad_enabled() and any(t is not None and t.requires_grad for t in tensors)


def deform_conv3d(input, offset, alpha, weight, bias, stride_d, stride_h, stride_w, pad_d, pad_h, pad_w,
                  dilation_d, dilation_h, dilation_w, groups, offset_groups):
    """dconv_native._ops.deform_conv3d (csrc/ops/dconv3d.h:188-226)."""
    return _lib.native().deform_conv3d(input, offset, alpha, weight, bias, (stride_d, stride_h, stride_w),
                                       (pad_d, pad_h, pad_w), (dilation_d, dilation_h, dilation_w), groups, offset_groups,
                                       False)


def dyn_dilated_conv3d(input, size_map, alpha, weight, bias, mode, stride, padding, dilation, groups,
                       offset_groups):
    """Deformable conv3d whose offsets come from a dilation field (no counterpart in
    the reference's compiled module: there the field is expanded to 3*K offset
    channels by offsets_from_size_map, utils/grid.py:72-98, before deform_conv3d)."""
    return _lib.native().dyn_dilated_conv3d(input, size_map, alpha, weight, bias, _lib.FIELD_MODES[mode], stride, padding,
                                            dilation, groups, offset_groups, False)


def deform_conv3d_head(input, raw, weight, bias, field_mode, modulated, mask_act, size_act, stride, padding, dilation,
                       groups, offset_groups):
    """The layer's op on the predictor's raw output `raw` = [geometry channels | G*K mask logits (if modulated)]:
    geometry = 3*G*K offsets (field_mode None) or the 1..3 channels of a dilation field ("x", "xy", "xxz", "xyz").
    The split and the activations (network/layers.py:107-120, 171-181, 302-313) happen inside the kernels, and the
    backward returns the gradient w.r.t. the raw tensor.
    mask_act: "sigmoid" | "relu" | "tanh" | "linear" | "none"; size_act: "elu" | "relu" | "relu_plus_one" | "linear".
    No counterpart in the reference's compiled module, which is called after the split and the activations."""
    K = weight.shape[2] * weight.shape[3] * weight.shape[4]
    geo = 3 * offset_groups * K if field_mode is None else _lib.FIELD_CHANNELS[field_mode]
    want = geo + (offset_groups * K if modulated else 0)
    if raw.dim() != 5 or raw.shape[1] != want:
        raise RuntimeError(f"the deformation tensor must have {want} channels, got {tuple(raw.shape)}")
    differentiated = _will_differentiate(input, raw, weight, bias)
    desc = _lib.make_desc(input, weight, stride, padding, dilation, groups, offset_groups) if differentiated else None
    cache = _lib.SampleCache.for_forward(desc, input.device, differentiated)
    return _lib.native().deform_conv3d_head(
        input, raw, weight, bias, -1 if field_mode is None else _lib.FIELD_MODES[field_mode], geo if modulated else -1,
        _lib.MASK_ACTS[mask_act], _lib.SIZE_ACTS[size_act] if field_mode is not None else 0, stride, padding, dilation,
        groups, offset_groups, None if cache is None else cache.buf)


def deform_conv1d(input, offset, alpha, weight, bias, stride, padding, dilation, groups, offset_groups):
    """dconv_native._ops.deform_conv1d (csrc/ops/dconv1d.h:158-186, dconv1d_gpu.cu): modulated deformable conv1d
    with one offset per (offset group, tap, output position) and linear interpolation, out-of-range neighbours
    read as 0.  Forward, grad_input, grad_weight and grad_bias run on the library's generic kernels over the
    [B, C, 1, 1, L] view of the problem; grad_offset / grad_alpha come from a kernel of their own that follows the
    1-D reference's rule at integer sampling positions (`x0 -= 1`, dconv1d_gpu.cu:334-337)."""
    one = lambda v: int(v[0]) if isinstance(v, (tuple, list)) else int(v)
    return _lib.native().deform_conv1d(input, offset, alpha, weight, bias, one(stride), one(padding), one(dilation),
                                       groups, offset_groups, False)


def corners(input_shape, weight_shape, offset, stride, padding, dilation, offset_groups):
    """Integer floor corners [B, G*K, 3, V] the kernels derive from `offset`."""
    offset = offset.contiguous()
    desc = _lib.ConvDesc(_lib.dtype_code(offset), input_shape[0], input_shape[1], weight_shape[0],
                         input_shape[2], input_shape[3], input_shape[4], weight_shape[2], weight_shape[3],
                         weight_shape[4], *stride, *padding, *dilation, 1, offset_groups)
    V = 1
    for d in _lib.output_dims(desc):
        V *= d
    K = weight_shape[2] * weight_shape[3] * weight_shape[4]
    out = torch.empty((input_shape[0], offset_groups * K, 3, V), dtype=torch.int32, device=offset.device)
    with torch.cuda.device(offset.device):
        _lib.check(_lib.lib().d2c_deform_conv3d_corners(ctypes.byref(desc), _lib.ptr(offset), _lib.ptr(out),
                                                        _lib.stream_of(offset)), "corners")
    return out


def field_corners(input_shape, weight_shape, size_map, mode, stride, padding, dilation, offset_groups):
    size_map = size_map.contiguous()
    desc = _lib.ConvDesc(_lib.dtype_code(size_map), input_shape[0], input_shape[1], weight_shape[0],
                         input_shape[2], input_shape[3], input_shape[4], weight_shape[2], weight_shape[3],
                         weight_shape[4], *stride, *padding, *dilation, 1, offset_groups)
    V = 1
    for d in _lib.output_dims(desc):
        V *= d
    K = weight_shape[2] * weight_shape[3] * weight_shape[4]
    out = torch.empty((input_shape[0], offset_groups * K, 3, V), dtype=torch.int32, device=size_map.device)
    with torch.cuda.device(size_map.device):
        _lib.check(_lib.lib().d2c_dyn_dilated_conv3d_corners(
            ctypes.byref(desc), _lib.FIELD_MODES[mode], _lib.ptr(size_map), _lib.ptr(out),
            _lib.stream_of(size_map)), "field corners")
    return out


def _get_max_intermediate_elements():
    return int(_lib.lib().d2c_get_max_intermediate_elements())


def _set_max_intermediate_elements(n):
    _lib.lib().d2c_set_max_intermediate_elements(int(n))


# dconv_native._ops.config (csrc/ops/dconv.cpp:9-11)
config = types.SimpleNamespace(
    get_max_intermediate_elements=_get_max_intermediate_elements,
    set_max_intermediate_elements=_set_max_intermediate_elements,
)
