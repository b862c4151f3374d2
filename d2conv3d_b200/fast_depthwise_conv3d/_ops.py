"""Stand-in for the reference's compiled `fast_depthwise_conv3d._ops`
(ops/fast-depthwise-conv3d/csrc/python_bindings.cpp:4-6):
`depthwise_separable_conv3d(input, weight, bias, stride, padding, dilation)` with the
autograd of DepthwiseConv3dFunction (csrc/grouped_conv3d.h:29-106), native in csrc/torch_ops.cpp."""
from torch.nn.modules.utils import _triple

from .. import _lib


def depthwise_separable_conv3d(input, weight, bias, stride, padding, dilation):
    return _lib.native().depthwise_conv3d(input, weight, bias, _triple(stride), _triple(padding), _triple(dilation))
