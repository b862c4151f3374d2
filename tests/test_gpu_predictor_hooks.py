"""Inference through a layer shows its predictor to whoever watches: hooks of the module, hooks of every module, a replaced forward."""
import pytest
import torch
from torch import nn

pytestmark = pytest.mark.gpu


def _own_hook(conv, see):
    return conv.register_forward_hook(lambda mod, args, out: see(mod)).remove


def _own_pre_hook(conv, see):
    return conv.register_forward_pre_hook(lambda mod, args: see(mod)).remove


def _global_hook(conv, see):
    return nn.modules.module.register_module_forward_hook(lambda mod, args, out: see(mod)).remove


def _global_pre_hook(conv, see):
    return nn.modules.module.register_module_forward_pre_hook(lambda mod, args: see(mod)).remove


def _forward(conv, see):
    plain = conv.forward
    conv.forward = lambda x: (see(conv), plain(x))[1]
    return lambda: vars(conv).pop("forward")


@pytest.mark.parametrize("watch", [_own_hook, _own_pre_hook, _global_hook, _global_pre_hook, _forward])
def test_predictor_is_seen(watch):
    from d2conv3d_b200 import dconv_native as dn
    layer = dn.modules.XYZSizeConditionedMDConv3d(64, 64, 3, 1, 1, offset_groups=2).cuda()
    x = torch.randn(1, 64, 3, 7, 9, device="cuda")
    seen = []
    with torch.no_grad():
        want = layer(x)
        remove = watch(layer.deform_params, seen.append)
        try:
            got = layer(x)
        finally:
            remove()
    assert seen.count(layer.deform_params) == 1
    # the predictor's weights are zero: both ways give the same geometry; sums in another order of atomics
    assert (got - want).abs().max() <= 1e-5 * want.abs().max()
