"""Predictor of a fused layer in inference: the filter padded to a multiple of eight output channels gives what the plain
convolution gives (channel counts off the multiple, with and without bias, one clip and several)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("G", [1, 2, 8])
@pytest.mark.parametrize("B", [1, 2])
@pytest.mark.parametrize("bias", [True, False])
def test_padded_predictor_equals_plain(G, B, bias):
    from d2conv3d_b200 import dconv_native as dn
    torch.manual_seed(0)
    layer = dn.modules.XYZSizeConditionedMDConv3d(64, 64, 3, 1, 1, offset_groups=G, bias=bias).cuda()
    torch.nn.init.normal_(layer.deform_params.weight, std=0.05)
    x = torch.randn(B, 64, 3, 7, 9, device="cuda")
    want = torch.nn.functional.conv3d(x.double(), layer.deform_params.weight.double(),
                                      None if not bias else layer.deform_params.bias.double(), 1, 1)
    with torch.no_grad():
        raw = layer._raw(x)
    assert raw.shape == want.shape and (B > 1 or raw.is_contiguous())
    assert (raw.double() - want).abs().max() <= 2e-3 * want.abs().max()
    assert layer._raw(x).requires_grad
