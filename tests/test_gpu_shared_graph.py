"""Backward over one graph from several threads: a thread gets the gradients, or the error that the graph was used up."""
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


def _cases():
    from d2conv3d_b200 import dconv_native as dn, fast_depthwise_conv3d as dw
    r = lambda *s: torch.randn(s, device="cuda", requires_grad=True)  # noqa: E731
    x, off, mask, w, b = r(1, 64, 2, 6, 7), r(1, 81, 2, 6, 7), r(1, 27, 2, 6, 7), r(64, 64, 3, 3, 3), r(64)
    size = r(1, 3, 2, 6, 7)
    wd = r(64, 1, 3, 3, 3)
    return {
        "deform": ((x, off, mask, w, b), lambda: dn.deform_conv3d(x, off, mask, w, b, 1, 1)),
        "field": ((x, size, mask, w, b), lambda: dn.dyn_dilated_conv3d(x, size, mask, w, b, "xyz", 1, 1)),
        "depthwise": ((x, wd, b), lambda: dw._ops.depthwise_separable_conv3d(x, wd, b, 1, 1, 1)),
    }


@pytest.mark.parametrize("kind", ["deform", "field", "depthwise"])
@pytest.mark.parametrize("retain", [True, False])
def test_threads_share_a_graph(kind, retain):
    inputs, op = _cases()[kind]
    y = op()
    gy = torch.randn_like(y)
    want = torch.autograd.grad(y, inputs, gy, retain_graph=True)
    with pytest.raises(RuntimeError, match="backward through the graph a second time"):
        torch.autograd.grad(y, inputs, gy)
        torch.autograd.grad(y, inputs, gy)
    torch.cuda.synchronize()
    threads_n, unexpected, got = 4, [], []
    for _ in range(10):
        y = op()
        torch.cuda.synchronize()
        start = threading.Barrier(threads_n)

        def work():
            # without the engine's own thread, every caller runs the nodes itself
            with torch.autograd.set_multithreading_enabled(False):
                start.wait()
                try:
                    got.append(torch.autograd.grad(y, inputs, gy, retain_graph=retain))
                except RuntimeError as exc:
                    if retain or "a second time" not in str(exc):
                        unexpected.append(exc)
                torch.cuda.synchronize()

        threads = [threading.Thread(target=work) for _ in range(threads_n)]
        [t.start() for t in threads]
        [t.join() for t in threads]
    assert not unexpected
    assert len(got) == 10 * threads_n if retain else len(got) >= 10
    # sums in another order of atomics: fp32 rounding
    assert all(((a - b).abs() <= 1e-5 * b.abs().max()).all() for grads in got for a, b in zip(grads, want))
