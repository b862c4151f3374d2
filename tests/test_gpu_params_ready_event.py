"""The event of a backward's parameter gradients: fires with them, is not moved by a later backward, and depends on no work of
other streams."""
import pytest
import torch

pytestmark = pytest.mark.gpu

SLEEP = int(1e9)          # clocks, half a second


def _backward():
    from d2conv3d_b200 import dconv_native as dn
    x, off, mask, w, b = (torch.randn(s, device="cuda", requires_grad=True)
                          for s in ((1, 64, 2, 5, 6), (1, 81, 2, 5, 6), (1, 27, 2, 5, 6), (64, 64, 3, 3, 3), (64,)))
    dn.deform_conv3d(x, off, mask, w, b, 1, 1).sum().backward()


def test_event_belongs_to_its_backward():
    from d2conv3d_b200.dconv_native import _ops
    side = torch.cuda.Stream()                   # the first one takes a while
    _backward()
    torch.cuda.synchronize()
    first = _ops.params_ready_event()
    assert isinstance(first, torch.cuda.Event) and first.query() and _ops.params_ready_event() is first
    torch.cuda._sleep(SLEEP)
    _backward()
    second = _ops.params_ready_event()
    assert first.query() and not second.query() and second is not first
    side.wait_event(second)
    done = side.record_event()
    assert not done.query()
    torch.cuda.synchronize()
    assert second.query() and done.query()
    _backward()
    _backward()                                  # events that nobody asked for are recorded again
    torch.cuda.synchronize()
    third = _ops.params_ready_event()
    assert third not in (first, second) and third.query()


def test_event_does_not_wait_for_streams_of_the_pool():
    """PyTorch hands out its pool of streams in turn: a stream taken for the event could be one that is busy."""
    from d2conv3d_b200.dconv_native import _ops
    _backward()
    torch.cuda.synchronize()
    pool = [torch.cuda.Stream()]
    while True:                                  # once around: the next one handed out is pool[1]
        s = torch.cuda.Stream()
        if s.cuda_stream == pool[0].cuda_stream:
            break
        pool.append(s)
    with torch.cuda.stream(pool[1]):
        torch.cuda._sleep(SLEEP)
        busy = pool[1].record_event()
    event = _ops.params_ready_event()
    fired = event.query()
    assert not busy.query() and fired
    torch.cuda.synchronize()


def test_events_of_two_threads():
    """Backwards at the same time record different events."""
    import threading

    from d2conv3d_b200.dconv_native import _ops
    errors = []

    def work():
        try:
            stream = torch.cuda.Stream()
            with torch.cuda.stream(stream), torch.autograd.set_multithreading_enabled(False):
                for _ in range(20):
                    _backward()
                    _ops.params_ready_event().synchronize()
        except Exception as exc:                 # noqa: BLE001
            errors.append(exc)

    threads = [threading.Thread(target=work) for _ in range(4)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    torch.cuda.synchronize()
    assert not errors
