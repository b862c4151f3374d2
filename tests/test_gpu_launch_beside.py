"""The kernels of a tensor-core forward that run beside one another: calls one after the other on the same buffers, a call on each of
two streams, capture into a graph and its replays on new inputs, a NaN in one call and none in the next (whose workspace may be the
same memory).  Small calls, whose last kernel starts beside the staging too, and larger ones."""
import numpy as np
import pytest
import torch

from oracle import oracle as orc

pytestmark = pytest.mark.gpu

SIZES = [(64, 64, (4, 16, 16)), (256, 256, (8, 15, 27)), (256, 128, (8, 60, 70))]


def problem(cin, cout, dims, seed):
    gen = torch.Generator("cuda").manual_seed(seed)
    rand = lambda *s: torch.randn(s, generator=gen, device="cuda")  # noqa: E731
    return [rand(1, cin, *dims), 2 * rand(1, 81, *dims), torch.sigmoid(rand(1, 27, *dims)), rand(cout, cin, 3, 3, 3) * (27 * cin) ** -0.5,
            rand(cout)]


def close(a, b):
    # the same kernels on the same inputs: partial tiles meet in another order
    return float((a - b).abs().max()) <= 1e-5 * float(b.abs().max())


@pytest.mark.parametrize("cin,cout,dims", SIZES)
def test_calls_streams_and_graphs(cin, cout, dims):
    from d2conv3d_b200 import _lib, dconv_native
    call = lambda p: dconv_native.deform_conv3d(*p, 1, 1, 1, 1, 1)  # noqa: E731
    p, q = problem(cin, cout, dims, 1), problem(cin, cout, dims, 2)
    with torch.no_grad():
        want = []
        for s in (p, q):
            want.append(call(s))
            torch.cuda.synchronize()
        for y, w in zip([call(s) for s in (p, q, p, q)], want + want):
            assert close(y, w)
        bad = [p[0].clone()] + p[1:]
        bad[0][0, 0, 0, 0, 0] = float("nan")
        y = call(bad)
        assert torch.isnan(y).any()
        del y
        assert close(call(q), want[1])
        side = [torch.cuda.Stream(), torch.cuda.Stream()]
        got = [[], []]
        torch.cuda.synchronize()
        for _ in range(4):
            for i, s in enumerate((p, q)):
                with torch.cuda.stream(side[i]):
                    got[i].append(call(s))
        torch.cuda.synchronize()
        for i in range(2):
            assert all(close(y, want[i]) for y in got[i])
        graph, into = torch.cuda.CUDAGraph(), [t.clone() for t in p]
        with torch.cuda.graph(graph):
            y = call(into)
        for s, w in ((p, want[0]), (q, want[1]), (p, want[0])):
            for a, b in zip(into, s):
                a.copy_(b)
            graph.replay()
            torch.cuda.synchronize()
            assert close(y, w)
    _lib.device_status()


@pytest.mark.parametrize("mode", ["auto", "bf16"])
@pytest.mark.parametrize("cin,cout,dims", SIZES[:2])
def test_which_outputs_are_nan(mode, cin, cout, dims):
    """Calls with and without a NaN in turn: the outputs whose samples give the voxel a weight are NaN in the one, and none but those
    that read it with weight zero at most; none at all in the other."""
    import d2conv3d_b200
    from d2conv3d_b200 import _lib, dconv_native
    p = problem(cin, cout, dims, 3)
    at = tuple(d // 2 for d in dims)
    bad = [p[0].clone()] + p[1:]
    bad[0][(0, cin // 2) + at] = float("nan")

    def reached(corners):
        ind = np.zeros((1, 1) + dims)
        for c in corners:
            ind[(0, 0) + tuple(c)] = 1.0
        geo, mask = (t.double().cpu().numpy() for t in p[1:3])
        y = orc.deform_conv3d_fwd(ind, geo, mask, np.ones((1, 1, 3, 3, 3)), None, padding=1)
        return torch.from_numpy(y > 0).cuda().expand(1, cout, *dims)

    touched, allowed = reached([at]), reached([np.subtract(at, d) for d in np.ndindex(2, 2, 2)])
    assert touched.any() and not allowed.all()
    d2conv3d_b200.set_math_mode(mode)
    try:
        with torch.no_grad():
            want = dconv_native.deform_conv3d(*p, 1, 1, 1, 1, 1)
            for _ in range(4):
                y = dconv_native.deform_conv3d(*bad, 1, 1, 1, 1, 1)
                assert y[touched].isnan().all() and not y[~allowed].isnan().any()
                assert float((y - want)[~allowed].abs().max()) <= 1e-5 * float(want.abs().max())
                assert close(dconv_native.deform_conv3d(*p, 1, 1, 1, 1, 1), want)
    finally:
        d2conv3d_b200.set_math_mode("auto")
    _lib.device_status()


@pytest.mark.parametrize("dims", [(8, 12, 20), (8, 15, 27)])
def test_both_sides_of_the_line_for_many_outputs(dims):
    """Single pass, 512 outputs: 22 units a CTA start beside the staging, 38 do not.  New inputs in every call."""
    import d2conv3d_b200
    from d2conv3d_b200 import _lib, dconv_native
    ps = [problem(512, 512, dims, seed) for seed in range(3)]
    try:
        with torch.no_grad():
            d2conv3d_b200.set_math_mode("fp32")
            want = [dconv_native.deform_conv3d(*p, 1, 1, 1, 1, 1) for p in ps]
            d2conv3d_b200.set_math_mode("bf16")
            for y, w in zip([dconv_native.deform_conv3d(*p, 1, 1, 1, 1, 1) for p in ps * 3], want * 3):
                assert float((y - w).abs().max()) <= 2e-2 * float(w.abs().max())      # the mode's bound
    finally:
        d2conv3d_b200.set_math_mode("auto")
    _lib.device_status()


def test_nan_word_is_this_calls_own():
    """The word by which a forward chooses its loop, in a workspace of the caller's that holds anything: it tells of this call's input,
    not of what the memory held or of an earlier call, in replays of a graph too."""
    import ctypes
    import d2conv3d_b200
    from d2conv3d_b200 import _lib
    cin, cout, dims = SIZES[0]
    x, offset, mask, w, bias = problem(cin, cout, dims, 4)
    d = _lib.ConvDesc(dtype=_lib.F32, batch=1, in_channels=cin, out_channels=cout, in_d=dims[0], in_h=dims[1], in_w=dims[2], kd=3, kh=3,
                      kw=3, stride_d=1, stride_h=1, stride_w=1, pad_d=1, pad_h=1, pad_w=1, dil_d=1, dil_h=1, dil_w=1, groups=1,
                      offset_groups=1)
    L = _lib.lib()
    d2conv3d_b200.set_math_mode("auto")
    n = L.d2c_workspace_bytes(_lib.OP_DEFORM_FWD, ctypes.byref(d))
    records = 27 * dims[0] * dims[1] * dims[2] * 48                    # the word's 256 bytes lie before them, at the end
    ws, y = torch.full((n,), 255, dtype=torch.uint8, device="cuda"), torch.empty(1, cout, *dims, device="cuda")
    word = ws[n - records - 256:][:4].view(torch.int32)
    clean, into = x.clone(), x.clone()

    def call():
        st = L.d2c_deform_conv3d_fwd(ctypes.byref(d), into.data_ptr(), offset.data_ptr(), mask.data_ptr(), w.data_ptr(), bias.data_ptr(),
                                     y.data_ptr(), ws.data_ptr(), n, torch.cuda.current_stream().cuda_stream)
        assert st == 0

    x[0, 5, 1, 2, 3] = float("nan")
    graph = torch.cuda.CUDAGraph()
    side = torch.cuda.Stream()
    with torch.cuda.graph(graph, stream=side):
        call()
    for run in (call, graph.replay):
        for src, found in ((clean, 0), (x, 1), (clean, 0)):
            into.copy_(src)
            run()
            assert int(word) == found
    _lib.device_status()
