"""Out-of-bounds guard for every output and scratch buffer of the C ABI: each buffer sits between sentinel
pads; after the full forward + backward stage sequence the pads must be untouched (the CUDA kernels write
through TMA stores and plain stores; compute-sanitizer is not available on the GPU pool).  The reference
runs its kernels under mssanitizer memcheck for the same purpose (mamba2_ssd_mssanitizer_test.py:70-78)."""
import ctypes

import pytest
import torch

from oracle import ssd_oracle as O

pytestmark = pytest.mark.gpu

PAD = 4096  # floats on each side (keeps 16-byte alignment of the payload)
SENTINEL = 12345.678


class Padded:
    def __init__(self, shape, dev, dtype=torch.float32):
        n = 1
        for d in shape:
            n *= d
        self.raw = torch.full((n + 2 * PAD,), SENTINEL, device=dev, dtype=dtype)
        self.view = self.raw[PAD:PAD + n].view(shape)

    def intact(self):
        return bool((self.raw[:PAD] == SENTINEL).all()) and bool((self.raw[-PAD:] == SENTINEL).all())


@pytest.mark.parametrize("shape", [(2, 384, 6, 64, 64, 64, 2), (1, 640, 4, 64, 64, 64, 4)])
def test_no_stage_writes_outside_its_buffers(shape):
    from ascend_kernel import _capi, mamba2 as M

    dev = torch.device("cuda:0")
    b, l, h, p, n, _chunk, g = shape
    k = l // 128
    x, dt, a, bm, cm = [t.to(dev) for t in O.make_inputs(shape, 91)]
    dout = torch.randn(b, l, h, p, device=dev)
    dfinal = torch.randn(b, h, p, n, device=dev)
    bufs = {name: Padded(shp, dev, dty) for name, shp, dty in [
        ("q", (b, h, l), torch.float32), ("cs", (b, h, l), torch.float32),
        ("states", (b, h, k, p, n), torch.float32), ("final", (b, h, p, n), torch.float32),
        ("out", (b, l, h, p), torch.float32), ("dstates", (b, h, k, p, n), torch.float32),
        ("g_last", (b, h, k), torch.float32), ("d_initial", (b, h, p, n), torch.float32),
        ("fold", (b, h, p, n), torch.float32),
        ("dx", (b, l, h, p), torch.float32), ("ddt_t", (b, h, l), torch.float32),
        ("dA_part", (b, h, k), torch.float64), ("dB", (b, l, g, n), torch.float32),
        ("dC", (b, l, g, n), torch.float32), ("ddt", (b, l, h), torch.float32), ("dA", (h,), torch.float32)]}
    v = {name: pb.view for name, pb in bufs.items()}
    lib = _capi.lib
    shp = M.make_shape(x, bm, True)
    sp = ctypes.byref(shp)
    st = torch.cuda.current_stream().cuda_stream
    status = torch.zeros(1, dtype=torch.int32, device=dev)
    P = lambda t: t.data_ptr()  # noqa: E731
    calls = [
        ("dt_cumsum", lambda: lib.ssd_dt_cumsum(sp, P(dt), None, P(a), P(v["q"]), P(v["cs"]), st)),
        ("chunk_state", lambda: lib.ssd_chunk_state(sp, P(x), P(bm), P(v["q"]), P(v["cs"]), P(v["states"]), 0, P(status), st)),
        ("state_passing_fwd", lambda: lib.ssd_state_passing_fwd(sp, P(v["states"]), P(v["cs"]), None, P(v["final"]), st)),
        ("chunk_scan_fwd", lambda: lib.ssd_chunk_scan_fwd(sp, P(x), P(bm), P(cm), P(v["states"]), P(v["q"]), P(v["cs"]),
                                                         P(v["out"]), P(status), st)),
        ("chunk_state_bwd", lambda: lib.ssd_chunk_state(sp, P(dout), P(cm), P(v["q"]), P(v["cs"]), P(v["dstates"]), 1, P(status), st)),
        ("state_passing_bwd", lambda: lib.ssd_state_passing_bwd(sp, P(v["dstates"]), P(v["states"]), P(v["cs"]), P(dfinal),
                                                               P(v["g_last"]), P(v["d_initial"]), st)),
        ("chunk_dx_bwd", lambda: lib.ssd_chunk_dx_bwd(sp, P(x), P(bm), P(cm), P(dout), P(v["out"]), P(v["dstates"]), P(v["q"]),
                                                     P(v["cs"]), P(dt), None, P(a), P(v["g_last"]), P(v["dx"]), P(v["ddt_t"]),
                                                     P(v["dA_part"]), None, 0, P(status), st)),
        ("chunk_dbc_bwd", lambda: lib.ssd_chunk_dbc_bwd(sp, P(x), P(bm), P(cm), P(dout), P(v["states"]), P(v["dstates"]),
                                                       P(v["q"]), P(v["cs"]), P(v["dB"]), P(v["dC"]), P(v["g_last"]),
                                                       P(status), st)),
        ("dt_finalize_bwd", lambda: lib.ssd_dt_finalize_bwd(sp, P(v["ddt_t"]), P(v["dA_part"]), P(v["ddt"]), P(v["dA"]), st)),
        # the fused state stages and the read-only fold write the same buffers again
        ("chunk_state_scan", lambda: lib.ssd_chunk_state_scan(sp, P(x), P(bm), P(v["q"]), P(v["cs"]), None, P(v["states"]),
                                                             P(v["final"]), 0, P(status), st)),
        ("chunk_state_scan_bwd", lambda: lib.ssd_chunk_state_scan(sp, P(dout), P(cm), P(v["q"]), P(v["cs"]), P(dfinal),
                                                                 P(v["dstates"]), P(v["d_initial"]), 1, P(status), st)),
        ("state_fold", lambda: lib.ssd_state_fold(sp, P(v["dstates"]), P(v["cs"]), None, P(v["fold"]), 0, st)),
    ]
    for name, call in calls:
        _capi.check(call(), name)
        torch.cuda.synchronize()
        assert status.item() == 0, name
        broken = [bn for bn, pb in bufs.items() if not pb.intact()]
        assert not broken, f"{name} wrote outside {broken}"
    # every payload was written in full (no sentinel left) and is finite
    for name, pb in bufs.items():
        assert torch.isfinite(pb.view).all(), name
        assert not bool((pb.view == SENTINEL).any()), name
    # and the results are the real ones
    want = O.fp64_forward_backward(x.cpu(), dt.cpu(), a.cpu(), bm.cpu(), cm.cpu(), 64, dt_softplus=True,
                                   dout=dout.cpu(), dfinal=dfinal.cpu())
    got = [v["out"], v["final"], v["dx"], v["ddt"], v["dA"], v["dB"], v["dC"]]
    for gt, w, name in zip(got, want, ["out", "final", "dx", "ddt", "dA", "dB", "dC"]):
        assert O.rel_l2(gt.cpu(), w) <= 2e-3, name


def _between_pads(shapes, dev):
    return {name: Padded(shp, dev, torch.float64 if name == "dA_part" else torch.float32) for name, shp in shapes.items()}


def _check_pads(bufs, status, name):
    torch.cuda.synchronize()
    assert status.item() == 0, name
    broken = [bn for bn, pb in bufs.items() if not pb.intact()]
    assert not broken, f"{name} wrote outside {broken}"


EXTENTS = [  # b, l, h, p, n, g, parts
    (2, 129, 3, 60, 36, 3, 1),   # one token over a tile, quads that end inside a box
    (1, 257, 8, 36, 100, 1, 1),  # two column blocks, the heads of the group dealt to several work items
    (1, 384, 2, 64, 128, 2, 3),  # three kernel heads per head, two column blocks
    (2, 127, 4, 20, 64, 2, 1),   # one box narrower than the channels of another
]


@pytest.mark.parametrize("b,l,h,p,n,g,parts", EXTENTS)
def test_no_stage_writes_outside_tensors_of_any_extent(b, l, h, p, n, g, parts):
    from ascend_kernel import _capi, mamba2 as M

    dev = torch.device("cuda:0")
    hk, cols, k = h * parts, 64 if n <= 64 else 128, (l + 127) // 128
    rnd = lambda *s: torch.randn(*s, device=dev)  # noqa: E731
    x, dt, a, bm, cm = rnd(b, l, hk, p), torch.rand(b, l, h, device=dev), -torch.rand(h, device=dev), rnd(b, l, g, n), rnd(b, l, g, n)
    bias, dout, dfinal, D = 0.1 * rnd(h), rnd(b, l, hk, p), rnd(b, hk, p, n), rnd(h)
    shp = M.extents_shape(x, bm, h, True, (0.0, float("inf")))
    sp, lib, st = ctypes.byref(shp), _capi.lib, torch.cuda.current_stream().cuda_stream
    split = max(2, lib.ssd_dbc_split(sp)) if hk // g % 2 == 0 else 1
    bufs = _between_pads({
        "q": (b, hk, k * 128), "cs": (b, hk, k * 128), "states": (b, hk, k, 64, cols), "final": (b, hk, p, n),
        "out": (b, l, hk, p), "copy": (b, l, hk, p), "dstates": (b, hk, k, 64, cols), "g_last": (cols // 64, b, hk, k),
        "d_initial": (b, hk, p, n), "dx": (b, l, hk, p), "ddt_t": (b, hk, k * 128), "dA_part": (b, hk, k),
        "dB": (b, l, g, n), "dC": (b, l, g, n), "partial": (2, split, b, l, g, n), "ddt": (b, l, h), "dA": (h,), "dbias": (h,)}, dev)
    v = {name: pb.view.data_ptr() for name, pb in bufs.items()}
    status = torch.zeros(1, dtype=torch.int32, device=dev)
    P = lambda t: t.data_ptr()  # noqa: E731
    calls = [
        ("dt_cumsum", lambda: lib.ssd_dt_cumsum(sp, P(dt), P(bias), P(a), v["q"], v["cs"], st)),
        ("chunk_state", lambda: lib.ssd_chunk_state(sp, P(x), P(bm), v["q"], v["cs"], v["states"], 0, P(status), st)),
        ("state_passing_fwd", lambda: lib.ssd_state_passing_fwd(sp, v["states"], v["cs"], P(dfinal), v["final"], st)),
        ("chunk_scan", lambda: lib.ssd_chunk_scan_copy_fwd(sp, P(x), P(bm), P(cm), v["states"], v["q"], v["cs"], v["out"],
                                                           v["copy"], P(status), st)),
        ("chunk_state_bwd", lambda: lib.ssd_chunk_state(sp, P(dout), P(cm), v["q"], v["cs"], v["dstates"], 1, P(status), st)),
        ("state_passing_bwd", lambda: lib.ssd_state_passing_bwd(sp, v["dstates"], None, v["cs"], P(dfinal), None, v["d_initial"], st)),
        ("chunk_dbc", lambda: lib.ssd_chunk_dbc_split_bwd(sp, P(x), P(bm), P(cm), P(dout), v["states"], v["dstates"], v["q"], v["cs"],
                                                          v["dB"], v["dC"], v["g_last"], split, v["partial"] if split > 1 else None,
                                                          P(status), st)),
        ("chunk_dx", lambda: lib.ssd_chunk_dx_bwd(sp, P(x), P(bm), P(cm), P(dout), v["out"], v["dstates"], v["q"], v["cs"], P(dt),
                                                  P(bias), P(a), v["g_last"], v["dx"], v["ddt_t"], v["dA_part"], P(D), 1, P(status), st)),
        ("dt_finalize", lambda: lib.ssd_dt_finalize_bias_bwd(sp, v["ddt_t"], v["dA_part"], v["ddt"], v["dA"], v["dbias"], st)),
    ]
    for name, call in calls:
        _capi.check(call(), name)
        _check_pads(bufs, status, name)
    for name, pb in bufs.items():
        if name != "partial" or split > 1:
            assert torch.isfinite(pb.view).all() and not bool((pb.view == SENTINEL).any()), name


@pytest.mark.parametrize("with_d,with_z", [(True, True), (False, False)])
@pytest.mark.parametrize("b,l,h,p,n,g,parts", EXTENTS)
def test_whole_calls_stay_inside_their_buffers_and_workspaces(b, l, h, p, n, g, parts, with_d, with_z):
    from ascend_kernel import _capi, mamba2 as M

    dev = torch.device("cuda:0")
    hk = h * parts
    rnd = lambda *s: torch.randn(*s, device=dev)  # noqa: E731
    x, dt, a, bm, cm = rnd(b, l, hk, p), torch.rand(b, l, h, device=dev), -torch.rand(h, device=dev), rnd(b, l, g, n), rnd(b, l, g, n)
    bias, start, dout, dfinal = 0.1 * rnd(h), rnd(b, hk, p, n), rnd(b, l, hk, p), rnd(b, hk, p, n)
    D, z = rnd(h) if with_d else None, rnd(b, l, hk, p) if with_z else None
    shp = M.extents_shape(x, bm, h, True, (0.0, float("inf")))
    sp, lib, st = ctypes.byref(shp), _capi.lib, torch.cuda.current_stream().cuda_stream
    bufs = _between_pads({
        "y": (b, l, hk, p), "out": (b, l, hk, p), "final": (b, hk, p, n), "work": (lib.ssd_forward_work_bytes(sp) // 4,),
        "dx": (b, l, hk, p), "ddt": (b, l, h), "dA": (h,), "dB": (b, l, g, n), "dC": (b, l, g, n), "dD": (h,),
        "dz": (b, l, hk, p), "dbias": (h,), "d_initial": (b, hk, p, n),
        "scratch": (lib.ssd_backward_work_bytes(sp, with_d, with_z) // 4,)}, dev)
    v = {name: pb.view.data_ptr() for name, pb in bufs.items()}
    status = torch.zeros(1, dtype=torch.int32, device=dev)
    P = lambda t: None if t is None else t.data_ptr()  # noqa: E731
    fwd = _capi.SsdForwardArgs(P(x), P(dt), P(bias), P(a), P(bm), P(cm), P(D), P(z), P(start), v["y"], v["out"], v["final"],
                               v["work"], P(status), 1 if with_d else 0)
    bwd = _capi.SsdBackwardArgs(P(x), P(dt), P(bias), P(a), P(bm), P(cm), P(D), P(z), v["y"], P(dout), P(dfinal), v["work"],
                                v["dx"], v["ddt"], v["dA"], v["dB"], v["dC"], v["dD"] if with_d else None,
                                v["dz"] if with_z else None, v["dbias"], v["d_initial"], v["scratch"], P(status), 1 if with_d else 0)
    _capi.check(lib.ssd_forward(sp, ctypes.byref(fwd), 2, st), "ssd_forward")
    _check_pads(bufs, status, "ssd_forward")
    _capi.check(lib.ssd_backward(sp, ctypes.byref(bwd), 2, st), "ssd_backward")
    _check_pads(bufs, status, "ssd_backward")
    for name, pb in bufs.items():
        if name not in ("work", "scratch") and (with_d or name != "dD") and (with_z or name != "dz"):
            assert torch.isfinite(pb.view).all() and not bool((pb.view == SENTINEL).any()), name


@pytest.mark.parametrize("b,l,h,p,n,g", [(2, 17, 4, 33, 36, 2), (1, 1, 3, 64, 128, 1), (3, 32, 2, 5, 4, 1)])
def test_the_recurrence_stays_inside_its_outputs(b, l, h, p, n, g):
    from ascend_kernel import _capi

    dev = torch.device("cuda:0")
    rnd = lambda *s: torch.randn(*s, device=dev)  # noqa: E731
    x, z, dt, a, bm, cm = rnd(b, l, h, p), rnd(b, l, h, p), torch.rand(b, l, h, device=dev), -torch.rand(h, device=dev), rnd(b, l, g, n), rnd(b, l, g, n)
    D, start = rnd(h, p), rnd(b, h, p, n)
    bufs = _between_pads({"out": (b, l, h, p), "final": (b, h, p, n)}, dev)
    shp = _capi.SsdShape(b, l, h, p, n, 128, g, 1, 0.0, float("inf"), 0)
    status = torch.zeros(1, dtype=torch.int32, device=dev)
    P = lambda t: t.data_ptr()  # noqa: E731
    _capi.check(_capi.lib.ssd_recurrent_fwd(ctypes.byref(shp), P(x), P(dt), None, P(a), P(bm), P(cm), P(D), 2, P(z), P(start),
                                            P(bufs["out"].view), P(bufs["final"].view),
                                            torch.cuda.current_stream().cuda_stream), "ssd_recurrent_fwd")
    _check_pads(bufs, status, "ssd_recurrent_fwd")
    for name, pb in bufs.items():
        assert torch.isfinite(pb.view).all() and not bool((pb.view == SENTINEL).any()), name


@pytest.mark.parametrize("b,l,h,p,parts", [(2, 129, 3, 60, 1), (1, 200, 2, 64, 3), (1, 5, 1, 4, 1)])
def test_the_gate_stays_inside_tensors_of_any_extent(b, l, h, p, parts):
    from ascend_kernel import _capi, mamba2 as M

    dev = torch.device("cuda:0")
    hk = h * parts
    rnd = lambda *s: torch.randn(*s, device=dev)  # noqa: E731
    y, x, z, dout, D = rnd(b, l, hk, p), rnd(b, l, hk, p), rnd(b, l, hk, p), rnd(b, l, hk, p), rnd(h)
    shp = M.extents_shape(x, rnd(b, l, 1, 64), h, True, (0.0, float("inf")))
    sp, lib, st = ctypes.byref(shp), _capi.lib, torch.cuda.current_stream().cuda_stream
    bufs = _between_pads({"out": (b, l, hk, p), "dy": (b, l, hk, p), "dz": (b, l, hk, p), "dD": (h,),
                          "part": (lib.ssd_gate_partial_floats(sp),)}, dev)
    v = {name: pb.view.data_ptr() for name, pb in bufs.items()}
    status, P = torch.zeros(1, dtype=torch.int32, device=dev), torch.Tensor.data_ptr
    _capi.check(lib.ssd_gate_skip_fwd(sp, P(y), P(x), P(D), 1, P(z), v["out"], st), "gate_fwd")
    _check_pads(bufs, status, "gate_fwd")
    _capi.check(lib.ssd_gate_skip_bwd(sp, P(dout), P(y), P(x), P(D), 1, P(z), v["dy"], v["dz"], v["part"], v["dD"], st), "gate_bwd")
    _check_pads(bufs, status, "gate_bwd")
    want = M.gate_forward(y, x, None, D, z, h)
    assert torch.equal(bufs["out"].view, want)
    for got, ref in zip((bufs["dy"].view, bufs["dz"].view, bufs["dD"].view), M.gate_backward(dout, y, x, None, D, z, h)):
        assert torch.equal(got, ref)
