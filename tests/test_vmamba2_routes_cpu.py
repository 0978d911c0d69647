"""Which projections of the Vision block run as the library's own kernel, which takes bare pointers: decided by the layer and
its tensors alone, so that tensors on the CPU stand in.  What is not taken goes to the layer."""
import pytest
import torch

from ascend_kernel import vmamba2 as V


def _layer(n=96, k=64, **kw):
    return torch.nn.Linear(k, n, bias=False, **kw)


@pytest.mark.parametrize("shape,residual,taken", [
    ((3, 5, 64), None, True), ((64,), None, True), ((3, 5, 64), (3, 5, 96), True),
    ((3, 5, 128), None, False),          # twice the layer's width: twice the rows
    ((3, 5, 32), None, False),           # half of it
    ((3, 5, 64), (96,), False),          # a residual that the framework would broadcast
    ((3, 5, 64), (3, 1, 96), False),
    ((3, 5, 64), (5, 3, 96), False),
])
def test_widths_and_residuals_that_fit(shape, residual, taken):
    r = None if residual is None else torch.zeros(residual)
    assert V._plain_projection(_layer(), torch.zeros(shape), r) is taken


def test_a_width_that_does_not_fit_is_refused_by_the_layer():
    with torch.no_grad(), pytest.raises(RuntimeError):
        V._linear(_layer(), torch.zeros(3, 128))


@pytest.mark.parametrize("where", ["weight", "x", "residual"])
def test_tensors_of_different_devices_are_left_to_the_layer(where):
    dev = lambda name: "meta" if name == where else "cpu"  # noqa: E731
    x, r = torch.zeros(3, 64, device=dev("x")), torch.zeros(3, 96, device=dev("residual"))
    assert not V._plain_projection(_layer(device=dev("weight")), x, r)


@pytest.mark.parametrize("value,taken", [("ieee", True), ("none", True), ("tf32", False)])
def test_the_precision_policy_of_either_interface_is_kept(value, taken):
    matmul = torch.backends.cuda.matmul
    before = matmul.fp32_precision
    try:
        matmul.fp32_precision = value
        assert V._plain_projection(_layer(), torch.zeros(3, 64), None) is taken
    finally:
        matmul.fp32_precision = before
    try:
        torch.set_float32_matmul_precision("high")
        assert not V._plain_projection(_layer(), torch.zeros(3, 64), None)
    finally:
        torch.set_float32_matmul_precision("highest")
        matmul.fp32_precision = before


def test_autocast_and_hooks_are_left_to_the_layer():
    layer, x = _layer(), torch.zeros(3, 64)
    try:
        torch.set_autocast_enabled("cuda", True)
        assert not V._plain_projection(layer, x, None)
    finally:
        torch.set_autocast_enabled("cuda", False)
    handle = layer.register_forward_pre_hook(lambda *a: None)
    assert not V._plain_projection(layer, x, None)
    handle.remove()
    handle = torch.nn.modules.module.register_module_forward_hook(lambda *a: None)
    assert not V._plain_projection(layer, x, None)
    handle.remove()
    assert V._plain_projection(layer, x, None)


class _Wrapped(torch.Tensor):
    """A tensor subclass, as quantisation and sharding libraries put in place of a weight."""


def test_weights_and_inputs_without_storage_of_their_own_are_left_to_the_layer():
    layer, x = _layer(), torch.zeros(3, 64)
    layer.weight = torch.nn.Parameter(torch.zeros(96, 64).as_subclass(_Wrapped))
    assert not V._plain_projection(layer, x, None)
    assert not V._plain_projection(_layer(), x.as_subclass(_Wrapped), None)
    assert not V._plain_projection(_layer(), x, torch.zeros(3, 96).as_subclass(_Wrapped))
    taken, layer = [], _layer()

    def of_one(row):
        taken.append(V._plain_projection(layer, row, None))
        return row

    torch.func.vmap(of_one)(x)
    assert taken == [False]


def test_other_layers_are_left_alone():
    assert not V._plain_projection(torch.nn.Identity(), torch.zeros(3, 64), None)
    assert not V._plain_projection(torch.nn.Linear(64, 96), torch.zeros(3, 64), None)  # with a bias


def test_a_replaced_forward_is_kept():
    layer = _layer()
    layer.forward = lambda x: x
    assert not V._plain_projection(layer, torch.zeros(3, 64), None)


@pytest.mark.parametrize("t,taken", [
    (torch.ones(6), True), (torch.nn.Parameter(torch.ones(6)), True),
    (torch.ones(6, 64), False), (torch.ones(1), False), (torch.ones(()), False), (torch.ones(12)[::2], False),
    (torch.ones(6, dtype=torch.float64), False), (torch.ones(6, device="meta"), False),
    (torch.ones(6).as_subclass(_Wrapped), False),
])
def test_per_head_parameters_that_the_block_kernels_read(t, taken):
    assert V._per_head(t, torch.device("cpu"), 6) is taken


def test_kernels_run_on_the_device_and_stream_of_their_tensors(monkeypatch):
    import contextlib

    from ascend_kernel import mamba2 as M

    current = ["cuda:0"]

    @contextlib.contextmanager
    def guard(device):
        before, current[0] = current[0], str(device)
        yield
        current[0] = before

    monkeypatch.setattr(M, "_device_guard", guard)
    monkeypatch.setattr(M, "_stream", lambda: "stream of " + current[0])
    calls = []
    V._launch("norm", torch.device("cuda:1"), lambda *a: calls.append(a) or 0, 7)
    assert calls == [(7, "stream of cuda:1")] and current == ["cuda:0"]
    with pytest.raises(RuntimeError):
        V._launch("norm", torch.device("cuda:1"), lambda *a: -3)
