"""The projection kernel (three bf16 parts per operand) at the edges of its tiles, against fp64.

Tolerance: the parts hold 24 bits and the dropped products are below 2^-24; an accumulator truncates on each of its four
additions of full size, at most 2^-23 of its sum each, and the accumulators are added with rounding: 5e-7 up to K = 384, 1e-6
beyond leave room for both."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("residual", [False, True])
@pytest.mark.parametrize("rows,cols,k", [
    (1, 1, 64),        # one row, one column, one block of K
    (128, 96, 192),    # exactly one tile
    (129, 97, 128),    # one row and one column more, two blocks
    (300, 902, 192),   # rows of 8-byte alignment only, the tiles of a row dealt to several CTAs
    (130, 192, 384),   # two chunks of K
    (70, 200, 576),    # three chunks, three tiles on two CTAs
    (20000, 300, 64),  # more row tiles than SMs, several tiles per CTA
])
def test_against_fp64(rows, cols, k, residual):
    from ascend_kernel import _capi, check_status, mamba2 as M

    gen = torch.Generator(device="cuda").manual_seed(rows + cols + k)
    rnd = lambda *s: torch.randn(*s, generator=gen, device="cuda")  # noqa: E731
    x, w, r = rnd(rows, k), rnd(cols, k), rnd(rows, cols)
    out = torch.full((rows * cols + 64,), float("nan"), device="cuda")
    work = torch.empty(_capi.lib.ssd_linear_work_bytes(cols, k), device="cuda", dtype=torch.uint8)
    _capi.check(_capi.lib.ssd_linear_fwd(x.data_ptr(), w.data_ptr(), r.data_ptr() if residual else None, out.data_ptr(), rows,
                                         cols, k, work.data_ptr(), M._status(x.device).data_ptr(),
                                         torch.cuda.current_stream().cuda_stream), "linear")
    check_status()
    want = x.double() @ w.double().T + (r.double() if residual else 0)
    got = out[:rows * cols].view(rows, cols).double()
    assert torch.isnan(out[rows * cols:]).all()  # nothing beyond the end
    assert ((got - want).norm() / want.norm()).item() <= (5e-7 if k <= 384 else 1e-6)


def test_sizes_that_are_not_taken():
    from ascend_kernel import _capi

    assert _capi.lib.ssd_linear_work_bytes(100, 100) == 0 and _capi.lib.ssd_linear_pays(1 << 20, 100, 100) == 0
    x = torch.zeros(64, 104, device="cuda")
    args = (x.data_ptr(), x.data_ptr(), None, x.data_ptr(), 4, 4, 104, x.data_ptr(), x.data_ptr(), None)
    assert _capi.lib.ssd_linear_fwd(*args) == -3


def test_layers_with_hooks_or_a_lower_precision_policy_are_left_alone():
    from ascend_kernel import vmamba2 as V

    layer = torch.nn.Linear(192, 902, bias=False).cuda()
    x = torch.randn(4096, 192, device="cuda")
    seen = []
    with torch.no_grad():
        plain = V._linear(layer, x)
        assert ((plain - layer(x)).norm() / plain.norm()).item() < 1e-6
        handle = layer.register_forward_hook(lambda *a: seen.append(1))
        assert torch.equal(V._linear(layer, x), layer(x)) and len(seen) == 2
        handle.remove()
        matmul, before = torch.backends.cuda.matmul, torch.backends.cuda.matmul.fp32_precision
        try:
            matmul.fp32_precision = "tf32"
            assert torch.equal(V._linear(layer, x), layer(x)) and not torch.equal(layer(x), plain)
        finally:
            matmul.fp32_precision = before
        with torch.autocast("cuda", dtype=torch.bfloat16):
            assert V._linear(layer, x).dtype == torch.bfloat16
    assert V._linear(layer, x).requires_grad  # with gradients: the layer


def _run(x, w, residual=None):
    from ascend_kernel import _capi, check_status, mamba2 as M

    (rows, k), cols = x.shape, w.shape[0]
    out = torch.full((rows, cols), float("nan"), device="cuda")
    work = torch.empty(_capi.lib.ssd_linear_work_bytes(cols, k), device="cuda", dtype=torch.uint8)
    _capi.check(_capi.lib.ssd_linear_fwd(x.data_ptr(), w.data_ptr(), residual.data_ptr() if residual is not None else None,
                                         out.data_ptr(), rows, cols, k, work.data_ptr(), M._status(x.device).data_ptr(),
                                         torch.cuda.current_stream().cuda_stream), "linear")
    check_status()
    return out


@pytest.mark.parametrize("one_sign", [False, True])
@pytest.mark.parametrize("k", [64, 128, 192, 256, 320, 384, 448, 576, 768, 1536])
def test_error_is_no_larger_than_that_of_an_fp32_product(k, one_sign):
    """Against fp64, beside the framework's fp32 product of the same operands, at sizes that this kernel takes over: of both signs,
    and of one sign, where truncated additions add up.  K over every split into chunks: whole ones, ones filled up with zeros
    (320, 448), two to eight."""
    gen = torch.Generator(device="cuda").manual_seed(k)
    x, w = (torch.randn(s, k, generator=gen, device="cuda") for s in (2100, 902))
    if one_sign:
        x, w = x.abs(), w.abs()
    want = x.double() @ w.double().T
    assert torch.backends.cuda.matmul.fp32_precision in ("none", "ieee")
    ours, library = (((v.double() - want).norm() / want.norm()).item() for v in (_run(x, w), x @ w.T))
    assert ours <= library, (ours, library)


@pytest.mark.parametrize("k", [64, 256])
def test_infinities_nan_and_the_largest_values(k):
    inf, nan, largest = float("inf"), float("nan"), torch.finfo(torch.float32).max
    x, w = torch.randn(140, k, device="cuda"), torch.randn(100, k, device="cuda")
    x[3, 5], x[4, 6], x[5, 7], x[5, 8], x[6, 9] = inf, -inf, inf, -inf, nan
    w[7, 5], w[8, 5], w[9, 11], w[10, 12] = inf, 0.0, -inf, nan
    x[20, 11] = 0.0
    x[130], x[130, 13] = 0.0, largest
    w[:, 13] = 0.5 * torch.sign(w[:, 13])
    got, want = _run(x, w), x.double() @ w.double().T
    assert torch.equal(torch.isnan(got), torch.isnan(want))
    assert torch.equal(torch.isposinf(got), torch.isposinf(want)) and torch.equal(torch.isneginf(got), torch.isneginf(want))
    finite = torch.isfinite(want)
    assert finite[130, :7].all() and ((got[130, :7].double() - want[130, :7]).abs() <= 1e-6 * want[130, :7].abs()).all()
    finite[130] = False
    assert ((got.double() - want)[finite].norm() / want[finite].norm()).item() <= 5e-7
