"""The projection kernel (three bf16 parts per operand) at the edges of its tiles, against fp64.

Tolerance: the parts hold 24 bits and the dropped products are below 2^-24; the accumulator truncates on each of the
K / 16 additions of full size, at most 2^-23 of the sum each and on average a tenth of that: 5e-7 up to K = 384, 1e-6 beyond."""
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
    assert V._linear(layer, x).requires_grad  # with gradients: the layer
