"""Shapes with fewer (batch, group, tile) work items than SMs, where the heads of a group are dealt to several work items:
every divisor class of the heads per group, against the fp64 oracle.

Tolerance: that of the tensor-core path anywhere else (operands with 16 mantissa bits, fp32 sums): 3e-5 of the norm on every
output and gradient but ddt, a suffix sum of up to 128 signed terms (sqrt(128) * 6e-6 of a term: 1e-4), and dA, whose sum over
all tokens cancels (2e-3, as the parity tests allow)."""
import pytest
import torch

from oracle import ssd_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [
    (1, 128, 2, 64, 64, 64, 1),     # one tile, one head per work item
    (1, 128, 7, 64, 64, 64, 1),     # a prime number of heads: all or none
    (1, 256, 12, 64, 64, 64, 1),    # many divisors, pairs in the state kernel
    (2, 384, 18, 64, 64, 64, 2),    # nine heads per group
    (1, 128, 32, 64, 64, 64, 1),    # the largest split
    (3, 640, 10, 64, 64, 64, 2),    # several tiles per work item walk
])
def test_forward_and_backward(shape):
    from ascend_kernel import check_status, mamba2_ssd_fwd

    inputs = O.make_inputs(shape, 3)
    want = O.fp64_forward_backward(*inputs, shape[5], dt_softplus=True)
    leaves = [t.cuda().requires_grad_(True) for t in inputs]
    out, final = mamba2_ssd_fwd(*leaves, shape[5], dt_softplus=True, return_final_state=True)
    O.loss_fn(out, final).backward()
    check_status()
    got = [out.detach(), final.detach()] + [t.grad for t in leaves]
    for g, w, name in zip(got, want, ["out", "final", "dx", "ddt", "dA", "dB", "dC"]):
        assert O.rel_l2(g.cpu(), w) <= (2e-3 if name == "dA" else 1e-4 if name == "ddt" else 3e-5), name


@pytest.mark.parametrize("shape", [(1, 128, 6, 64, 128, 64, 1), (1, 384, 16, 64, 128, 64, 2)])
def test_forward_with_state_size_128(shape):
    from ascend_kernel import check_status, mamba2_ssd_fwd

    inputs = O.make_inputs(shape, 4)
    want = O.fp64_forward_backward(*inputs, shape[5], dt_softplus=True)
    out, final = mamba2_ssd_fwd(*(t.cuda() for t in inputs), shape[5], dt_softplus=True, return_final_state=True)
    check_status()
    assert O.rel_l2(out.cpu(), want[0]) <= 3e-5 and O.rel_l2(final.cpu(), want[1]) <= 3e-5


def test_work_item_walk_with_a_split():
    """What a split must not change: with it or without, the stages give the same bits where no sum crosses heads."""
    from ascend_kernel import mamba2 as M

    shape = (2, 256, 8, 64, 64, 64, 1)
    x, dt, A, B, C = (t.cuda() for t in O.make_inputs(shape, 9))
    few = M.forward_stages(x, dt, A, B, C, True)
    rep = lambda t: t.repeat(80, 1, 1, 1)  # noqa: E731  (enough work items that no split pays)
    many = M.forward_stages(rep(x), dt.repeat(80, 1, 1), A, rep(B), rep(C), True)
    assert torch.equal(few[0], many[0][:2]) and torch.equal(few[0], many[0][-2:])
    assert torch.allclose(few[1], many[1][:2], rtol=1e-5, atol=1e-5)
