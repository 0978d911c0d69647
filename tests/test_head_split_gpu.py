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


# slots per SM, heads treated at once and overhead of each kernel's call of the rule: state, output, dB / dC, dx
RULES = ((2, 2, 1), (1, 1, 2), (1, 1, 5), (1, 1, 3))


def test_work_item_walk_with_a_split():
    """What a split must not change: with it and without, the stages give the same bits where no sum crosses heads."""
    from ascend_kernel import _capi, mamba2 as M

    sms = torch.cuda.get_device_properties(0).multi_processor_count
    times = 16 * sms // 2  # enough work items that the rule does not split for any kernel
    shape = (2, 256, 4, 64, 64, 64, 1)
    for per_sm, unit, overhead in RULES:
        rule = lambda items: _capi.lib.ssd_selftest_head_split(items, 4, per_sm * sms, unit, overhead)  # noqa: E731
        assert rule(4) > 1 and rule(4 * times) == 1
    x, dt, A, B, C = (t.cuda() for t in O.make_inputs(shape, 9))
    dout = torch.randn(x.shape, device="cuda")
    rep = lambda t: t.repeat(times, *[1] * (t.dim() - 1))  # noqa: E731
    previous = M.set_state_scan("off")  # the tile-parallel state kernel for both
    try:
        results = []
        for f in (lambda t: t, rep):
            xs, dts, Bs, Cs, ds = (f(t) for t in (x, dt, B, C, dout))
            out, final, q, cs, states = M.forward_stages(xs, dts, A, Bs, Cs, True)
            dx, ddt, _, dB, dC, _ = M.backward_stages(xs, dts, A, Bs, Cs, out, q, cs, states, ds, None, True)
            results.append([(t[:2].clone(), t[-2:].clone()) for t in (out, final, states, dx, ddt, dB, dC)])
            del xs, dts, Bs, Cs, ds, out, final, q, cs, states, dx, ddt, dB, dC
    finally:
        M.set_state_scan(previous)
    M.check_status()
    for name, (few, _), (first, last) in zip(("out", "final", "states", "dx", "ddt", "dB", "dC"), *results):
        assert torch.equal(first, last), name
        if name in ("dB", "dC"):  # sums over the heads of a group, in another order
            assert ((few - first).norm() <= 1e-5 * first.norm()).item(), name
        else:
            assert torch.equal(few, first), name


def test_partial_gradients_of_every_split():
    from ascend_kernel import _capi, mamba2 as M

    import ctypes

    shape = (2, 256, 8, 64, 64, 64, 2)
    x, dt, A, B, C = (t.cuda() for t in O.make_inputs(shape, 10))
    dout = torch.randn(x.shape, device="cuda")
    out, _, q, cs, states = M.forward_stages(x, dt, A, B, C, True)
    dstates, s = torch.randn_like(states), M.make_shape(x, B, True)
    status, results = M._status(x.device), []
    for split in (1, 2, 4):
        dB, dC, g_last = torch.empty_like(B), torch.empty_like(C), torch.empty(2, 8, 2, device="cuda")
        part = torch.full((2 * split * B.numel(),), float("nan"), device="cuda")
        _capi.check(_capi.lib.ssd_chunk_dbc_split_bwd(
            ctypes.byref(s), x.data_ptr(), B.data_ptr(), C.data_ptr(), dout.data_ptr(), states.data_ptr(), dstates.data_ptr(),
            q.data_ptr(), cs.data_ptr(), dB.data_ptr(), dC.data_ptr(), g_last.data_ptr(), split,
            part.data_ptr() if split > 1 else None, status.data_ptr(), torch.cuda.current_stream().cuda_stream), "dbc")
        results.append((dB, dC, g_last))
    M.check_status()
    for dB, dC, g_last in results[1:]:
        assert torch.equal(g_last, results[0][2])  # per head
        for got, want in ((dB, results[0][0]), (dC, results[0][1])):
            assert ((got - want).norm() <= 1e-5 * want.norm()).item()
    assert _capi.lib.ssd_chunk_dbc_split_bwd(*[ctypes.byref(s)] + [x.data_ptr()] * 11, 3, x.data_ptr(), status.data_ptr(), None) == -2
