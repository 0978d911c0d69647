"""Derivatives that the framework takes of the D skip connection and the z gate, at sizes where these are framework
operations under a transform: forward mode, vmap, and gradients that are batched or differentiated again, against the closed
form on the SSD output.

Tolerance: both sides start from the same SSD output, up to the fp32 rounding of the element-wise operations: 1e-5."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu

SHAPES = [(2, 256, 3, 64, 32, 1), (1, 128, 2, 64, 96, 2), (1, 200, 2, 64, 64, 1), (2, 5, 2, 64, 64, 1), (1, 128, 2, 32, 64, 1)]


def _case(shape):
    from ascend_kernel import mamba2_ssd_fwd

    b, l, h, p, n, g = shape
    gen = torch.Generator(device="cuda").manual_seed(5)
    rnd = lambda *s: torch.randn(*s, generator=gen, device="cuda")  # noqa: E731
    x, dt, A, B, C = rnd(b, l, h, p), rnd(b, l, h).abs(), -rnd(h).abs(), rnd(b, l, g, n), rnd(b, l, g, n)
    call = lambda D, z: mamba2_ssd_fwd(x, dt, A, B, C, 64, D=D, z=z, dt_softplus=True)  # noqa: E731
    y = call(None, None)

    def closed(D, z):
        return (y + x * D.view(1, 1, -1, 1)) * F.silu(z)

    return call, closed, rnd(h), rnd(b, l, h, p), rnd(h), rnd(b, l, h, p)


@pytest.mark.parametrize("shape", SHAPES)
def test_transforms_of_the_skip_connection_and_the_gate(shape):
    import torch.autograd.forward_ad as fwd

    call, closed, D, z, tD, tz = _case(shape)
    want = torch.func.jvp(closed, (D, z), (tD, tz))
    close = lambda a, b: ((a - b).norm() <= 1e-5 * b.norm()).item()  # noqa: E731
    with torch.no_grad(), fwd.dual_level():
        out = fwd.unpack_dual(call(fwd.make_dual(D, tD), fwd.make_dual(z, tz)))
        assert out.tangent is not None and close(out.primal, want[0]) and close(out.tangent, want[1])
    with torch.no_grad():
        stack = torch.stack([D, tD]), torch.stack([z, tz])
        assert close(torch.func.vmap(call)(*stack), torch.func.vmap(closed)(*stack))


@pytest.mark.parametrize("policy", ["save", "recompute"])
@pytest.mark.parametrize("alone", [False, True])
@pytest.mark.parametrize("shape", [(2, 256, 3, 64, 32, 1), (1, 200, 2, 64, 64, 1), (1, 128, 2, 64, 128, 1), (1, 130, 2, 128, 64, 1)])
def test_gradients_that_are_differentiated_again(shape, alone, policy):
    """create_graph at sizes other than the kernels' own: D and z as around the plain call."""
    import ascend_kernel as ak

    b, l, h, p, n, g = shape
    gen = torch.Generator(device="cuda").manual_seed(6)
    rnd = lambda *s: torch.randn(*s, generator=gen, device="cuda")  # noqa: E731
    t = [rnd(b, l, h, p), rnd(b, l, h).abs(), -rnd(h).abs(), rnd(b, l, g, n), rnd(b, l, g, n)]
    D, z, start, bias, up = rnd(h), rnd(b, l, h, p), rnd(b, h, p, n), 0.1 * rnd(h), rnd(b, l, h, p)
    inputs = [D, z, up] if alone else [*t, D, z, start, bias, up]
    for v in inputs:
        v.requires_grad_(True)
    weights = [rnd(*v.shape) for v in inputs[:-1]]

    def second(fused):
        kw = dict(dt_bias=bias, initial_states=start, dt_softplus=True)
        out = ak.mamba2_ssd_fwd(*t, 64, **(dict(kw, D=D, z=z) if fused else kw))
        if not fused:
            out = (out + t[0] * D.view(1, 1, -1, 1)) * F.silu(z)
        first = torch.autograd.grad(out, inputs[:-1], up, create_graph=True)
        return first + torch.autograd.grad(sum((w * v).sum() for w, v in zip(weights, first)), inputs, allow_unused=True)

    previous = ak.set_save_policy(policy)
    try:
        for got, want in zip(second(True), second(False)):
            assert (got is None) == (want is None)
            assert got is None or ((got - want).norm() <= 1e-5 * want.norm()).item()
        if alone:
            ups = torch.stack([up, 2 * up]).detach()
            batched = torch.autograd.grad(ak.mamba2_ssd_fwd(*t, 64, D=D, z=z, dt_softplus=True), [D, z], ups, is_grads_batched=True)
            assert all(torch.allclose(v[1], 2 * v[0], rtol=1e-5, atol=1e-6 * v.abs().max().item()) for v in batched)
    finally:
        ak.set_save_policy(previous)


@pytest.mark.parametrize("shape", [(1, 256, 2, 64, 64, 1), (1, 200, 2, 32, 100, 1)])
def test_saved_tensor_hooks_that_convert(shape):
    """Hooks that keep everything in another type.  fp64 holds every fp32 value, so the gradients are the same bits (bf16 would
    round cs, a logarithm of decay of up to a hundred, by up to 0.2)."""
    from ascend_kernel import mamba2_ssd_fwd

    b, l, h, p, n, g = shape
    gen = torch.Generator(device="cuda").manual_seed(8)
    rnd = lambda *s: torch.randn(*s, generator=gen, device="cuda")  # noqa: E731
    t = [rnd(b, l, h, p), rnd(b, l, h).abs(), -rnd(h).abs(), rnd(b, l, g, n), rnd(b, l, g, n)]
    for v in t:
        v.requires_grad_(True)
    up = rnd(b, l, h, p)
    want = torch.autograd.grad(mamba2_ssd_fwd(*t, 64, dt_softplus=True), t, up)
    with torch.autograd.graph.saved_tensors_hooks(lambda v: v.double(), lambda v: v.float()):
        out = mamba2_ssd_fwd(*t, 64, dt_softplus=True)
    for got, ref in zip(torch.autograd.grad(out, t, up), want):
        assert torch.equal(got, ref)


def test_what_is_kept_for_gradients_of_the_epilogue_alone():
    from ascend_kernel import SavedTensorStats, mamba2_ssd_fwd

    b, l, h, p, n, g = 1, 1000, 4, 64, 128, 1
    rnd = lambda *s: torch.randn(*s, device="cuda")  # noqa: E731
    x, dt, A, B, C, z = rnd(b, l, h, p), rnd(b, l, h).abs(), -rnd(h).abs(), rnd(b, l, g, n), rnd(b, l, g, n), rnd(b, l, h, p)
    z.requires_grad_(True)
    stats = SavedTensorStats()
    with stats.hooks():
        out, final = mamba2_ssd_fwd(x, dt, A, B, C, 64, z=z, dt_softplus=True, return_final_state=True)
    assert out.requires_grad and not final.requires_grad  # the state does not depend on z
    inputs = sum(4 * t.numel() for t in (x, dt, A, B, C, z))
    assert stats.unique_bytes <= inputs + 4 * out.numel() + 4096  # and the output before the gate, no states
    assert torch.isfinite(torch.autograd.grad(out.sum(), z)[0]).all()
