"""The recurrence kernel for short sequences, at the edges of its layout, against the token-by-token recurrence in fp64.

Tolerance: everything is fp32.  A result sums at most 128 products, and a state carries at most 32 updates, each rounded
to 2^-24 of its size: 2e-6 of the norm, and q = softplus(dt) with the exp of its product with A adds a few 1e-7."""
import pytest
import torch

pytestmark = pytest.mark.gpu

REL = 3e-6


def _reference(x, dt, A, B, C, D, z, bias, limit, init):
    x, dt, A, B, C = (t.double() for t in (x, dt, A, B, C))
    b, l, h, p = x.shape
    rep = h // B.shape[2]
    q = torch.nn.functional.softplus(dt + (0 if bias is None else bias.double())).clamp(*limit)
    s = torch.zeros(b, h, p, B.shape[3], dtype=torch.float64, device=x.device) if init is None else init.double()
    outs = []
    for t in range(l):
        bt, ct = B[:, t].repeat_interleave(rep, 1), C[:, t].repeat_interleave(rep, 1)
        s = torch.exp(A * q[:, t])[..., None, None] * s + (q[:, t, :, None] * x[:, t])[..., None] * bt[:, :, None]
        outs.append((s * ct[:, :, None]).sum(-1))
    y = torch.stack(outs, 1)
    if D is not None:
        y = y + x * (D.double()[:, None] if D.dim() == 1 else D.double())
    if z is not None:
        y = y * torch.nn.functional.silu(z.double())
    return y, s


@pytest.mark.parametrize("d_dims,with_z,with_init", [(0, False, False), (1, True, True), (2, False, True)])
@pytest.mark.parametrize("b,l,h,p,n,g", [
    (1, 1, 1, 1, 4, 1),       # one row, one column group
    (3, 1, 6, 64, 128, 2),    # whole rows of 32 lanes
    (2, 5, 4, 33, 36, 4),     # a ragged row block, lanes without columns
    (2, 16, 3, 70, 32, 1),    # rows of 8 lanes, two row blocks
    (1, 17, 4, 20, 100, 2),   # one token more than is staged at a time
    (1, 32, 2, 128, 64, 1),   # the longest
])
def test_matches_the_recurrence(b, l, h, p, n, g, d_dims, with_z, with_init):
    import ascend_kernel as ak
    from ascend_kernel import mamba2 as M

    gen = torch.Generator(device="cuda").manual_seed(b * l + h + p + n)
    rnd = lambda *s: torch.randn(*s, generator=gen, device="cuda")  # noqa: E731
    x, B, C = rnd(b, l, h, p), rnd(b, l, g, n), rnd(b, l, g, n)
    dt, A = torch.rand(b, l, h, generator=gen, device="cuda"), -torch.rand(h, generator=gen, device="cuda")
    D = None if d_dims == 0 else rnd(h) if d_dims == 1 else rnd(h, p)
    z = rnd(b, l, h, p) if with_z else None
    init = rnd(b, h, p, n) if with_init else None
    bias = rnd(h) if with_init else None
    limit = (0.3, 1.1) if with_z else (0.0, float("inf"))
    assert M._short_sequence(x, B, C, D, z, init)
    out, final = ak.mamba2_ssd_fwd(x, dt, A, B, C, 64, D=D, z=z, dt_bias=bias, dt_softplus=True, dt_limit=limit,
                                   initial_states=init, return_final_state=True)
    want_out, want_final = _reference(x, dt, A, B, C, D, z, bias, limit, init)
    for got, want in ((out, want_out), (final, want_final)):
        assert got.shape == want.shape
        assert ((got.double() - want).norm() / want.norm()).item() <= REL


def test_tile_kernels_agree_where_the_route_changes():
    import ascend_kernel as ak
    from ascend_kernel import mamba2 as M

    gen = torch.Generator(device="cuda").manual_seed(5)
    rnd = lambda *s: torch.randn(*s, generator=gen, device="cuda")  # noqa: E731
    l = M.SHORT_SEQUENCE
    x, B, C = rnd(2, l, 4, 64), rnd(2, l, 2, 64), rnd(2, l, 2, 64)
    dt, A = torch.rand(2, l, 4, generator=gen, device="cuda"), -torch.rand(4, generator=gen, device="cuda")
    short = ak.mamba2_ssd_fwd(x, dt, A, B, C, 64, dt_softplus=True, return_final_state=True)
    shifted = torch.empty(B.numel() + 1, device="cuda")[1:].view_as(B).copy_(B)  # not 16-byte aligned: the general route
    assert not M._short_sequence(x, shifted, C, None, None, None)
    tiles = ak.mamba2_ssd_fwd(x, dt, A, shifted, C, 64, dt_softplus=True, return_final_state=True)
    for got, want in zip(short, tiles):  # the tile kernels keep 16 bits of each operand
        assert ((got - want).norm() / want.norm()).item() <= 3e-5
