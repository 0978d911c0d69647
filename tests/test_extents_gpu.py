"""The tile kernels on tensors of any length, headdim and state size (tiles cut off at the tensors' ends instead of padded
copies), against the fp64 oracle and against the padded route.

Tolerance: that of the tensor-core path (operands with 16 mantissa bits, fp32 sums; 6e-6 of the norm per product), 3e-5 of
the norm.  ddt is a suffix sum of up to 128 such terms of either sign, whose errors add up to sqrt(128) * 6e-6 = 7e-5 of a
term while the sum may be no larger than one: 1e-4.  Gradients of per-head scalars are sums over all tokens that
cancel: 2e-3, as the parity tests allow."""
import pytest
import torch

from oracle import ssd_oracle as O

pytestmark = pytest.mark.gpu

SCALARS = ("dA", "dD", "dbias")
CASES = [  # b, l, h, p, n, g
    (1, 1, 1, 4, 4, 1),        # one token, one quad
    (2, 127, 4, 32, 32, 2),    # one token short of a tile, half the channels and columns
    (2, 129, 3, 60, 36, 3),    # one token over; quads that end inside a box of 32
    (1, 300, 6, 64, 96, 2),    # state columns that end inside the second block
    (2, 256, 4, 64, 128, 2),   # whole tiles, two column blocks
    (1, 257, 8, 36, 100, 1),   # everything ragged, head split
    (2, 200, 2, 128, 64, 1),   # two kernel heads per head
    (1, 384, 4, 192, 128, 2),  # three, two column blocks
    (1, 128, 3, 20, 64, 1),    # fewer channels than one box
]


def _inputs(b, l, h, p, n, g, full, seed=7):
    gen = torch.Generator().manual_seed(seed)
    rnd = lambda *s: torch.randn(*s, generator=gen)  # noqa: E731
    t = {"x": rnd(b, l, h, p), "dt": torch.rand(b, l, h, generator=gen), "A": -torch.rand(h, generator=gen),
         "B": rnd(b, l, g, n), "C": rnd(b, l, g, n)}
    if full:
        t.update(D=rnd(h) if full == 1 else rnd(h, p), z=rnd(b, l, h, p), dt_bias=0.3 * rnd(h), initial_states=rnd(b, h, p, n))
    return t, rnd(b, l, h, p), rnd(b, h, p, n)


def _call(fn, t, **kw):
    return fn(t["x"], t["dt"], t["A"], t["B"], t["C"], 64, D=t.get("D"), z=t.get("z"), dt_bias=t.get("dt_bias"),
              dt_softplus=True, dt_limit=(0.01, 1.5), initial_states=t.get("initial_states"), return_final_state=True, **kw)


def _ours(t, gout, gfinal):
    from ascend_kernel import check_status, mamba2_ssd_fwd

    leaves = {k: v.cuda().requires_grad_(True) for k, v in t.items()}
    out, final = _call(mamba2_ssd_fwd, leaves)
    grads = torch.autograd.grad([out, final], list(leaves.values()), [gout.cuda(), gfinal.cuda()])
    check_status()
    return [out.detach(), final.detach()] + list(grads)


def _names(t):
    return ["out", "final"] + ["d" + {"dt_bias": "bias"}.get(k, k) for k in t]


def _close(got, want, names):
    for g, w, nm in zip(got, want, names):
        assert g.shape == w.shape, nm
        assert O.rel_l2(g.cpu(), w.cpu()) <= (2e-3 if nm in SCALARS else 1e-4 if nm == "ddt" else 3e-5), nm


@pytest.mark.parametrize("full", [0, 1, 2])
@pytest.mark.parametrize("case", CASES)
def test_against_the_oracle(case, full):
    from ascend_kernel import mamba2 as M

    t, gout, gfinal = _inputs(*case, full)
    assert M._tile_extents(*(t[k].cuda() for k in "xBC"), None, None, None)
    leaves = {k: v.double().requires_grad_(True) for k, v in t.items()}
    out, final = _call(O.ssd_chunked, leaves, compute_dtype=None)
    want = [out.detach(), final.detach()] + list(torch.autograd.grad([out, final], list(leaves.values()),
                                                                     [gout.double(), gfinal.double()]))
    _close(_ours(t, gout, gfinal), want, _names(t))


@pytest.mark.parametrize("policy", ["save", "recompute"])
@pytest.mark.parametrize("case", CASES)
def test_against_the_padded_route(case, policy, monkeypatch):
    from ascend_kernel import mamba2 as M

    t, gout, gfinal = _inputs(*case, 1, seed=8)
    previous = M.set_save_policy(policy)
    try:
        new = _ours(t, gout, gfinal)
        monkeypatch.setattr(M, "_tile_extents", lambda *a: False)
        _close(new, _ours(t, gout, gfinal), _names(t))
    finally:
        M.set_save_policy(previous)


def test_fused_state_scan_on_cut_off_states():
    from ascend_kernel import set_state_scan

    t, gout, gfinal = _inputs(2, 300, 8, 36, 44, 4, 1, seed=9)
    previous = set_state_scan("on")
    try:
        fused = _ours(t, gout, gfinal)
        set_state_scan("off")
        _close(fused, _ours(t, gout, gfinal), _names(t))
    finally:
        set_state_scan(previous)


def test_output_may_be_changed_in_place_and_gradients_may_be_unaligned():
    from ascend_kernel import mamba2_ssd_fwd

    t, gout, gfinal = _inputs(2, 200, 4, 32, 128, 2, 0, seed=10)
    want = _ours(t, gout, gfinal)
    leaves = {k: v.cuda().requires_grad_(True) for k, v in t.items()}
    out, final = _call(mamba2_ssd_fwd, leaves)
    out.mul_(2.0)
    shifted = torch.empty(gout.numel() + 1, device="cuda")[1:].view_as(out).copy_(0.5 * gout)
    grads = torch.autograd.grad([out, final], list(leaves.values()), [shifted, gfinal.cuda()])
    _close(grads, want[2:], _names(t)[2:])


def test_gradients_of_the_epilogue_alone():
    from ascend_kernel import mamba2_ssd_fwd

    t, gout, gfinal = _inputs(1, 150, 4, 32, 64, 1, 2, seed=11)
    want = dict(zip(_names(t), _ours(t, gout, gfinal)))
    leaves = {k: v.cuda().requires_grad_(k in ("D", "z")) for k, v in t.items()}
    out, _ = _call(mamba2_ssd_fwd, leaves)
    dD, dz = torch.autograd.grad(out, [leaves["D"], leaves["z"]], gout.cuda())
    assert torch.equal(dz, want["dz"]) and torch.equal(dD, want["dD"])
