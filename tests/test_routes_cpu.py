"""Which calls the recurrence kernel and the tile kernels take as they are, and which go to the padded route: decided by sizes
and addresses alone, so tensors on the CPU stand in."""
import pytest
import torch

from ascend_kernel import mamba2 as M


def _tensors(b, l, h, p, g, n, shift=None):
    def make(name, *shape):
        count = 1
        for s in shape:
            count *= s
        t = torch.zeros(count + 1)
        return t[1:].view(shape) if shift == name else t[:count].view(shape)

    return {"x": make("x", b, l, h, p), "B": make("B", b, l, g, n), "C": make("C", b, l, g, n), "D": make("D", h, p),
            "z": make("z", b, l, h, p), "initial_states": make("initial_states", b, h, p, n)}


@pytest.mark.parametrize("l,p,n,taken", [
    (1, 4, 4, True), (127, 60, 100, True), (128, 64, 64, True), (300, 128, 128, True), (300, 1024, 8, True),
    (128, 62, 64, False), (128, 64, 66, False), (128, 96, 64, False), (128, 64, 192, False), (128, 1088, 64, False),
    (0, 64, 64, False),
])
def test_sizes_of_the_tile_kernels(l, p, n, taken):
    assert M._tile_extents(**_tensors(2, l, 2, p, 1, n)) is taken


@pytest.mark.parametrize("name", ["x", "B", "C", "D", "z", "initial_states"])
def test_unaligned_tensors_are_padded_wherever_they_were_before(name):
    assert not M._tile_extents(**_tensors(1, 200, 2, 64, 1, 64, shift=name))
    assert not M._tile_extents(**_tensors(1, 256, 2, 64, 1, 128, shift=name), grad=True)
    assert M._tile_extents(**_tensors(1, 256, 2, 64, 1, 64, shift=name))  # own sizes: refused further down


def test_sizes_of_the_recurrence():
    def taken(b, l, h, p, g, n, shift=None):
        t = _tensors(b, l, h, p, g, n, shift)
        return M._short_sequence(t["x"], t["B"], t["C"], t["D"], t["z"], t["initial_states"])

    assert taken(1, 1, 1, 1, 1, 4) and taken(2, M.SHORT_SEQUENCE, 3, 70, 3, 128) and taken(1, 2, 2, 64, 1, 64, "z")
    assert not taken(1, M.SHORT_SEQUENCE + 1, 2, 64, 1, 64) and not taken(1, 2, 2, 64, 1, 62)
    assert not taken(1, 2, 2, 64, 1, 132) and not taken(1, 2, 2, 64, 1, 64, "B") and not taken(0, 2, 2, 64, 1, 64)
    x = torch.empty(65536, 1, 1, 1)  # a batch beyond the range of the tile kernels is refused there
    assert not M._short_sequence(x, torch.empty(65536, 1, 1, 4), torch.empty(65536, 1, 1, 4), None, None, None)


@pytest.mark.parametrize("l,p,n,grad,taken", [
    (128, 64, 64, False, True), (128, 64, 64, True, True), (128, 64, 128, False, True),  # always without the framework
    (128, 64, 128, True, False), (128, 64, 32, False, False), (128, 64, 96, False, False), (128, 64, 32, True, False),
    (200, 64, 64, False, False), (128, 32, 64, False, False), (128, 128, 64, False, False),
])
def test_derivatives_of_the_framework_epilogue(l, p, n, grad, taken):
    """Under forward-mode derivatives and function transforms D and z stay framework operations wherever they were."""
    t = _tensors(1, l, 2, p, 1, n)
    assert M._tile_extents(**t, grad=grad)
    seen = []

    def inside(z):
        seen.append(M._tile_extents(**dict(t, z=z), grad=grad))
        s = _tensors(1, 4, 2, p, 1, n)
        seen.append(M._short_sequence(s["x"], s["B"], s["C"], s["D"], s["z"], s["initial_states"]))
        return z.sum()

    with torch.autograd.forward_ad.dual_level():
        inside(torch.autograd.forward_ad.make_dual(t["z"], t["z"]))
    torch.func.jvp(inside, (t["z"],), (t["z"],))
    assert seen == [taken, False] * 2
    if not taken:
        torch.func.vmap(inside)(t["z"][None])
        torch.func.grad(inside)(t["z"])
        assert seen == [False] * 8
