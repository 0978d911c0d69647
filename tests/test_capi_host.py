"""Host-side checks that need no GPU: the C-ABI library loads, exports every symbol the header
declares, validates shapes like the reference's host checks, and the Python layer raises the
reference's error types."""
import ctypes
import re
from pathlib import Path

import pytest
import torch

ROOT = Path(__file__).resolve().parent.parent


def _declared_functions():
    text = (ROOT / "include" / "ssd_b200.h").read_text()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return sorted(set(re.findall(r"\b(ssd_[a-z0-9_]+)\s*\(", text)))


def test_library_exports_every_declared_symbol():
    from ascend_kernel import _capi

    names = _declared_functions()
    assert len(names) >= 11
    for name in names:
        assert hasattr(_capi.lib, name), f"{name} declared in include/ssd_b200.h but not exported"
        assert name in _capi.SIGNATURES, f"{name} has no ctypes signature"
    assert sorted(_capi.SIGNATURES) == names


def _shape(b=1, l=128, h=2, p=64, n=64, t=128, g=1, flags=1):
    from ascend_kernel import _capi

    return _capi.SsdShape(b, l, h, p, n, t, g, flags, 0.0, float("inf"), 0)


@pytest.mark.parametrize("kwargs,code", [
    ({}, 0),
    ({"n": 128}, 0),
    ({"b": 0}, -2), ({"l": -1}, -2), ({"h": 3, "g": 2}, -2), ({"t": 0}, -2),   # SSD_ERR_SHAPE
    ({"p": 32}, -3), ({"n": 32}, -3), ({"l": 192}, -3), ({"t": 64}, -3),       # SSD_ERR_UNSUPPORTED
])
def test_check_shape_codes(kwargs, code):
    from ascend_kernel import _capi

    s = _shape(**kwargs)
    assert _capi.lib.ssd_check_shape(ctypes.byref(s)) == code
    assert _capi.error_string(code).startswith("ssd:")


def test_range_limits_have_their_own_code():
    """Sizes one launch cannot index: grid dimensions and the int32 coordinates of the tile loads."""
    from ascend_kernel import _capi

    for kwargs in ({"b": 65536}, {"g": 65536 * 2, "h": 65536 * 2}, {"b": 16384, "l": 131072}):
        assert _capi.lib.ssd_check_shape(ctypes.byref(_shape(**kwargs))) == -4, kwargs
    assert "out of range" in _capi.error_string(-4)
    assert _capi.lib.ssd_check_shape(ctypes.byref(_shape(b=65535))) == 0


def test_buffer_sizes_match_the_layouts_the_python_layer_allocates():
    from ascend_kernel import _capi

    s = _shape(b=2, l=384, h=6, g=3)
    b, l, h, p, n, k = 2, 384, 6, 64, 64, 3
    want = {0: 4 * b * h * l, 1: 4 * b * h * l, 2: 4 * b * h * k * p * n, 3: 4 * b * h * p * n, 4: 4 * b * h * k,
            5: 4 * b * h * l, 6: 8 * b * h * k, 7: 4 * _capi.lib.ssd_gate_partial_floats(ctypes.byref(s)), 8: 4}
    for which, nbytes in want.items():
        assert _capi.lib.ssd_buffer_bytes(ctypes.byref(s), which) == nbytes, which
    assert _capi.lib.ssd_buffer_bytes(ctypes.byref(s), 99) == 0
    assert _capi.lib.ssd_buffer_bytes(ctypes.byref(_shape(p=32)), 0) == 0
    assert _capi.lib.ssd_buffer_bytes(None, 0) == 0


def test_null_pointers_are_rejected_before_any_launch():
    from ascend_kernel import _capi

    s = _shape()
    assert _capi.lib.ssd_dt_cumsum(ctypes.byref(s), None, None, None, None, None, None) == -1
    assert _capi.lib.ssd_check_shape(None) == -1
    with pytest.raises(RuntimeError, match="ssd_dt_cumsum: ssd:"):
        _capi.check(-1, "ssd_dt_cumsum")


def test_python_layer_error_behaviour_matches_reference_style():
    """mamba2_ssd_fwd.cpp:15-112 raises RuntimeError("mamba2_ssd_fwd: ...") before launching."""
    from ascend_kernel import mamba2_ssd_fwd

    x = torch.zeros(1, 128, 2, 64)
    dt = torch.zeros(1, 128, 2)
    a = torch.zeros(2)
    b = torch.zeros(1, 128, 1, 64)
    with pytest.raises(RuntimeError, match="mamba2_ssd_fwd: x must be a CUDA tensor"):
        mamba2_ssd_fwd(x, dt, a, b, b, 64)


def test_validation_order_and_messages():
    from ascend_kernel import mamba2 as M

    class Fake(torch.Tensor):
        """CPU tensor that claims to be on CUDA so the shape checks can run without a device."""
        @property
        def is_cuda(self):
            return True

    def fake(*shape):
        return torch.zeros(*shape).as_subclass(Fake)

    x, dt, a, b = fake(1, 128, 2, 64), fake(1, 128, 2), fake(2), fake(1, 128, 1, 64)
    inf = float("inf")
    M._validate(x, dt, a, b, b, 64, None, None, None, (0.0, inf), None)
    with pytest.raises(RuntimeError, match="dt shape must equal"):
        M._validate(x, fake(1, 128, 3), a, b, b, 64, None, None, None, (0.0, inf), None)
    with pytest.raises(RuntimeError, match="B and C shapes must match"):
        M._validate(x, dt, a, b, fake(1, 128, 1, 32), 64, None, None, None, (0.0, inf), None)
    with pytest.raises(RuntimeError, match="divisible by ngroups"):
        M._validate(fake(1, 128, 3, 64), fake(1, 128, 3), fake(3), fake(1, 128, 2, 64), fake(1, 128, 2, 64), 64,
                    None, None, None, (0.0, inf), None)
    with pytest.raises(RuntimeError, match="chunk_size must be positive"):
        M._validate(x, dt, a, b, b, 0, None, None, None, (0.0, inf), None)
    with pytest.raises(RuntimeError, match="must be contiguous"):
        M._validate(fake(1, 128, 64, 2).transpose(2, 3), dt, a, b, b, 64, None, None, None, (0.0, inf), None)
    with pytest.raises(RuntimeError, match="must be float32"):
        M._validate(x.double().as_subclass(Fake), dt, a, b, b, 64, None, None, None, (0.0, inf), None)
    # optional inputs (mamba2_ssd_fwd.cpp:88-112): accepted with the right shapes, rejected otherwise
    M._validate(x, dt, a, b, b, 64, fake(2), fake(1, 128, 2, 64), fake(2), (1e-3, 1.0), fake(1, 2, 64, 64))
    M._validate(x, dt, a, b, b, 64, fake(2, 64), None, None, (0.0, inf), None)
    with pytest.raises(RuntimeError, match="D shape must equal"):
        M._validate(x, dt, a, b, b, 64, fake(3), None, None, (0.0, inf), None)
    with pytest.raises(RuntimeError, match="z shape must match x"):
        M._validate(x, dt, a, b, b, 64, None, fake(1, 128, 2, 32), None, (0.0, inf), None)
    with pytest.raises(RuntimeError, match="dt_bias shape must equal"):
        M._validate(x, dt, a, b, b, 64, None, None, fake(3), (0.0, inf), None)
    with pytest.raises(RuntimeError, match="initial_states shape must equal"):
        M._validate(x, dt, a, b, b, 64, None, None, None, (0.0, inf), fake(1, 2, 64, 32))
    with pytest.raises(RuntimeError, match="dt_limit min must not exceed max"):
        M._validate(x, dt, a, b, b, 64, None, None, None, (1.0, 0.5), None)


def test_persistent_tile_walk_matches_the_closed_form():
    """The persistent kernels find their (batch, group, tile, head) positions with an incremental, division-free
    walk (carries from token tile to group to batch).  The library's host-side hook runs that walk; here it is
    compared with the closed form for grids and shapes that exercise every carry."""
    import numpy as np

    from ascend_kernel import _capi

    rng = np.random.default_rng(5)
    cases = [(8, 4096, 256, 64, 148), (2, 1408, 14, 14, 148), (2, 4096, 48, 12, 148), (3, 384, 10, 5, 45),
             (1, 128, 7, 7, 7), (5, 640, 12, 3, 148), (2, 256, 6, 1, 4)]
    for _ in range(20):
        g = int(rng.integers(1, 9))
        r = int(rng.integers(1, 5))
        cases.append((int(rng.integers(1, 6)), 128 * int(rng.integers(1, 13)), g * r, g, int(rng.integers(1, 200))))
    for b, l, h, g, grid in cases:
        nchunks, hpg = l // 128, h // g
        tiles = b * g * nchunks
        grid = min(grid, tiles)
        shape = _capi.SsdShape(b, l, h, 64, 64, 128, g, 1, 0.0, float("inf"), 0)
        for cta in {0, grid // 2, grid - 1}:
            my_tiles = (tiles - cta + grid - 1) // grid
            count = my_tiles * hpg
            out = (ctypes.c_int * (4 * count))()
            rc = _capi.lib.ssd_selftest_tile_walk(ctypes.byref(shape), grid, cta, count, out)
            assert rc == 0
            got = np.array(out[:]).reshape(count, 4)
            for it in range(count):
                tile = cta + (it // hpg) * grid
                k, gi, bi = tile % nchunks, (tile // nchunks) % g, tile // (nchunks * g)
                head = gi * hpg + it % hpg
                want = (gi, head, bi * l + k * 128, (bi * h + head) * nchunks + k)
                assert tuple(got[it]) == want, (b, l, h, g, grid, cta, it, tuple(got[it]), want)


@pytest.mark.parametrize("h,p", [(1, 4), (1, 8), (3, 4), (1, 28), (1, 64), (6, 64), (33, 32), (256, 64), (1, 1024)])
@pytest.mark.parametrize("b,l", [(1, 1), (1, 129), (1, 1025), (4, 4096), (2, 1 << 20), (16, 1 << 20)])
def test_partial_sums_of_the_skip_gradient_cover_at_most_128_tokens(h, p, b, l):
    """dD is summed in fp32 inside a block of tokens and in fp64 over the blocks: one partial per block and channel."""
    from ascend_kernel import _capi

    s = _capi.SsdShape(b, l, h, p, 64, 128, 1, 0, 0.0, 0.0, 0)
    blocks, rest = divmod(_capi.lib.ssd_gate_partial_floats(ctypes.byref(s)), h * p)
    assert rest == 0 and 128 * blocks >= b * l


@pytest.mark.parametrize("b,l,h,g", [(2, 384, 24, 2), (1, 128, 12, 1), (3, 256, 30, 5)])
@pytest.mark.parametrize("split", [1, 2, 3, 6])
@pytest.mark.parametrize("blocks", [1, 2])
def test_work_items_of_a_split_group_cover_every_head_once(b, l, h, g, split, blocks):
    """The persistent kernels' walk with the heads of a group dealt to several work items, one set per column block."""
    from ascend_kernel import _capi

    shape = _shape(b=b, l=l, h=h, g=g)
    if (h // g) % split:
        return
    items, per_item, tiles = b * g * split * blocks * (l // 128), h // g // split, l // 128
    for grid in (1, 5, items):
        seen = {}
        for cta in range(grid):
            count = len(range(cta, items, grid)) * per_item
            out = (ctypes.c_int * (6 * count))()
            assert _capi.lib.ssd_selftest_split_walk(ctypes.byref(shape), grid, cta, split, blocks, count, out) == 0
            for i in range(count):
                wg, head, tok0, tile, group, block = out[6 * i:6 * i + 6]
                bb, k = tok0 // l, tok0 % l // 128
                assert group == head // (h // g) and tile == (bb * h + head) * tiles + k
                assert wg // blocks // split == group and block == wg % blocks and head // per_item == wg // blocks
                seen[bb, head, k, block] = seen.get((bb, head, k, block), 0) + 1
        assert len(seen) == b * h * tiles * blocks and set(seen.values()) == {1}


def test_rule_of_the_head_split():
    from ascend_kernel import _capi

    rule = _capi.lib.ssd_selftest_head_split
    for items in (1, 3, 64, 147, 148, 149, 300, 1000, 16 * 148 - 1, 16 * 148):
        for heads in (1, 2, 7, 12, 32):
            for unit, overhead in ((1, 2), (1, 3), (1, 5), (2, 1)):
                split = rule(items, heads, 148, unit, overhead)
                cost = lambda d: -(-items * d // 148) * (2 * -(-heads // d // unit) + overhead)  # noqa: E731
                assert split >= 1 and heads % split == 0
                assert split == 1 or (items < 16 * 148 and items * split <= 32 * 148 and 20 * cost(split) < 19 * cost(1))
    assert rule(320, 8, 148, 1, 2) == 2 and rule(64, 32, 148, 1, 2) > 1 and rule(1, 1, 148, 1, 2) == 1


def test_the_gate_counts_the_tokens_and_heads_of_the_callers_tensors():
    """A shape with SSD_FLAG_EXTENTS says the same to the gate as the tensors' own sizes: partial sums of as many blocks."""
    from ascend_kernel import _capi

    for b, l, h, parts in ((4, 37856, 6, 1), (1, 1000, 3, 4), (2, 129, 2, 16), (1, 256, 2, 2)):
        padded = -(-l // 128) * 128
        ext = _capi.SsdShape(b, padded, h * parts, 64, 64, 128, 1, _capi.SSD_FLAG_EXTENTS | _capi.head_parts_flag(parts), 0.0, 1.0,
                             l if l % 128 else 0)
        own = _capi.SsdShape(b, l, h, 64 * parts, 64, 128, 1, 0, 0.0, 0.0, 0)
        want = _capi.lib.ssd_gate_partial_floats(ctypes.byref(own))
        assert want > 0 and _capi.lib.ssd_gate_partial_floats(ctypes.byref(ext)) == want
        assert _capi.lib.ssd_buffer_bytes(ctypes.byref(ext), 7) == 4 * want


@pytest.mark.parametrize("rows,cols,k,pays", [
    (16384, 902, 192, 1), (16384, 192, 384, 1), (1024, 902, 192, 0), (4096, 192, 384, 0), (2048, 902, 384, 1), (4096, 192, 768, 0),
    (30000, 64, 768, 0), (30000, 96, 768, 1), (1024, 902, 1024, 0), (2048, 902, 1024, 1), (16384, 902, 200, 0), (0, 902, 192, 0),
])
def test_sizes_at_which_the_projection_kernel_pays(rows, cols, k, pays):
    from ascend_kernel import _capi

    assert _capi.lib.ssd_linear_pays(rows, cols, k) == pays
