"""The bandwidth-bound kernels at the edges of how they lay a shape over CTAs, against the same formulas in fp64.

Tolerances: each result is a handful of fp32 operations per element (relative error a few times 2^-24 of its largest
term; __expf adds about 2^-21), sums run in fp32 over at most 128 terms and in fp64 above that: 5e-6 of the norm."""
import pytest
import torch

pytestmark = pytest.mark.gpu

REL = 5e-6


def _rel(got, want):
    return ((got.double() - want).norm() / want.norm().clamp_min(1e-300)).item()


@pytest.mark.parametrize("with_z", [False, True])
@pytest.mark.parametrize("d_dims", [0, 1, 2])
@pytest.mark.parametrize("b,l,h,p", [
    (1, 1, 1, 4),        # one float4
    (1, 3, 5, 12),       # a row of 15 threads, 17 rows side by side, fewer tokens than that
    (2, 129, 6, 64),     # two rows side by side, the last row block holds two tokens
    (1, 200, 33, 32),    # 264 threads along a row: two uneven column blocks
    (3, 67, 17, 64),     # 272: the same with a ragged row count
    (1, 40, 1, 1024),    # headdim at its limit: one thread per channel in the dD reduction
])
def test_gate_and_skip_follow_the_shape(b, l, h, p, d_dims, with_z):
    from ascend_kernel import mamba2 as M

    gen = torch.Generator(device="cuda").manual_seed(b + l + h + p)
    rnd = lambda *s: torch.randn(*s, generator=gen, device="cuda")  # noqa: E731
    y, x, dout = rnd(b, l, h, p), rnd(b, l, h, p), rnd(b, l, h, p)
    z = rnd(b, l, h, p) if with_z else None
    D = None if d_dims == 0 else rnd(h) if d_dims == 1 else rnd(h, p)
    B = torch.empty(b, l, 1, 64, device="cuda")
    if D is None and z is None:
        return
    leaves = {k: v.double().requires_grad_(True) for k, v in (("y", y), ("z", z), ("D", D)) if v is not None}
    pre = leaves["y"]
    if D is not None:
        pre = pre + x.double() * (leaves["D"].view(1, 1, h, 1) if d_dims == 1 else leaves["D"].view(1, 1, h, p))
    want = pre * torch.nn.functional.silu(leaves["z"]) if with_z else pre
    want.backward(dout.double())
    assert _rel(M.gate_forward(y, x, B, D, z), want.detach()) < REL
    dy, dz, dD = M.gate_backward(dout, y, x, B, D, z)
    assert _rel(dy, leaves["y"].grad) < REL
    if with_z:
        assert _rel(dz, leaves["z"].grad) < REL
    if D is not None:
        # a sum of terms of either sign: relative to the norm of the terms
        terms = (leaves["y"].grad * x.double()).norm().item()
        assert (dD.double() - leaves["D"].grad).norm().item() < REL * terms * (p ** 0.5 if d_dims == 1 else 1.0)


@pytest.mark.parametrize("b,l,h", [(1, 128, 1), (2, 256, 6), (1, 384, 33), (3, 128, 64)])
def test_dt_stages_take_any_number_of_heads(b, l, h):
    """dt cumsum and the finalize launch (transpose, dA, d(dt_bias)) with less than, exactly and more than a block of 32
    heads."""
    import ctypes

    from ascend_kernel import _capi

    gen = torch.Generator(device="cuda").manual_seed(7 * h + l)
    rnd = lambda *s: torch.randn(*s, generator=gen, device="cuda")  # noqa: E731
    dt, bias, A = rnd(b, l, h), rnd(h), -rnd(h).abs()
    s = ctypes.byref(_capi.SsdShape(b, l, h, 64, 64, 128, h, 1, 0.0, float("inf"), l - 5))
    st = torch.cuda.current_stream().cuda_stream
    q, cs, ddt_t = (torch.empty(b, h, l, device="cuda") for _ in range(3))
    _capi.check(_capi.lib.ssd_dt_cumsum(s, dt.data_ptr(), bias.data_ptr(), A.data_ptr(), q.data_ptr(), cs.data_ptr(), st), "cumsum")
    want = torch.nn.functional.softplus(dt.double() + bias.double())
    want[:, l - 5:] = 0
    assert _rel(q.transpose(1, 2), want) < REL
    run = (want * A.double()).view(b, l // 128, 128, h).cumsum(2).view(b, l, h)
    assert _rel(cs.transpose(1, 2), run) < REL
    ddt_t.copy_(rnd(b, h, l))
    part = torch.randn(b, h, l // 128, generator=gen, device="cuda", dtype=torch.float64)
    ddt, dA, dbias = torch.empty(b, l, h, device="cuda"), torch.empty(h, device="cuda"), torch.empty(h, device="cuda")
    _capi.check(_capi.lib.ssd_dt_finalize_bias_bwd(s, ddt_t.data_ptr(), part.data_ptr(), ddt.data_ptr(), dA.data_ptr(),
                                                  dbias.data_ptr(), st), "finalize")
    assert torch.equal(ddt, ddt_t.transpose(1, 2))
    assert (dA.double() - part.sum((0, 2))).abs().max() < 1e-6 * part.abs().sum()
    assert (dbias.double() - ddt_t.double().sum((0, 2))).abs().max() < 1e-6 * ddt_t.double().norm()


@pytest.mark.parametrize("offset", [0, 1])  # 1: rows that are not 8-byte aligned
@pytest.mark.parametrize("with_z,with_skip", [(False, False), (True, False), (False, True), (True, True)])
@pytest.mark.parametrize("rows,d", [(1, 1), (9, 64), (5, 192), (17, 194), (3, 384), (8, 385), (4, 512)])
def test_norm_with_gate_and_skip(rows, d, with_z, with_skip, offset):
    from ascend_kernel import _capi

    gen = torch.Generator(device="cuda").manual_seed(rows + d)
    rnd = lambda *s: torch.randn(*s, generator=gen, device="cuda")  # noqa: E731
    headdim = 32 if d % 32 == 0 else 1
    wide, x, skip, w = rnd(rows, d + 7), rnd(rows * d + 1)[offset:offset + rows * d].view(rows, d), rnd(rows, d), rnd(d)
    D = rnd(d // headdim)
    out = torch.empty(rows, d, device="cuda")
    _capi.check(_capi.lib.ssd_block_skip_rmsnorm_fwd(
        x.data_ptr(), d, skip.data_ptr() if with_skip else None, D.data_ptr() if with_skip else None, headdim,
        wide.data_ptr() if with_z else None, d + 7, w.data_ptr(), out.data_ptr(), rows, d, 1e-5,
        torch.cuda.current_stream().cuda_stream), "norm")
    t = x.double()
    if with_skip:
        t = t + skip.double() * D.double().repeat_interleave(headdim)
    if with_z:
        t = t * torch.nn.functional.silu(wide[:, :d].double())
    assert _rel(out, t * torch.rsqrt(t.pow(2).mean(-1, keepdim=True) + 1e-5) * w.double()) <= REL


@pytest.mark.parametrize("batch,l,d_in,gn,heads", [(1, 1, 4, 4, 0), (2, 15, 64, 32, 3), (1, 16, 130, 7, 130), (3, 67, 384, 64, 6)])
def test_convolution_and_split(batch, l, d_in, gn, heads):
    from ascend_kernel import _capi

    gen = torch.Generator(device="cuda").manual_seed(l + d_in)
    rnd = lambda *s: torch.randn(*s, generator=gen, device="cuda")  # noqa: E731
    ch = d_in + 2 * gn
    src, weight, bias, a_log = rnd(batch, l, ch + heads + 5), rnd(ch, 4), rnd(ch), rnd(max(heads, 1))
    x, bm, cm, dt = (torch.empty(batch, l, n, device="cuda") for n in (d_in, gn, gn, heads))
    A = torch.empty(heads, device="cuda")
    _capi.check(_capi.lib.ssd_block_conv_split_fwd(
        src.data_ptr(), ch + heads + 5, weight.data_ptr(), bias.data_ptr(), a_log.data_ptr(), x.data_ptr(), bm.data_ptr(),
        cm.data_ptr(), dt.data_ptr(), A.data_ptr(), batch, l, d_in, gn, heads,
        torch.cuda.current_stream().cuda_stream), "conv")
    padded = torch.nn.functional.pad(src[..., :ch].double(), (0, 0, 3, 0))
    want = bias.double() + sum(padded[:, k:k + l] * weight[:, k].double() for k in range(4))
    assert _rel(torch.cat([x, bm, cm], -1), torch.nn.functional.silu(want)) <= REL
    assert torch.equal(dt, src[..., ch:ch + heads]) and torch.allclose(A, -torch.exp(a_log[:heads]), rtol=1e-6)


def test_finalize_takes_a_buffer_of_any_alignment():
    """ddt_t is the caller's own buffer in the C interface and was never asked to be 16-byte aligned."""
    import ctypes

    from ascend_kernel import _capi

    b, l, h = 2, 256, 5
    s = ctypes.byref(_capi.SsdShape(b, l, h, 64, 64, 128, 1, 1, 0.0, float("inf"), 0))
    part = torch.randn(b, h, l // 128, device="cuda", dtype=torch.float64)
    raw = torch.randn(b * h * l + 1, device="cuda")
    results = []
    for ddt_t in (raw[1:].clone(), raw[1:]):
        ddt, dA, dbias = torch.empty(b, l, h, device="cuda"), torch.empty(h, device="cuda"), torch.empty(h, device="cuda")
        _capi.check(_capi.lib.ssd_dt_finalize_bias_bwd(s, ddt_t.data_ptr(), part.data_ptr(), ddt.data_ptr(), dA.data_ptr(),
                                                      dbias.data_ptr(), torch.cuda.current_stream().cuda_stream), "finalize")
        results.append((ddt, dA, dbias))
    assert all(torch.equal(a, c) for a, c in zip(*results))
    assert torch.equal(results[0][0], raw[1:].view(b, h, l).transpose(1, 2))


def test_gate_with_more_row_blocks_than_one_grid_dimension_holds():
    from ascend_kernel import mamba2 as M

    b, l, h, p = 1, 65536 * 128 + 5, 1, 4
    gen = torch.Generator(device="cuda").manual_seed(12)
    y, x, z, dout = (torch.randn(b, l, h, p, generator=gen, device="cuda") for _ in range(4))
    D = torch.randn(h, p, generator=gen, device="cuda")
    sig = torch.sigmoid(z.double())
    pre = y.double() + x.double() * D.double()
    assert _rel(M.gate_forward(y, x, None, D, z), pre * z.double() * sig) < REL
    dy, dz, dD = M.gate_backward(dout, y, x, None, D, z)
    want = dout.double() * z.double() * sig
    assert _rel(dy, want) < REL
    assert _rel(dz, dout.double() * pre * sig * (1 + z.double() * (1 - sig))) < REL
    terms = want * x.double()
    assert (dD.double() - terms.sum((0, 1))).norm().item() < REL * terms.norm().item()
