"""GPU tests of the two-pass line kernels and the launches built on them, against the FP64
oracle: every supported line length in both directions with a level count that leaves
partial CTAs, the level differences around their eight-level chunks, and the pressure solve
on both sides of its column rule.  Tolerances are the repository's: 1e-12 (FP64) and 1e-5
(mixed) relative L2 per field."""
import numpy as np
import pytest

import overlappingbls_b200 as obl
from overlappingbls_b200 import fields
from conftest import identical_inputs, rel_l2

pytestmark = pytest.mark.gpu

TOL = {"f64": 1e-12, "mixed": 1e-5}
LENGTHS = (32, 48, 64, 80, 96, 128, 160, 192, 240, 256, 320, 384, 512, 640)
# each length once along x and once along y
PAIRS = [(n, LENGTHS[(i + 5) % len(LENGTHS)]) for i, n in enumerate(LENGTHS)]


def _pair(orc, nx, ny, nzt, prec, top="neumann"):
    ctx = obl.Context(nx, ny, nzt, precision=prec, top_bc=top, **fields.DOMAIN)
    g = orc.Grid(nx, ny, nzt, **fields.DOMAIN)
    return ctx, g, identical_inputs(fields.make_fields(nx, ny, nzt), prec)


@pytest.mark.parametrize("prec", ["f64", "mixed"])
@pytest.mark.parametrize("nx,ny", PAIRS)
def test_line_operations_every_length(orc, nx, ny, prec):
    ctx, g, f = _pair(orc, nx, ny, 6, prec)
    tol = TOL[prec]
    for name in ("ddx", "ddy"):
        out = ctx.field()
        getattr(ctx, name)(out, f["v"])
        assert rel_l2(out[:nx], getattr(g, name)(f["v"])[:nx]) < tol, name
    big, spec, back, filt = ctx.big_field(), ctx.spectral(), ctx.field(), f["u"].copy(order="F")
    ctx.zero_padding(f["v"], big)
    ctx.fftn(f["v"], spec)
    ctx.ifftn(spec, back)
    ctx.filter_data(filt)
    rng = np.random.default_rng(nx + ny)
    big2 = identical_inputs({"b": np.asfortranarray(rng.standard_normal(big.shape))}, prec)["b"]
    unp = ctx.field()
    ctx.zero_unpadding(big2, unp)
    ref_filt = f["u"].copy(order="F")
    ref = g.filter_data(ref_filt)
    ref_filt = ref_filt if ref is None else ref
    assert rel_l2(filt[:nx], ref_filt[:nx]) < tol
    for z in (0, 3, g.nz):
        s = g.fftn(f["v"][:, :, z])
        assert rel_l2(big[:, :, z], g.zero_padding(f["v"][:, :, z])) < tol
        assert rel_l2(spec[:, :, z], s) < tol
        assert rel_l2(back[:nx, :, z], g.ifftn(s)[:nx]) < tol
        assert rel_l2(unp[:, :, z], g.zero_unpadding(big2[:, :, z])) < tol
    for name in ("divstress_uv", "divstress_w"):
        out = ctx.field()
        getattr(ctx, name)(out, f["u"], f["v"], f["w"])
        want = getattr(g, name)(f["u"], f["v"], f["w"])
        n = g.nz if name == "divstress_uv" else g.nz + 1
        assert rel_l2(out[:, :, 1:n], want[:, :, 1:n]) < tol, name
        assert np.array_equal(out[:, :, 0], want[:, :, 0].astype(ctx.dtype).astype(np.float64)), name
    ctx.close()


@pytest.mark.parametrize("prec", ["f64", "mixed"])
@pytest.mark.parametrize("nzt", [6, 7, 14, 15, 16])
def test_level_differences_around_chunks(orc, nzt, prec):
    ctx, g, f = _pair(orc, 32, 48, nzt, prec)
    nx = g.nxt
    for name in ("ddz_uv", "ddz_w"):
        out, ref = ctx.field(), g.field()
        out[:], ref[:] = 7.0, 7.0
        getattr(ctx, name)(out, f["u"])
        want = getattr(g, name)(f["u"], ref)
        want = ref if want is None else want
        for z in range(g.nz + 1):
            assert rel_l2(out[:nx, :, z], want[:nx, :, z]) < TOL[prec], (name, z)
    d = ctx.dfield()
    ctx.dpdz(d, f["u"])
    assert rel_l2(d[:nx, :, : g.nz - 1], g.dpdz(f["u"])[:nx, :, : g.nz - 1]) < TOL[prec]
    ctx.close()


# (kx, ky) columns: 15488 and 16512 (FP32 whole columns from 16384 on), 2112
@pytest.mark.parametrize("prec", ["f64", "mixed"])
@pytest.mark.parametrize("nx,ny,nzt", [(240, 128, 34), (256, 128, 34), (64, 64, 19)])
def test_press_stag_array_column_rule(orc, nx, ny, nzt, prec):
    ctx, g, f = _pair(orc, nx, ny, nzt, prec)
    p, dx, dy = ctx.field(), ctx.dfield(), ctx.dfield()
    ctx.press_stag_array(p, dx, dy, f["u"], f["v"], f["w"])
    rp, rx, ry = g.press_stag_array(f["u"], f["v"], f["w"], npz=3)
    L = g.nz - 1
    assert rel_l2(p[:nx, :, : L + 1], rp[:nx, :, : L + 1]) < TOL[prec]
    assert rel_l2(dx[:nx, :, :L], rx[:nx, :, :L]) < TOL[prec]
    assert rel_l2(dy[:nx, :, :L], ry[:nx, :, :L]) < TOL[prec]
    ctx.close()
