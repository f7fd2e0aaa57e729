"""GPU test of the vertical differences on planes large enough for eight levels a thread
(test_gpu_twopass.py's small planes take one), at level counts around the chunks of eight."""
import pytest

import overlappingbls_b200 as obl
from overlappingbls_b200 import fields
from conftest import identical_inputs, rel_l2

pytestmark = pytest.mark.gpu

TOL = {"f64": 1e-12, "mixed": 1e-5}


# 193 CTAs a chunk: nzt = 6 is one chunk and stays with one level a thread
@pytest.mark.parametrize("prec", ["f64", "mixed"])
@pytest.mark.parametrize("nzt", [6, 14, 15, 16, 17])
def test_eight_levels_a_thread(orc, nzt, prec):
    ctx = obl.Context(384, 256, nzt, precision=prec, **fields.DOMAIN)
    g = orc.Grid(384, 256, nzt, **fields.DOMAIN)
    f = identical_inputs(fields.make_fields(384, 256, nzt), prec)
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
