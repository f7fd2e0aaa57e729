"""GPU test of the pressure solve where two spectral planes lie more than 2^31 bytes apart
(640x640 points, 653 solve levels in FP64; about 40 GB on the device)."""
import pytest

import overlappingbls_b200 as obl
from overlappingbls_b200 import fields

pytestmark = pytest.mark.gpu


def test_absent_planes_of_a_tall_domain():
    """Absent surface planes are zero planes: both calls give the same numbers."""
    import torch
    nx = ny = 640
    nzt = 654
    if torch.cuda.mem_get_info(0)[0] < 60 << 30:
        pytest.skip("needs 60 GB of free device memory")
    ctx = obl.Context(nx, ny, nzt, precision="f64", **fields.DOMAIN)
    assert 16 * ctx.lhx * ny * (ctx.nz - 1 + 1) > 2 ** 31 - 1
    g = torch.Generator(device="cuda")
    g.manual_seed(3)
    plane = torch.randn((ny, ctx.ldx), generator=g, device="cuda", dtype=torch.float64)
    u, v, w = (torch.empty((ctx.nz + 1, ny, ctx.ldx), device="cuda", dtype=torch.float64) for _ in range(3))
    for z in range(ctx.nz + 1):     # a plane rolled along x and y: every level another one
        for k, t in enumerate((u, v, w)):
            t[z] = torch.roll(plane, (7 * z + k, 3 * z + 11 * k), (0, 1))
    zero = torch.zeros_like(plane)
    outs = []
    for pl in (None, zero.data_ptr()):
        p = torch.full_like(u, float("nan"))
        d = [torch.full((ctx.nz, ny, ctx.ldx), float("nan"), device="cuda", dtype=torch.float64) for _ in range(2)]
        torch.cuda.synchronize()
        ctx.press_stag_array_dev(p.data_ptr(), d[0].data_ptr(), d[1].data_ptr(), u.data_ptr(), v.data_ptr(),
                                 w.data_ptr(), pl, pl)
        ctx.synchronize()
        L = ctx.nz - 1
        outs.append([p[: L + 1, :, :nx], d[0][:L, :, :nx], d[1][:L, :, :nx]])
    for a, b in zip(*outs):
        assert bool(torch.isfinite(a).all()) and torch.equal(a, b)
    ctx.close()
    del outs, u, v, w
    torch.cuda.empty_cache()
