"""GPU test of the step's choice between segmented and whole columns in the pressure solve:
both sides of each line of the rule, level counts that the segments do not divide among
them, against the oracle."""
import pytest

from test_gpu_forward_batch import TOL, DevStep, _launches, _setup

pytestmark = pytest.mark.gpu


# columns (nx/2+1)*ny: 192x160 15520, 192x192 18624, 320x240 38640, 256x384 49536
@pytest.mark.parametrize("prec,nx,ny,levels,segmented", [
    ("mixed", 192, 160, 112, True), ("mixed", 192, 192, 16, True), ("mixed", 192, 192, 51, True),
    ("mixed", 192, 192, 104, True), ("mixed", 192, 192, 106, False), ("mixed", 320, 240, 72, True),
    ("mixed", 320, 240, 74, False), ("mixed", 256, 384, 48, True), ("mixed", 256, 384, 51, False),
    ("f64", 320, 240, 51, True), ("f64", 256, 384, 48, True), ("f64", 256, 384, 50, False)])
def test_both_sides_of_the_rule(orc, prec, nx, ny, levels, segmented):
    ctx, g, f = _setup(orc, nx, ny, levels + 1, prec)
    s = DevStep(ctx, f, prec)
    names = _launches(ctx, s.run)
    assert ("tdma_seg_solve" in names) == segmented, names
    assert segmented or {"tdma", "tdma_reg", "tdma_staged"} & set(names), names
    s.check(g.step(f["u"], f["v"], f["w"], f["theta"], npz=2 if levels % 2 == 0 else 3), TOL[prec])
    ctx.close()
