"""GPU test of press_stag_array on real(8) host arrays of an FP32-storage context: its
results stay what they were to far below single-precision rounding.

golden/real8_press.npz holds samples of p, dpdx, dpdy computed by the three-radix kernels
(every supported line length once along x and once along y, both top modes, with and
without surface planes).  The bound is the one of the returned type, 1e-9 in relative L2:
FP32 transforms factored another way are 3e-7 off."""
import os

import numpy as np
import pytest

import overlappingbls_b200 as obl
from overlappingbls_b200 import fields
from conftest import identical_inputs, rel_l2

pytestmark = pytest.mark.gpu

GOLDEN = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "real8_press.npz")
LENGTHS = (32, 48, 64, 80, 96, 128, 160, 192, 240, 256, 320, 384, 512, 640)
# (nxt, nyt, nzt, precision, top, planes); 140 levels: the copy-fed form of the solve
CASES = [(n, LENGTHS[(i + 5) % len(LENGTHS)], 8, "mixed", ("neumann", "single")[i % 2], i % 3 == 0)
         for i, n in enumerate(LENGTHS)]
CASES += [(64, 48, 34, "mixed", "single", True), (64, 80, 35, "mixed", "neumann", True),
          (48, 64, 141, "mixed", "neumann", False), (96, 32, 18, "f32", "neumann", True)]


def _key(c):
    return "%dx%dx%d_%s_%s_%d" % c


def samples(c):
    """about 250 values of each output of case c"""
    nx, ny, nzt, prec, top, planes = c
    f = identical_inputs(fields.make_fields(nx, ny, nzt), "mixed")
    ctx = obl.Context(nx, ny, nzt, precision=prec, top_bc=top, **fields.DOMAIN)
    bot, up = (np.asfortranarray(1e-3 * f[k][:, :, 2]) for k in ("v", "w"))
    bot, up = (np.asfortranarray(a.astype(np.float32).astype(np.float64)) for a in (bot, up))
    p, dx, dy = ctx.field(), ctx.dfield(), ctx.dfield()
    ctx.press_stag_array(p, dx, dy, f["u"], f["v"], f["w"], bot if planes else None, up if planes else None)
    L = ctx.nz - 1
    out = []
    for a in (p[:nx, :, : L + 1], dx[:nx, :, :L], dy[:nx, :, :L]):
        a = a.ravel(order="F")
        out.append(a[:: max(1, a.size // 250) | 1])
    ctx.close()
    return out


@pytest.mark.parametrize("case", CASES, ids=_key)
def test_results_keep_their_rounding(case):
    gold = np.load(GOLDEN)
    for name, a in zip(("p", "dpdx", "dpdy"), samples(case)):
        b = gold[_key(case) + "_" + name].astype(np.float64)
        assert a.shape == b.shape
        assert rel_l2(a, b) < 1e-9, name


if __name__ == "__main__":   # writes the samples of the library that is loaded
    import sys
    np.savez_compressed(sys.argv[1] if len(sys.argv) > 1 else GOLDEN,
                        **{_key(c) + "_" + n: a.astype(np.float32) for c in CASES
                           for n, a in zip(("p", "dpdx", "dpdy"), samples(c))})
