"""GPU tests of the device step's batched forward pass (all four fields' rows, then columns,
in two launches) and of the memory it takes: every line length once along x and once along
y, with partial CTAs, with and without surface planes, in G form (FP64, whole columns) and
not, against the oracle; both sides of its 512 MB line; and the same under index checks."""
import os
import subprocess
import sys

import numpy as np
import pytest

import overlappingbls_b200 as obl
from overlappingbls_b200 import build, fields
from conftest import ROOT, identical_inputs, rel_l2

pytestmark = pytest.mark.gpu

TOL = {"f64": 1e-12, "mixed": 1e-5}


class DevStep:
    """device buffers of one step; outputs start as NaN"""

    def __init__(self, ctx, f, prec, planes=None):
        import torch
        dt = torch.float64 if prec == "f64" else torch.float32
        self.ctx, self.planes = ctx, planes or {}
        nz, ny, ldx, nx2, ny2 = ctx.nz, ctx.nyt, ctx.ldx, ctx.nxt2, ctx.nyt2

        def up(a):
            return torch.from_numpy(np.ascontiguousarray(a.T)).to("cuda", dt)

        def nan(*sh):
            return torch.full(sh, float("nan"), device="cuda", dtype=dt)
        self.f = {k: up(f[k]) for k in ("u", "v", "w", "theta")}
        self.pl = {k: up(v) for k, v in self.planes.items()}
        self.d = [nan(nz + 1, ny, ldx) for _ in range(8)]
        self.big = [nan(nz + 1, ny2, nx2) for _ in range(4)]
        self.p, self.dp = nan(nz + 1, ny, ldx), [nan(nz, ny, ldx) for _ in range(3)]

    def run(self):
        import torch
        q = lambda t: t.data_ptr()   # noqa: E731
        torch.cuda.synchronize()
        self.ctx.step_dev(q(self.f["u"]), q(self.f["v"]), q(self.f["w"]), q(self.f["theta"]), [q(t) for t in self.d],
                          [q(t) for t in self.big], q(self.p), [q(t) for t in self.dp],
                          *(q(self.pl[k]) if k in self.pl else None for k in ("bot", "top")))
        self.ctx.synchronize()

    def check(self, ref, tol):
        ctx, h = self.ctx, lambda t: t.double().cpu().numpy().T   # noqa: E731
        nx, L = ctx.nxt, ctx.nz - 1
        for i in range(8):
            assert rel_l2(h(self.d[i])[:nx], ref["d"][i][:nx]) < tol, ("d", i)
        for i in range(4):
            assert rel_l2(h(self.big[i]), ref["big"][i]) < tol, ("big", i)
        assert rel_l2(h(self.p)[:nx, :, : L + 1], ref["p"][:nx, :, : L + 1]) < tol, "p"
        for t, k in zip(self.dp, ("dpdx", "dpdy", "dpdz")):
            assert rel_l2(h(t)[:nx, :, :L], ref[k][:nx, :, :L]) < tol, k
        for k in "uvw":
            assert rel_l2(h(self.f[k]), ref[k]) < tol, k


def _setup(orc, nx, ny, nzt, prec, top="neumann"):
    ctx = obl.Context(nx, ny, nzt, precision=prec, top_bc=top, **fields.DOMAIN)
    g = orc.Grid(nx, ny, nzt, **fields.DOMAIN)
    return ctx, g, identical_inputs(fields.make_fields(nx, ny, nzt), prec)


def _launches(ctx, call):
    """kernel launches of a call by name"""
    ctx.timing(True)
    ctx.timing_report()
    call()
    names = {k: v[0] for k, v in ctx.timing_report().items()}
    ctx.timing(False)
    return names


LENGTHS = (32, 48, 64, 80, 96, 128, 160, 192, 240, 256, 320, 384, 512, 640)


@pytest.mark.parametrize("prec", ["f64", "mixed"])
@pytest.mark.parametrize("i,nx", list(enumerate(LENGTHS)))
def test_batched_step_every_length(orc, i, nx, prec):
    ny = LENGTHS[(i + 5) % len(LENGTHS)]
    ctx, g, f = _setup(orc, nx, ny, 10, prec)      # 9 levels: whole columns
    planes = {}
    if i % 2:
        planes = {k: np.asfortranarray((1e-3 * f[v][:, :, 2]).astype(np.float32).astype(np.float64))
                  for k, v in (("bot", "v"), ("top", "w"))}
    s = DevStep(ctx, f, prec, planes)
    names = _launches(ctx, s.run)
    assert names["rows_fwd3"] == 1 and names["cols_fwd"] == 1 and "pad_cols" not in names, names
    assert ("press_gform_cols" in names) == (prec == "f64"), names
    ref = g.step(f["u"], f["v"], f["w"], f["theta"], npz=3)
    if planes:
        p, dx, dy = g.press_stag_array(f["u"], f["v"], f["w"], planes["bot"], planes["top"], npz=3)
        dz = g.dpdz(p)
        ref.update(p=p, dpdx=dx, dpdy=dy, dpdz=dz, **dict(zip("uvw", g.project(f["u"], f["v"], f["w"], dx, dy, dz))))
    s.check(ref, TOL[prec])
    ctx.close()


# 4 fields of 960 x 640 x nlev doubles: 530.8 MB at 27 stored levels, 550.5 MB at 28 (limit 536.9)
@pytest.mark.parametrize("nzt,batched", [(26, True), (27, False)])
def test_both_sides_of_the_memory_line(orc, nzt, batched):
    ctx, g, f = _setup(orc, 640, 640, nzt, "f64")
    s = DevStep(ctx, f, "f64")
    names = _launches(ctx, s.run)
    assert ("cols_fwd" in names) == batched and ("pad_cols" in names) != batched, names
    s.check(g.step(f["u"], f["v"], f["w"], f["theta"], npz=5 if nzt == 26 else 2), TOL["f64"])
    ctx.close()


def test_batched_step_under_index_checks():
    if os.environ.get("OBL_CHECKED_RUN") == "1":
        pytest.skip("already the child run")
    env = dict(os.environ, OBL_LIB=build.LIB_CHECK, OBL_CHECKED_RUN="1")
    r = subprocess.run([sys.executable, "-m", "pytest", "-q", "-x", "-p", "no:cacheprovider", __file__, "-k", "every_length"],
                       cwd=ROOT, env=env, capture_output=True, text=True, timeout=1200)
    tail = "\n".join(r.stdout.splitlines()[-25:])
    assert r.returncode == 0 and "28 passed" in tail, tail


def test_batch_holds_no_buffer_of_its_own(orc):
    """The x-padded rows wait in the padded outputs: a first device step allocates the five
    spectra and the solve's c', and no seventh buffer."""
    ctx, g, f = _setup(orc, 64, 48, 10, "f64")
    s = DevStep(ctx, f, "f64")
    ctx.set_param("fail_alloc", 7)     # spectra 5, c' 1
    s.run()
    assert ctx.get_param("fail_alloc") == 1
    s.check(g.step(f["u"], f["v"], f["w"], f["theta"], npz=3), TOL["f64"])
    ctx.close()


def test_captured_call_survives_a_first_step(orc):
    """The intermediate of a zero_padding captured in a CUDA graph stays where it was when
    the context then makes its first step."""
    import torch
    ctx, g, f = _setup(orc, 64, 48, 17, "f64")
    s = DevStep(ctx, f, "f64")
    var = s.f["v"].clone()
    big = torch.full_like(s.big[0], float("nan"))
    st = torch.cuda.Stream()
    ctx.set_stream(st.cuda_stream)
    call = lambda: ctx.zero_padding_dev(var.data_ptr(), big.data_ptr(), ctx.nz + 1)   # noqa: E731
    torch.cuda.synchronize()
    call()
    st.synchronize()
    want = big.clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=st):
        call()
    free0 = torch.cuda.mem_get_info(0)[0]
    s.run()
    held = torch.full((1 << 20,), -7.0, device="cuda", dtype=torch.float64)   # what may land in freed memory
    big.fill_(float("nan"))
    torch.cuda.synchronize()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(big, want) and free0 >= torch.cuda.mem_get_info(0)[0]
    assert bool((held == -7.0).all())
    ctx.close()
