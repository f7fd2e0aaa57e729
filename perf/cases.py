"""Performance cases of the library: the calls its users make, over the sizes they make them with.

A case is a dict of plain values.  Its "kind" is the call:

  step      obl_step_dev: the fused projection-plus-derivative step of a time loop
  slice     press_stag_array + dpdz + project: the three calls of the unmodified time loop
  derivs    ddx, ddy, ddz and the stress divergence of one right-hand side
  dealias   zero_padding of two factors and zero_unpadding of a product
  filter    fftn, ifftn and filter_data of one field
  rollout   rollout_grad_dev: forward rollout, checkpoints and the reverse sweep
  ensemble  many uneven instances, one captured graph on concurrent streams
  host      press_stag_array on real(8) host arrays, as a Fortran caller passes them

Grid sizes are the line lengths the library has plans for, with any number of levels.
Fields follow the recipe of overlappingbls_b200.fields (log-law mean, k^-5/3 random-phase
fluctuations of 0.5 m/s, stratified theta with 0.1 K noise), drawn on the GPU from the seed.
`exact` restates every call in float64 torch (torch.fft, a Thomas sweep over the levels,
autograd for the gradient).
"""
import math

import numpy as np
import torch

import overlappingbls_b200 as obl
from overlappingbls_b200 import fields

LENGTHS = (32, 48, 64, 80, 96, 128, 160, 192, 240, 256, 320, 384, 512, 640)
TADV1 = 1.5
BOGUS = -1234567890.0
KE_BAND = (0.0, 100.0)


def listed():
    return [
        # the smallest whole step, a single small domain in FP64: launches and latency
        dict(name="step_64x64x64_f64", kind="step", nx=64, ny=64, levels=64, prec="f64", top="neumann", divtz=False),
        # a middle-sized production domain in mixed precision
        dict(name="step_256x256x128_mixed", kind="step", nx=256, ny=256, levels=128, prec="mixed", top="neumann",
             divtz=False),
        # the headline workload, mixed precision and the plain FP64 form
        dict(name="step_512x512x256_mixed", kind="step", nx=512, ny=512, levels=256, prec="mixed", top="neumann",
             divtz=False),
        dict(name="step_512x512x256_f64", kind="step", nx=512, ny=512, levels=256, prec="f64", top="neumann",
             divtz=False),
        # factor-5 lengths, an odd number of levels, the npz = 1 top row and surface planes
        dict(name="step_320x240x65_mixed_top1", kind="step", nx=320, ny=240, levels=65, prec="mixed", top="single",
             divtz=True),
        # the reference's own time loop: separate calls, FP64 as its real(8) fields
        dict(name="slice_192x192x128_f64", kind="slice", nx=192, ny=192, levels=128, prec="f64", top="neumann",
             divtz=True),
        # the derivatives and stress divergence of a right-hand side between projections
        dict(name="derivs_384x384x128_mixed", kind="derivs", nx=384, ny=384, levels=128, prec="mixed", top="neumann",
             divtz=False),
        # dealiased product of a scalar transport term
        dict(name="dealias_256x192x96_f64", kind="dealias", nx=256, ny=192, levels=96, prec="f64", top="neumann",
             divtz=False),
        # test filtering in the dynamic SGS model
        dict(name="filter_160x128x64_mixed", kind="filter", nx=160, ny=128, levels=64, prec="mixed", top="neumann",
             divtz=False),
        # gradient of the near-wall kinetic energy through 16 steps
        dict(name="rollout_128x128x128_16_mixed", kind="rollout", nx=128, ny=128, levels=128, prec="mixed",
             top="neumann", divtz=False, nsteps=16),
        # 48 uneven instances advanced together
        dict(name="ensemble_48_mixed", kind="ensemble", members="96x96x64*16,128x128x96*16,192x192x128*16",
             prec="mixed", top="neumann", divtz=False),
        # the drop-in on host arrays: copies over PCIe and the solve
        dict(name="host_press_128x128x64_f64", kind="host", nx=128, ny=128, levels=64, prec="f64", top="neumann",
             divtz=True),
    ]


def draw(rng):
    kind = rng.choice(("step", "step", "step", "slice", "derivs", "dealias", "filter", "rollout", "ensemble", "host"))
    prec = rng.choice(("mixed", "mixed", "f64"))
    if kind == "ensemble":
        parts = []
        for _ in range(rng.randint(2, 4)):
            n = rng.choice((64, 80, 96, 128, 160, 192))
            parts.append("%dx%dx%d*%d" % (n, rng.choice((n, 96, 128)), int(round(math.exp(rng.uniform(math.log(16), math.log(128))))),
                                          rng.randint(2, 10)))
        return dict(kind=kind, members=",".join(parts), prec=prec, top="neumann", divtz=False)
    # points: log-uniform between a small domain and the kind's largest
    most = {"rollout": 128 ** 3, "host": 128 * 128 * 64}.get(kind, 512 * 512 * 256)
    points = math.exp(rng.uniform(math.log(32 * 32 * 16), math.log(most)))
    while True:
        nx = rng.choice(LENGTHS)
        ny = rng.choice(LENGTHS)
        levels = int(round(points / (nx * ny)))
        if max(nx, ny) <= 4 * min(nx, ny) and 8 <= levels <= 256:
            break
    c = dict(kind=kind, nx=nx, ny=ny, levels=levels, prec=prec, top="neumann", divtz=False)
    if kind in ("step", "slice", "host"):
        c["top"] = rng.choice(("neumann", "neumann", "single"))
        c["divtz"] = rng.random() < 0.5
    if kind == "rollout":
        c["nsteps"] = rng.randint(2, 16)
    return c


# ----------------------------------------------------------------------------- inputs
def _dtype(case):
    return torch.float64 if case["prec"] == "f64" else torch.float32


def _gen(seed, salt=0):
    g = torch.Generator(device="cuda")
    g.manual_seed((int(seed) * 1000003 + salt) & 0x7FFFFFFFFFFFFFFF)
    return g


def _fluct(g, nx, ny, nlev, rms=0.5):
    """k^-5/3 random-phase fluctuations of the given rms on every level, (nlev, ny, nx) float64."""
    lhx = nx // 2 + 1
    ky = torch.fft.fftfreq(ny, 1.0 / ny, device="cuda", dtype=torch.float64)[:, None]
    kx = torch.arange(lhx, device="cuda", dtype=torch.float64)[None, :]
    k = torch.sqrt(kx * kx + ky * ky)
    amp = torch.where(k > 0, k.clamp(min=1e-30) ** (-4.0 / 3.0), torch.zeros_like(k))
    amp[:, lhx - 1] = 0.0
    amp[ny // 2, :] = 0.0
    ph = 2.0 * math.pi * torch.rand((nlev, ny, lhx), generator=g, device="cuda", dtype=torch.float64)
    f = torch.fft.irfft2(torch.polar(amp.expand_as(ph).contiguous(), ph), s=(ny, nx))
    return f.mul_(rms / f.square().mean(dim=(1, 2), keepdim=True).sqrt())


def _field(f, nx, dtype):
    """(nlev, ny, nx) -> the library's layout (nlev, ny, nx + 2), zero pads."""
    out = torch.zeros((f.shape[0], f.shape[1], nx + 2), device="cuda", dtype=dtype)
    out[:, :, :nx] = f
    return out


def _heights(levels):
    return (torch.arange(levels + 2, device="cuda", dtype=torch.float64) - 0.5) * (fields.DOMAIN["lz_tot"] / levels)


def _velocity(seed, nx, ny, levels, dtype, z0=0.1, salt=0):
    """u, v, w on levels 0..nz as one tensor (3, nz+1, ny, ldx)."""
    out = torch.zeros((3, levels + 2, ny, nx + 2), device="cuda", dtype=dtype)
    g = _gen(seed, salt)
    for c in range(3):
        f = _fluct(g, nx, ny, levels)
        if c == 0:
            f += ((0.45 / 0.4) * torch.log(_heights(levels)[1:-1] / z0))[:, None, None]
        out[c, 1:-1, :, :nx] = f
        if c < 2:
            out[c, 0] = out[c, 1]
            out[c, -1] = out[c, -2]
        else:
            out[c, 1] = 0.0
    return out


def _theta(seed, nx, ny, levels, dtype, grad=0.01, salt=0):
    g = _gen(seed, 7919 + salt)
    f = 300.0 + grad * _heights(levels)[1:-1, None, None] + \
        0.1 * torch.randn((levels, ny, nx), generator=g, device="cuda", dtype=torch.float64)
    out = _field(torch.cat((f[:1], f, f[-1:])), nx, dtype)
    return out


def _planes(case, seed, dtype):
    if not case["divtz"]:
        return None, None
    f = _fluct(_gen(seed, 104729), case["nx"], case["ny"], 2, rms=1e-3)
    p = _field(f, case["nx"], dtype)
    return p[0].contiguous(), p[1].contiguous()


def _ptr(t):
    return None if t is None else t.data_ptr()


def _ctx(case):
    return obl.Context(case["nx"], case["ny"], case["levels"] + 1, precision=case["prec"], top_bc=case["top"],
                       **fields.DOMAIN)


def _members(case):
    out = []
    for part in case["members"].split(","):
        size, n = part.split("*")
        nx, ny, levels = (int(v) for v in size.split("x"))
        out += [(nx, ny, levels)] * int(n)
    return out


def _member_inputs(case, seed, k, size):
    """One instance's roughness and stratification, from its own stream."""
    g = torch.Generator()
    g.manual_seed((int(seed) * 1000003 + 31 * k + 17) & 0x7FFFFFFFFFFFFFFF)
    r = torch.rand(2, generator=g, dtype=torch.float64)
    nx, ny, levels = size
    uvw = _velocity(seed, nx, ny, levels, _dtype(case), z0=float(10.0 ** (-2.0 + 2.0 * r[1])), salt=k + 1)
    return uvw, _theta(seed, nx, ny, levels, _dtype(case), grad=float(0.03 * r[0]), salt=k + 1)


def _step_shapes(nx, ny, levels):
    nz, ldx = levels + 1, nx + 2
    sh = {"d%d" % i: (nz + 1, ny, ldx) for i in range(8)}
    sh.update({"big%d" % i: (nz + 1, 3 * ny // 2, 3 * nx // 2) for i in range(4)})
    sh["p"] = (nz + 1, ny, ldx)
    sh.update({"dp%d" % i: (nz, ny, ldx) for i in range(3)})
    return sh


# ----------------------------------------------------------------------------- prepare / run
def prepare(case, seed):
    kind, dt = case["kind"], _dtype(case)
    if kind == "ensemble":
        return _prepare_ensemble(case, seed)
    nx, ny, levels = case["nx"], case["ny"], case["levels"]
    nz, ldx = levels + 1, nx + 2
    s = {"kind": kind, "ctx": _ctx(case), "nx": nx}
    zeros = lambda *sh: torch.zeros(sh, device="cuda", dtype=dt)   # noqa: E731
    uvw = _velocity(seed, nx, ny, levels, dt)
    bot, top = _planes(case, seed, dt)
    if kind in ("step", "slice"):
        # the predicted velocity of the time loop, and the fields it is projected in
        s.update(pred=uvw, uvw=torch.empty_like(uvw), bot=bot, top=top)
        if kind == "step":
            s["theta"] = _theta(seed, nx, ny, levels, dt)
            s["out"] = {k: zeros(*sh) for k, sh in _step_shapes(nx, ny, levels).items()}
        else:
            s["out"] = dict(p=zeros(nz + 1, ny, ldx), dpdx=zeros(nz, ny, ldx), dpdy=zeros(nz, ny, ldx),
                            dpdz=zeros(nz, ny, ldx))
    elif kind == "derivs":
        s["uvw"] = uvw
        s["tau"] = 0.1 * _velocity(seed + 1000, nx, ny, levels, dt)
        s["out"] = {k: zeros(nz + 1, ny, ldx) for k in ("dudx", "dudy", "dudz", "dwdz", "divuv", "divw")}
    elif kind == "dealias":
        s["uvw"] = uvw
        g = _gen(seed, 5)
        s["prod"] = _fluct(g, 3 * nx // 2, 3 * ny // 2, nz + 1).to(dt)
        s["out"] = dict(ub=zeros(nz + 1, 3 * ny // 2, 3 * nx // 2), wb=zeros(nz + 1, 3 * ny // 2, 3 * nx // 2),
                        back=zeros(nz + 1, ny, ldx))
    elif kind == "filter":
        s["uvw"] = uvw
        s["filt"] = uvw[0].clone()
        s["out"] = dict(spec=zeros(nz + 1, ny, ldx), back=zeros(nz + 1, ny, ldx))
    elif kind == "rollout":
        s.update(uvw=uvw, nsteps=case["nsteps"], grad=zeros(3, nz + 1, ny, ldx))
    elif kind == "host":
        F = lambda t: np.asfortranarray(t.double().cpu().numpy().T)   # noqa: E731
        s["uvw"] = [F(uvw[c]) for c in range(3)]
        s["planes"] = [None if t is None else F(t) for t in (bot, top)]
        s["out"] = [s["ctx"].field(), s["ctx"].dfield(), s["ctx"].dfield()]
    return s


def _prepare_ensemble(case, seed):
    dt, sizes = _dtype(case), _members(case)
    grids = [dict(nxt=nx, nyt=ny, nzt=levels + 1, **fields.DOMAIN) for nx, ny, levels in sizes]
    ens = obl.Ensemble(grids, precision=case["prec"], top_bc=case["top"])
    ens.set_mode("concurrent")
    # each kind of field of all instances in one allocation, the instances one after another
    align = 64
    flat, off = {}, []
    shapes = []
    for nx, ny, levels in sizes:
        sh = dict(uvw=(3, levels + 2, ny, nx + 2), theta=(levels + 2, ny, nx + 2), **_step_shapes(nx, ny, levels))
        shapes.append(sh)
    for key in shapes[0]:
        o, n = [], 0
        for sh in shapes:
            o.append(n)
            n += -(-math.prod(sh[key]) // align) * align
        off.append(o)
        flat[key] = torch.zeros(n, device="cuda", dtype=dt)
    pred = torch.zeros_like(flat["uvw"])
    ios = []
    for k, size in enumerate(sizes):
        view = {key: flat[key][o[k]:o[k] + math.prod(shapes[k][key])].view(shapes[k][key])
                for key, o in zip(shapes[0], off)}
        uvw, theta = _member_inputs(case, seed, k, size)
        pred[off[0][k]:off[0][k] + uvw.numel()] = uvw.reshape(-1)
        view["theta"].copy_(theta)
        ios.append(obl.stepio_dev(*(view["uvw"][c].data_ptr() for c in range(3)), theta=view["theta"].data_ptr(),
                                  d=[view["d%d" % i].data_ptr() for i in range(8)],
                                  big=[view["big%d" % i].data_ptr() for i in range(4)], p=view["p"].data_ptr(),
                                  dp=[view["dp%d" % i].data_ptr() for i in range(3)]))
    flat["uvw"].copy_(pred)
    torch.cuda.synchronize()
    ens.capture_dev(ios)
    return {"kind": "ensemble", "ens": ens, "pred": pred, "flat": flat}


def run(s):
    kind = s["kind"]
    if kind == "ensemble":
        # the ensemble's streams are its own: the predictor is complete before the graph is
        # launched, and the step before the buffers are used again
        s["flat"]["uvw"].copy_(s["pred"])
        torch.cuda.current_stream().synchronize()
        s["ens"].replay()
        s["ens"].synchronize()
        return {k: v for k, v in s["flat"].items() if k != "theta"}
    ctx, nx = s["ctx"], s["nx"]
    if kind == "step":
        o = s["out"]
        s["uvw"].copy_(s["pred"])
        ctx.step_dev(*(s["uvw"][c].data_ptr() for c in range(3)), theta=s["theta"].data_ptr(),
                     d=[o["d%d" % i].data_ptr() for i in range(8)],
                     big=[o["big%d" % i].data_ptr() for i in range(4)], p=o["p"].data_ptr(),
                     dp=[o["dp%d" % i].data_ptr() for i in range(3)], divtz_bot=_ptr(s["bot"]), divtz_top=_ptr(s["top"]))
        return dict(o, uvw=s["uvw"])
    if kind == "slice":
        o = s["out"]
        s["uvw"].copy_(s["pred"])
        u, v, w = (s["uvw"][c].data_ptr() for c in range(3))
        p, dx, dy, dz = (o[k].data_ptr() for k in ("p", "dpdx", "dpdy", "dpdz"))
        ctx.press_stag_array_dev(p, dx, dy, u, v, w, _ptr(s["bot"]), _ptr(s["top"]))
        ctx.dpdz_dev(dz, p)
        ctx.project_dev(u, v, w, dx, dy, dz)
        return dict(o, uvw=s["uvw"])
    if kind == "derivs":
        o, nlev = s["out"], s["uvw"].shape[1]
        u, w = s["uvw"][0].data_ptr(), s["uvw"][2].data_ptr()
        tau = [s["tau"][c].data_ptr() for c in range(3)]
        ctx.ddx_dev(o["dudx"].data_ptr(), u, nlev)
        ctx.ddy_dev(o["dudy"].data_ptr(), u, nlev)
        ctx.ddz_uv_dev(o["dudz"].data_ptr(), u)
        ctx.ddz_w_dev(o["dwdz"].data_ptr(), w)
        ctx.divstress_uv_dev(o["divuv"].data_ptr(), *tau)
        ctx.divstress_w_dev(o["divw"].data_ptr(), *tau)
        # the marker levels (BOGUS) hide the values in a whole field's norm: the computed
        # levels are returned by themselves too
        return dict(o, dudz_in=o["dudz"][1:], dwdz_in=o["dwdz"][1:], divuv_in=o["divuv"][1:-1], divw_in=o["divw"][1:])
    if kind == "dealias":
        o, nlev = s["out"], s["uvw"].shape[1]
        ctx.zero_padding_dev(s["uvw"][0].data_ptr(), o["ub"].data_ptr(), nlev)
        ctx.zero_padding_dev(s["uvw"][2].data_ptr(), o["wb"].data_ptr(), nlev)
        ctx.zero_unpadding_dev(s["prod"].data_ptr(), o["back"].data_ptr(), nlev)
        return o
    if kind == "filter":
        o, nlev = s["out"], s["uvw"].shape[1]
        ctx.fftn_dev(s["uvw"][1].data_ptr(), o["spec"].data_ptr(), nlev)
        ctx.ifftn_dev(o["spec"].data_ptr(), o["back"].data_ptr(), nlev)
        ctx.filter_data_dev(s["filt"].data_ptr(), nlev)
        return dict(o, filt=s["filt"])
    if kind == "rollout":
        u, g = s["uvw"], s["grad"]
        J = ctx.rollout_grad_dev(s["nsteps"], u[0].data_ptr(), u[1].data_ptr(), u[2].data_ptr(), *KE_BAND,
                                 g[0].data_ptr(), g[1].data_ptr(), g[2].data_ptr())
        # the pad columns of a gradient hold nothing (include/obl.h); J in the storage type
        return {"J": torch.tensor(J, dtype=g.dtype), "grad": g[..., :nx]}
    if kind == "host":
        ctx.press_stag_array(*s["out"], *s["uvw"], *s["planes"])
        return [a.T for a in s["out"]]
    raise ValueError(kind)


# ----------------------------------------------------------------------------- work
def _line(n):
    return 2.5 * n * math.log2(n)   # a real transform of length n


def _pad_flops(nx, ny):
    return ny * (_line(nx) + _line(1.5 * nx)) + 1.5 * nx * (_line(ny) + _line(1.5 * ny))


def _press_flops(nx, ny):
    """Per level: three forward transforms, the solve, four inverses."""
    return 7 * (ny * _line(nx) + nx * _line(ny)) + 40 * (nx / 2 + 1) * ny


def _step_work(nx, ny, levels, eb):
    f = 4 * (2 * ny * _line(nx) + 2 * nx * _line(ny) + _pad_flops(nx, ny)) + _press_flops(nx, ny)
    # in: u, v, w, theta; out: 8 derivatives, 4 padded fields, p, 3 gradients, u, v, w
    return 28.0 * nx * ny * levels * eb, f * levels


def work(case):
    eb = 8 if case["prec"] == "f64" else 4
    if case["kind"] == "ensemble":
        w = [_step_work(*m, eb) for m in _members(case)]
        return {"bytes": sum(b for b, _ in w), "flops": sum(f for _, f in w)}
    nx, ny, levels = case["nx"], case["ny"], case["levels"]
    n = float(nx * ny * levels) * eb
    kind = case["kind"]
    if kind == "step":
        b, f = _step_work(nx, ny, levels, eb)
    elif kind in ("slice", "host"):
        b, f = (10 if kind == "slice" else 6) * n, _press_flops(nx, ny) * levels
    elif kind == "derivs":      # u, w, tau in; six fields out
        b, f = 11 * n, 3 * 2 * (ny * _line(nx) + nx * _line(ny)) * levels
    elif kind == "dealias":
        b, f = 3 * 3.25 * n, 3 * _pad_flops(nx, ny) * levels
    elif kind == "filter":      # a field in, its spectrum and two fields out, the filtered field in
        b, f = 5 * n, 4 * (ny * _line(nx) + nx * _line(ny)) * levels
    else:                       # rollout: forward and reverse sweep of every step
        step = 4 * (ny * _line(nx) + nx * _line(ny)) + 9 * _pad_flops(nx, ny) + _press_flops(nx, ny)
        vjp = 8 * (ny * _line(nx) + nx * _line(ny)) + 15 * _pad_flops(nx, ny) + _press_flops(nx, ny)
        b, f = 6 * n, case["nsteps"] * (step + vjp) * levels
    return {"bytes": b, "flops": f}


# ----------------------------------------------------------------------------- exact (float64 torch)
class _Grid:
    def __init__(self, nx, ny, levels, top):
        d = fields.DOMAIN
        self.nx, self.ny, self.L, self.nz, self.top = nx, ny, levels, levels + 1, top
        self.lhx = nx // 2 + 1
        lx, ly = d["lx_tot"] / d["z_i"], d["ly_tot"] / d["z_i"]
        self.dz = d["lz_tot"] / levels / d["z_i"]
        self.dt = d["dt"] * d["u_scale"] / d["z_i"]
        self.z_i = d["z_i"]
        k = lambda n, l: torch.arange(n // 2 + 1, device="cuda", dtype=torch.float64) * (2.0 * math.pi / l)   # noqa: E731
        self.kx, self.ky1 = k(nx, lx), k(ny, ly)
        self.kx[-1] = 0.0
        self.ky1[-1] = 0.0
        self.ky = torch.fft.fftfreq(ny, 1.0 / ny, device="cuda", dtype=torch.float64) * (2.0 * math.pi / ly)
        self.ky[ny // 2] = 0.0


def _ddx(G, f):
    return torch.fft.irfft(torch.fft.rfft(f, dim=-1) * (1j * G.kx), n=G.nx, dim=-1)


def _ddy(G, f):
    return torch.fft.irfft(torch.fft.rfft(f, dim=-2) * (1j * G.ky1)[:, None], n=G.ny, dim=-2)


def _pad1(f, n, dim):
    F = torch.fft.rfft(f, dim=dim, norm="forward").narrow(dim, 0, n // 2)
    return torch.fft.irfft(F, n=3 * n // 2, dim=dim, norm="forward")   # zero-extended, Nyquist dropped


def _unpad1(f, n, dim):
    F = torch.fft.rfft(f, dim=dim, norm="forward").narrow(dim, 0, n // 2)
    return torch.fft.irfft(F, n=n, dim=dim, norm="forward")


def _padding(G, f):
    return _pad1(_pad1(f, G.nx, -1), G.ny, -2)


def _unpadding(G, f):
    return _unpad1(_unpad1(f, G.nx, -1), G.ny, -2)


def _keep(G):
    """1 on the modes the 2D transforms keep, 0 on the x- and y-Nyquist ones."""
    m = torch.ones((G.ny, G.lhx), device="cuda", dtype=torch.float64)
    m[:, -1] = 0.0
    m[G.ny // 2] = 0.0
    return m


def _fftn(G, f):
    return torch.fft.rfft2(f) * _keep(G)


def _ifftn(G, F):
    return torch.fft.irfft2(F * _keep(G), s=(G.ny, G.nx), norm="forward")


def _pressure(G, u, v, w, bot=None, top=None):
    """p on levels 0..L, dpdx, dpdy, dpdz on levels 1..L from u, v, w (levels 0..nz, x < nx)."""
    cst = 1.0 / (G.nx * G.ny)
    sc = cst / TADV1 / G.dt
    L, dz, id2 = G.L, G.dz, 1.0 / (G.dz * G.dz)
    Hx, Hy, Hz = (_fftn(G, sc * f[1:L + 1]) for f in (u, v, w))
    zero = torch.zeros_like(Hz[0])
    H0 = zero if bot is None else _fftn(G, cst * bot)
    Ht = _fftn(G, cst * top) if top is not None and G.top == "neumann" else zero
    kx, ky = G.kx[None, :] * _keep(G), G.ky[:, None] * _keep(G)
    k2 = kx * kx + ky * ky
    mean = torch.zeros_like(k2)
    mean[0, 0] = 1.0
    div = _keep(G) * (1.0 - mean)
    one = torch.ones_like(k2)
    cp, d = [], []
    for i in range(L):               # row i + 1
        r = 1j * (kx * Hx[i] + ky * Hy[i]) + ((Hz[i + 1] if i + 1 < L else Ht) - Hz[i] + (H0 if i == 0 else 0)) / dz
        last = i == L - 1 and G.top == "neumann"
        b = torch.where(div > 0, -(k2 + (id2 if i == 0 or last else 2 * id2) * one), one)
        a = div * (0.0 if i == 0 else id2)
        c = div * (0.0 if last else id2)
        den = b - (a * cp[-1] if i else 0.0)
        cp.append(c / den)
        d.append((r * div - (a * d[-1] if i else 0.0)) / den)
    # the mean mode: first-order differences of H_z from p(1) = 0
    m, acc = [zero], zero
    for i in range(1, L):
        acc = acc + dz * (Hz[i] * mean)
        m.append(acc)
    p = [None] * (L + 1)
    p[L] = d[L - 1] + m[L - 1] if G.top == "neumann" else zero
    pn = d[L - 1] if G.top == "neumann" else zero
    for i in range(L - 2, -1, -1):
        pn = d[i] - cp[i] * pn
        p[i + 1] = pn + m[i]
    p[0] = p[1] - dz * H0
    P = torch.stack(p) * _keep(G)
    del p, d, cp, m, Hx, Hy, Hz
    pr = _ifftn(G, P)
    return pr, _ifftn(G, 1j * kx * P[1:]), _ifftn(G, 1j * ky * P[1:]), (pr[1:] - pr[:-1]) / dz


def _project(G, u, v, w, dx, dy, dz):
    f, L = G.dt * TADV1, G.L
    z = torch.zeros_like(w[:1])
    return (torch.cat((u[:1], u[1:L + 1] - f * dx, u[L + 1:])), torch.cat((v[:1], v[1:L + 1] - f * dy, v[L + 1:])),
            torch.cat((w[:1], z, w[2:L + 1] - f * dz[1:], z)))


def _convec(G, u, v, w):
    nz, idz = G.nz, 1.0 / G.dz
    dudy, dvdx, dwdx, dwdy = _ddy(G, u), _ddx(G, v), _ddx(G, w), _ddy(G, w)
    zero = torch.zeros_like(u[:1])

    def ddz(f):     # levels 1..nz
        m = (f[2:nz] - f[1:nz - 1]) * idz
        return torch.cat((m[:1], m, zero))

    def half(f):    # levels 1..nz: the uvp-node average at the two ends
        return torch.cat((0.5 * (f[1:2] + f[2:3]), f[2:nz], 0.5 * (f[nz:nz + 1] + f[nz - 1:nz])))

    o1 = half(dwdy) - ddz(v)
    o2 = ddz(u) - half(dwdx)
    o3 = (dvdx - dudy)[1:]
    U, V, W = (_padding(G, f) for f in (u, v, w))
    O1, O2, O3 = (_padding(G, f) for f in (o1, o2, o3))      # index k - 1
    WO2, WO1 = W[1:] * O2, W[1:] * O1
    # levels 1..nz-1
    lo2 = torch.cat((torch.zeros_like(WO2[:1]), WO2[1:nz - 1]))
    lo1 = torch.cat((torch.zeros_like(WO1[:1]), WO1[1:nz - 1]))
    X = -V[1:nz] * O3[:nz - 1] + 0.5 * (WO2[1:nz] + lo2)
    Y = U[1:nz] * O3[:nz - 1] - 0.5 * (WO1[1:nz] + lo1)
    Z = 0.5 * (-(U[2:nz] + U[1:nz - 1]) * O2[1:nz - 1] + (V[2:nz] + V[1:nz - 1]) * O1[1:nz - 1])
    Z = torch.cat((torch.zeros_like(Z[:1]), Z))
    return tuple(_unpadding(G, f) for f in (X, Y, Z))


def _rollout(G, uvw, nsteps):
    x0 = [uvw[c][..., :G.nx].double().clone().requires_grad_(True) for c in range(3)]
    u, v, w = x0
    f = G.dt * TADV1
    for _ in range(nsteps):
        c = _convec(G, u, v, w)
        u, v, w = (torch.cat((a[:1], a[1:G.L + 1] - f * b, a[G.L + 1:])) for a, b in zip((u, v, w), c))
        _, dx, dy, dz = _pressure(G, u, v, w)
        u, v, w = _project(G, u, v, w, dx, dy, dz)
    J = 0.0
    for k in range(1, G.nz):
        z = (k - 0.5) * G.dz * G.z_i
        if KE_BAND[0] < z < KE_BAND[1]:
            J = J + 0.5 * (u[k].square().sum() + v[k].square().sum() + (0.5 * (w[k] + w[k + 1])).square().sum())
    if not torch.is_tensor(J):
        return torch.zeros((), dtype=torch.float64), torch.zeros_like(torch.stack(x0))
    g = torch.autograd.grad(J, x0, allow_unused=True)
    return J.detach().cpu(), torch.stack([torch.zeros_like(a) if b is None else b for a, b in zip(x0, g)])


def _lay(f, shape, first=0):
    """f into a zero field of the given shape from level `first`."""
    out = torch.zeros(shape, device="cuda", dtype=torch.float64)
    out[first:first + f.shape[0], :, :f.shape[2]] = f
    return out


def _exact_step(nx, ny, levels, top, uvw, theta, bot, tp):
    G = _Grid(nx, ny, levels, top)
    sh = _step_shapes(nx, ny, levels)
    f = [uvw[c][..., :nx].double() for c in range(3)]
    out = {}
    for i, a in enumerate(f + [theta[..., :nx].double()]):
        out["d%d" % (2 * i)] = _lay(_ddx(G, a), sh["d0"])
        out["d%d" % (2 * i + 1)] = _lay(_ddy(G, a), sh["d0"])
        out["big%d" % i] = _padding(G, a)
    pl = [None if t is None else t[:, :nx].double() for t in (bot, tp)]
    p, *g = _pressure(G, *f, *pl)
    out["p"] = _lay(p, sh["p"])
    for i in range(3):
        out["dp%d" % i] = _lay(g[i], sh["dp0"])
    out["uvw"] = torch.stack([_lay(a, sh["p"]) for a in _project(G, *f, *g)])
    return out


def exact(case, seed):
    kind, dt = case["kind"], _dtype(case)
    if kind == "ensemble":
        parts = {}
        for k, size in enumerate(_members(case)):
            uvw, theta = _member_inputs(case, seed, k, size)
            for key, v in _exact_step(*size, case["top"], uvw, theta, None, None).items():
                v = v.reshape(-1)
                parts.setdefault(key, []).append(torch.nn.functional.pad(v, (0, -v.numel() % 64)))
        return {key: torch.cat(v) for key, v in parts.items()}
    nx, ny, levels = case["nx"], case["ny"], case["levels"]
    nz, ldx = levels + 1, nx + 2
    uvw = _velocity(seed, nx, ny, levels, dt)
    G = _Grid(nx, ny, levels, case["top"])
    bot, top = _planes(case, seed, dt)
    if kind == "step":
        return _exact_step(nx, ny, levels, case["top"], uvw, _theta(seed, nx, ny, levels, dt), bot, top)
    f = [uvw[c][..., :nx].double() for c in range(3)]
    full = (nz + 1, ny, ldx)
    if kind in ("slice", "host"):
        p, dx, dy, dz = _pressure(G, *f, *[None if t is None else t[:, :nx].double() for t in (bot, top)])
        o = dict(p=_lay(p, full), dpdx=_lay(dx, (nz, ny, ldx)), dpdy=_lay(dy, (nz, ny, ldx)), dpdz=_lay(dz, (nz, ny, ldx)))
        if kind == "host":
            return [o["p"].cpu(), o["dpdx"].cpu(), o["dpdy"].cpu()]
        return dict(o, uvw=torch.stack([_lay(a, full) for a in _project(G, *f, dx, dy, dz)]))
    if kind == "derivs":
        tau = 0.1 * _velocity(seed + 1000, nx, ny, levels, dt)
        t = [tau[c][..., :nx].double() for c in range(3)]
        o = dict(dudx=_lay(_ddx(G, f[0]), full), dudy=_lay(_ddy(G, f[0]), full))
        o["dudz"] = _lay((f[0][2:nz] - f[0][1:nz - 1]) / G.dz, full, 2)
        o["dwdz"] = _lay((f[2][2:nz + 1] - f[2][1:nz]) / G.dz, full, 1)
        h = _ddx(G, t[0]) + _ddy(G, t[1])
        a = h.clone()
        a[1:nz] += (t[2][2:nz + 1] - t[2][1:nz]) / G.dz
        o["divuv"] = _lay(a[1:nz], full, 1)
        b = h.clone()
        b[2:nz] += (t[2][2:nz] - t[2][1:nz - 1]) / G.dz
        o["divw"] = _lay(b[1:], full, 1)
        for k in ("dudz", "dwdz", "divuv", "divw"):
            o[k][0] = BOGUS
        o["divuv"][nz] = BOGUS
        return dict(o, dudz_in=o["dudz"][1:], dwdz_in=o["dwdz"][1:], divuv_in=o["divuv"][1:-1], divw_in=o["divw"][1:])
    if kind == "dealias":
        prod = _fluct(_gen(seed, 5), 3 * nx // 2, 3 * ny // 2, nz + 1).to(dt).double()
        back = _unpadding(G, prod)
        return dict(ub=_padding(G, f[0]), wb=_padding(G, f[2]), back=torch.cat((back, back[..., :2]), dim=-1))
    if kind == "filter":
        F = _fftn(G, f[1])
        flt = _ifftn(G, _fftn(G, f[0])) / (nx * ny)
        return dict(spec=torch.view_as_real(F).reshape(full), back=_lay(_ifftn(G, F), full), filt=_lay(flt, full))
    if kind == "rollout":
        J, g = _rollout(G, uvw, case["nsteps"])
        return {"J": J, "grad": g}
    return None
