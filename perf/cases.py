"""The work that is timed: HydroC runs through the package's public entry points.

A case is a plain dict.  ``api`` says which entry points a pass goes through:

* ``domain``  -- a resident state (``Domain``): the initial state is copied into it on the
  domain's own stream, the clock is set, ``launch_steps`` advances it.  Step counts are odd: a
  run that ends on an even step leaves no fused Courant maxima behind, so the copy that the
  next pass makes into the state is what its first dt comes from.
* ``dropin``  -- the reference's own loop over ``compute_deltat`` and ``hydro_godunov`` on a
  host array (``HydroRun``): upload, steps, download.
* ``noalloc`` -- ``hydro_b200_godunov_noalloc`` on a torch tensor, one x-y and one y-x step.
* ``batch``   -- many grids in one ``Batch``: each pass retires the last runs, admits new ones
  generated on the device, advances them together and downloads every state.

``init`` says what the grid holds:

* ``centre`` / ``corner`` / ``edge``: the reference's three test cases (one hot cell at the
  centre or in the corner, or a hot column), with a seeded energy and density; most of the
  grid is at rest, as in the headline benchmark.
* ``energy_noise``: the centred blast with every cell's energy times 1 + 0.01 U(-1, 1): no two
  cells are equal, so no Riemann problem is trivial.
* ``density_noise``: the corner blast with every cell's density times 1 + 0.01 U(-1, 1), the
  mixed-precision workload's input.
* ``smooth``: a smooth moving flow with small noise, every cell with its own velocity and
  pressure: what a run looks like once its waves have crossed the grid.
"""
import ctypes
import math
import random

import numpy as np
import torch

from hydro_b200 import Batch, Domain, HydroRun, load, make_params
from hydro_b200.batch import blast_spec

_BASE = {"scheme": 1, "iorder": 2, "slope": 1.0, "bnd": "1111", "niter": 10}


def _case(name, api, nx, ny, steps, init, precision="fp64", **more):
    return {**_BASE, "name": name, "api": api, "nx": nx, "ny": ny, "steps": steps, "init": init,
            "precision": precision, **more}


def listed():
    return [
        # The smallest call: two time steps on a caller's device array that allocate nothing,
        # inside another framework's program.  Launches and latency.
        _case("noalloc_250x125", "noalloc", 250, 125, 2, "smooth"),
        # The reference application's own small run (250x125 corner blast, 100 steps) linked
        # against the library: its host loop, a Courant read-back every second step.
        _case("dropin_corner_250x125", "dropin", 250, 125, 100, "corner"),
        # The same grid in the device-resident loop, mixed precision: a parameter study's run.
        _case("mixed_corner_250x125", "domain", 250, 125, 101, "corner", "mixed"),
        # A middle-sized bit-exact run, most of it still at rest.
        _case("fp64_centre_1024", "domain", 1024, 1024, 41, "centre"),
        # The headline benchmark's grid and input, bit-exact.
        _case("fp64_centre_4096", "domain", 4096, 4096, 11, "centre"),
        # Bit-exact where every interface iterates.
        _case("fp64_energy_noise_2048", "domain", 2048, 2048, 11, "energy_noise"),
        # Odd sides, open and periodic walls, the PLMDE scheme and another slope limiter, as in
        # the reference's Sod inputs; the flow covers the grid.
        _case("fp64_plmde_3001x777", "domain", 3001, 777, 11, "smooth", scheme=2, slope=1.5,
              bnd="2233"),
        # The FP64 tier that is held to 1e-12 and not to the reference's bits, developed flow.
        _case("fma_smooth_2047x1533", "domain", 2047, 1533, 11, "smooth", "fma"),
        # The benchmark's grid and input in mixed precision.
        _case("mixed_centre_4096", "domain", 4096, 4096, 21, "centre", "mixed"),
        # The mixed-precision workload: 8192^2 corner blast with density noise.
        _case("mixed_density_noise_8192", "domain", 8192, 8192, 5, "density_noise", "mixed"),
        # The batched workload: 256 blasts of sides 64..1024, 100 steps each, mixed precision.
        _case("batch_mixed_256", "batch", 64, 1024, 100, "blasts", "mixed", count=256, mix=20261203),
        # A parameter study in bit-exact FP64: 64 small and middle grids.
        _case("batch_fp64_64", "batch", 64, 512, 40, "blasts", "fp64", count=64, mix=7),
    ]


def _side(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    api = rng.choice(["domain"] * 7 + ["dropin", "noalloc", "batch"])
    if api == "batch":
        c = _case("", "batch", 64, _side(rng, 160, 640), rng.randrange(20, 61), "blasts",
                  rng.choice(["mixed", "fp64"]), count=_side(rng, 8, 96),
                  mix=rng.randrange(1 << 30))
    elif api == "noalloc":
        c = _case("", "noalloc", _side(rng, 64, 1020), _side(rng, 64, 1020), 2,
                  rng.choice(["corner", "smooth", "energy_noise"]))
    elif api == "dropin":
        c = _case("", "dropin", _side(rng, 64, 1000), _side(rng, 64, 1000),
                  2 * rng.randrange(5, 31), rng.choice(["corner", "centre", "energy_noise"]))
    else:
        nx, ny = _side(rng, 64, 5000), _side(rng, 64, 5000)
        room = 1.6e8 / (nx * ny)  # cell-steps of a pass, kept below the largest listed case
        c = _case("", "domain", nx, ny, 2 * rng.randrange(2, max(3, min(30, int(room / 2)))) + 1,
                  rng.choice(["centre", "corner", "edge", "energy_noise", "density_noise",
                              "smooth"]),
                  rng.choice(["fp64", "fp64", "fma", "mixed", "mixed"]))
        if rng.random() < 0.4:  # the options of the reference's other inputs
            c["scheme"] = rng.choice([1, 2, 3])
            c["slope"] = rng.choice([1.0, 1.5])
            c["bnd"] = rng.choice(["1111", "2222", "3333", "2233"])
    del c["name"]
    return c


# ------------------------------------------------------------------ inputs


def _params(case):
    return make_params(case["nx"], case["ny"], scheme=case["scheme"], iorder=case["iorder"],
                       slope_type=case["slope"], niter_riemann=case["niter"],
                       boundary=tuple(int(b) for b in case["bnd"]))


def _initial(case, seed, device):
    """The padded initial state [4, ny + 4, nx + 4] on `device`: ghost cells 0, as the reference
    starts, or next to an open wall ("2", which keeps what it finds there) the cell inside it."""
    u = _interior(case, seed, device)
    if "2" in case["bnd"]:
        pad = torch.nn.functional.pad(u[None, :, 2:-2, 2:-2], (2, 2, 2, 2), mode="replicate")
        return pad[0].contiguous()
    return u


def _interior(case, seed, device):
    nx, ny, kind = case["nx"], case["ny"], case["init"]
    dx = 1.0 / nx
    rng = random.Random(seed)
    rho, e0 = 0.5 + 1.5 * rng.random(), math.exp(math.log(10.0) * rng.uniform(-1, 1))
    gen = torch.Generator(device=device).manual_seed(seed)

    def noise():
        return torch.rand((ny, nx), generator=gen, dtype=torch.float64, device=device) * 2 - 1

    u = torch.zeros((4, ny + 4, nx + 4), dtype=torch.float64, device=device)
    inner = u[:, 2:-2, 2:-2]
    if kind == "smooth":
        y = torch.linspace(0, 1, ny, dtype=torch.float64, device=device)[:, None]
        x = torch.linspace(0, 1, nx, dtype=torch.float64, device=device)[None, :]
        a, b = 6.2 * rng.random(), 6.2 * rng.random()
        r = 1.0 + 0.5 * torch.sin(6.3 * x + a) * torch.cos(4.1 * y) + 0.01 * noise()
        vx = 0.8 * torch.sin(3.1 * y + b) + 0.01 * noise()
        vy = -0.6 * torch.cos(2.7 * x + a) + 0.01 * noise()
        p = 1.0 + 0.3 * torch.cos(5.0 * x * y + b) + 0.01 * noise()
        inner[0], inner[1], inner[2] = r, r * vx, r * vy
        inner[3] = p / 0.4 + 0.5 * r * (vx * vx + vy * vy)
        return u
    inner[0], inner[3] = rho, 1e-5
    hot = e0 / dx / dx
    if kind in ("corner", "density_noise"):
        u[3, 2, 2] = hot
    elif kind == "edge":
        inner[3, :, 0] = hot
    else:
        u[3, (ny + 4) // 2, (nx + 4) // 2] = hot
    if kind == "energy_noise":
        inner[3] *= 1.0 + 0.01 * noise()
    if kind == "density_noise":
        inner[0] *= 1.0 + 0.01 * noise()
    return u


def _blasts(case, seed):
    """blast_spec's arguments of a batch: the shapes belong to the case, the blasts to the seed."""
    shape, rng = random.Random(case["mix"]), random.Random(seed)
    lo, hi = case["nx"], case["ny"]
    got = []
    for _ in range(case["count"]):
        nx, ny = (max(lo, min(hi, 8 * round(_side(shape, lo, hi) / 8))) for _ in range(2))
        got.append((nx, ny, rng.random(), rng.random(),
                    math.exp(math.log(10.0) * rng.uniform(-1, 1)), 0.5 + 1.5 * rng.random()))
    return got


class _Resident:
    """A domain's state as a tensor; the tensor keeps the domain."""

    def __init__(self, dom):
        self.dom = dom
        self.__cuda_array_interface__ = {"shape": dom.shape, "typestr": "<f8", "version": 3,
                                         "data": (dom.state_ptr, False), "strides": None}


def prepare(case, seed):
    torch.cuda.init()
    if case["api"] == "batch":
        specs = [blast_spec(*b) for b in _blasts(case, seed)]
        need = sum(Batch.bytes_needed(s[0]) for s in specs)
        b = Batch(specs[0][0], len(specs), need + (1 << 20), precision=case["precision"])
        b.set_tuning(32, 1, 0, 64)  # what the autotuner settles on for such mixes
        cells = [4 * (s[0].nx + 4) * (s[0].ny + 4) for s in specs]
        out = torch.empty(sum(cells), dtype=torch.float64, pin_memory=True)
        at = [out.data_ptr() + 8 * sum(cells[:k]) for k in range(len(cells))]
        return {"case": case, "batch": b, "specs": specs, "slots": [], "out": out, "at": at}
    H = _params(case)
    if case["api"] == "dropin":
        u0 = np.ascontiguousarray(_initial(case, seed, "cpu").numpy())
        return {"case": case, "u0": u0, "run": HydroRun(H, u0.copy())}
    u0 = _initial(case, seed, "cuda")
    if case["api"] == "noalloc":
        return {"case": case, "u0": u0, "u": torch.empty_like(u0), "H": H, "lib": load()}
    dom = Domain(H, precision=case["precision"])
    torch.cuda.current_stream().synchronize()  # u0 is read on the domain's stream
    return {"case": case, "u0": u0, "dom": dom,
            "state": torch.as_tensor(_Resident(dom), device="cuda"),
            "stream": torch.cuda.ExternalStream(dom.stream_ptr)}


def _dt(case):
    """A step below the Courant bound of the allocation-free cases' inputs: sound speed and
    velocity stay under 4 in the smooth flow; a blast's follow from its hot cell's energy."""
    dx = 1.0 / case["nx"]
    return 0.2 * dx if case["init"] == "smooth" else 0.05 * dx * dx


def run(st):
    case = st["case"]
    if case["api"] == "domain":
        with torch.cuda.stream(st["stream"]):
            st["state"].copy_(st["u0"])
        st["dom"].set_clock()
        st["dom"].launch_steps(case["steps"])
        return st["state"]
    if case["api"] == "noalloc":
        st["u"].copy_(st["u0"])
        stream = torch.cuda.current_stream().cuda_stream
        for k in range(case["steps"]):
            rc = st["lib"].hydro_b200_godunov_noalloc(ctypes.byref(st["H"]), st["u"].data_ptr(),
                                                      1 + k % 2, _dt(case), stream)
            if rc:
                raise RuntimeError("noalloc step failed")
        return st["u"]
    if case["api"] == "dropin":
        r = st["run"]
        np.copyto(r.uold, st["u0"])
        r.t, r.nstep, r.dt = 0.0, 0, 0.0
        r.sync_to_device()
        dts = r.run_host_loop(case["steps"])
        return {"state": r.sync_to_host(), "dts": dts}
    b = st["batch"]
    for slot in st["slots"]:
        b.remove(slot)
    st["slots"] = [b.try_add_blast(*s, nstepmax=case["steps"]) for s in st["specs"]]
    b.steps(case["steps"])
    for slot, at in zip(st["slots"], st["at"]):
        if b.lib.hydro_b200_batch_download(b.h, slot, at):
            raise RuntimeError("download failed")
    return st["out"]


def work(case):
    """A step reads and writes each cell's four doubles once at least; its arithmetic is about
    2 x 190 operations a cell where the interface's iteration takes two rounds."""
    if case["api"] == "batch":
        cells = sum(b[0] * b[1] for b in _blasts(case, 0))
    else:
        cells = case["nx"] * case["ny"]
    return {"bytes": 64.0 * cells * case["steps"], "flops": 380.0 * cells * case["steps"]}


# ------------------------------------------------------------------ 64-bit values
# The dimensionally split Godunov step in plain torch, 64 bits.

_GAMMA, _SMALLR, _SMALLC = 1.4, 1e-10, 1e-10
_SMALLP = _SMALLC * _SMALLC / _GAMMA


def _prims(u):
    r = u[0].clamp_min(_SMALLR)
    vn, vt = u[1] / r, u[2] / r
    p = torch.maximum((_GAMMA - 1.0) * r * (u[3] / r - 0.5 * (vn * vn + vt * vt)), r * _SMALLP)
    return torch.stack([r, vn, vt, p]), torch.sqrt(_GAMMA * p / r)


def _slopes(q, case):
    if case["iorder"] == 1:
        return torch.zeros_like(q[..., 1:-1])
    st = case["slope"]
    left, right = st * (q[..., 1:-1] - q[..., :-2]), st * (q[..., 2:] - q[..., 1:-1])
    mid = 0.5 * (left + right) / st
    lim = torch.where(left * right <= 0, 0.0, torch.minimum(left.abs(), right.abs()))
    return torch.sign(mid) * torch.minimum(lim, mid.abs())


def _traced(q, dq, c, dtdx, scheme):
    r, u, v, p = q
    zl, zr, pr = ((-100.0 / dtdx, 100.0 / dtdx, 1.0) if scheme == 1 else
                  (0.0, 0.0, 1.0 if scheme == 2 else 0.0))
    dp = dq[3] / (r * c)
    am, ap = 0.5 * (dp - dq[1]) * r / c, 0.5 * (dp + dq[1]) * r / c
    a0 = dq[0] - dq[3] / (c * c)

    def side(s):
        f = [torch.where(w >= zr, pr, w * dtdx + 1.0) if s > 0 else
             torch.where(w <= zl, -pr, w * dtdx - 1.0) for w in (u - c, u + c, u)]
        m, a, z, zv = -0.5 * f[0] * am, -0.5 * f[1] * ap, -0.5 * f[2] * a0, -0.5 * f[2] * dq[2]
        return torch.stack([r + (a + m + z), u + (a - m) * c / r, v + zv, p + (a + m) * c * c])

    return side(-1), side(1)


def _fluxes(L, R, niter):
    g6 = (_GAMMA + 1.0) / (2.0 * _GAMMA)
    rl, ul, rr, ur = L[0].clamp_min(_SMALLR), L[1], R[0].clamp_min(_SMALLR), R[1]
    pl, pr = torch.maximum(L[3], rl * _SMALLP), torch.maximum(R[3], rr * _SMALLP)
    cl, cr = _GAMMA * pl * rl, _GAMMA * pr * rr
    wl, wr = torch.sqrt(cl), torch.sqrt(cr)
    p = (((wr * pl + wl * pr) + wl * wr * (ul - ur)) / (wl + wr)).clamp_min(0.0)
    go = torch.ones_like(p, dtype=torch.bool)
    for _ in range(niter):
        a = torch.sqrt(cl * (1.0 + g6 * (p - pl) / pl))
        b = torch.sqrt(cr * (1.0 + g6 * (p - pr) / pr))
        ql, qr = 2.0 * a ** 3 / (a * a + cl), 2.0 * b ** 3 / (b * b + cr)
        d = torch.maximum(qr * ql / (qr + ql) * ((ul - (p - pl) / a) - (ur + (p - pr) / b)), -p)
        p = torch.where(go, p + d, p)
        go = go & ((d / (p + _SMALLR * _SMALLP)).abs() > 1e-6)
        if not bool(go.any()):
            break
    wr = torch.sqrt(cr * (1.0 + g6 * (p - pr) / pr))
    wl = torch.sqrt(cl * (1.0 + g6 * (p - pl) / pl))
    us = 0.5 * (ul + (pl - p) / wl + ur - (pr - p) / wr)
    left = us > 0
    s = torch.where(left, 1.0, -1.0)
    ro, uo, po, wo = (torch.where(left, a, b) for a, b in ((rl, rr), (ul, ur), (pl, pr), (wl, wr)))
    co = torch.sqrt((_GAMMA * po / ro).abs()).clamp_min(_SMALLC)
    rs = (ro / (1.0 + ro * (po - p) / (wo * wo))).clamp_min(_SMALLR)
    cs = torch.sqrt((_GAMMA * p / rs).abs()).clamp_min(_SMALLC)
    out, inn, shock = co - s * uo, cs - s * us, wo / ro - s * uo
    out, inn = torch.where(p >= po, shock, out), torch.where(p >= po, shock, inn)
    f = (0.5 * (1.0 + (out + inn) / torch.maximum(out - inn, _SMALLC + (out + inn).abs())))
    f = f.clamp(0.0, 1.0)
    r, u, q = (torch.where(out < 0, o, torch.where(inn > 0, a, f * a + (1.0 - f) * o))
               for a, o in ((rs, ro), (us, uo), (p, po)))
    v = torch.where(left, L[2], R[2])
    m = r * u
    e = u * (q / (_GAMMA - 1.0) + 0.5 * r * (u * u + v * v) + q)
    return torch.stack([m, m * u + q, m * v, e])


def _ghosts(w, along_x, lo, hi):
    """Fill the two ghost cells at each end of the last axis (w: [4, lines, n])."""
    n = w.shape[-1]
    nl = n - 4
    for k, bt in ((0, lo), (1, lo), (n - 2, hi), (n - 1, hi)):
        if bt <= 0:
            continue
        if k < 2:
            src = 3 - k if bt == 1 else (2 if along_x else 4) if bt == 2 else nl + k
        else:
            src = 2 * nl + 3 - k if bt == 1 else (nl + 2 if along_x else nl + 1) if bt == 2 \
                else k - nl
        w[..., k] = w[..., src].clone()
        if bt == 1:
            w[1, :, k] *= -1.0


def _exact_sweep(u, along_x, dtdx, case):
    b = [int(x) for x in case["bnd"]]
    # Lines along the last axis, normal momentum in slot 1.
    w = u[:, 2:-2, :] if along_x else u[[0, 2, 1, 3]].transpose(1, 2)[:, 2:-2, :].contiguous()
    _ghosts(w, along_x, *(b[:2] if along_x else b[2:]))
    step = max(1, (1 << 23) // w.shape[-1])
    for l in range(0, w.shape[1], step):
        c = w[:, l:l + step]
        q, cs = _prims(c)
        xm, xp = _traced(q[..., 1:-1], _slopes(q, case), cs[..., 1:-1], dtdx, case["scheme"])
        f = _fluxes(xm[..., :-1], xp[..., 1:], case["niter"])
        c[..., 2:-2] += (f[..., :-1] - f[..., 1:]) * dtdx
    if not along_x:
        u[:, :, 2:-2] = w.transpose(1, 2)[[0, 2, 1, 3]]


def _exact_steps(u, case, dx, steps, fixed_dt=None):
    dts, dt = [], fixed_dt
    for n in range(steps):
        if n % 2 == 0 and fixed_dt is None:
            top = _SMALLC
            for j in range(2, u.shape[1] - 2, 1024):
                q, c = _prims(u[:, j:min(j + 1024, u.shape[1] - 2), 2:-2])
                top = max(top, float((c + q[1].abs()).max()), float((c + q[2].abs()).max()))
            dt = 0.8 * dx / top
            dt = dt / 2.0 if n == 0 else dt
        for along_x in ((True, False) if n % 2 == 0 else (False, True)):
            _exact_sweep(u, along_x, dt / dx, case)
        dts.append(dt)
    return dts


def exact(case, seed):
    device = "cuda" if torch.cuda.is_available() else "cpu"
    if case["api"] == "batch":
        if case["count"] * case["steps"] > 2600:
            return None  # minutes of small tensors
        got = []
        for b in _blasts(case, seed):
            H, rho, e_bg, cell, hot = blast_spec(*b)
            u = torch.zeros((4, H.ny + 4, H.nx + 4), dtype=torch.float64, device=device)
            u[0, 2:-2, 2:-2], u[3, 2:-2, 2:-2] = rho, e_bg
            u[3, cell[1], cell[0]] = hot
            _exact_steps(u, case, H.dx, case["steps"])
            got.append(u.reshape(-1).cpu())
        return torch.cat(got)
    u = _initial(case, seed, "cpu" if case["api"] == "dropin" else device).to(device)
    dts = _exact_steps(u, case, 1.0 / case["nx"], case["steps"],
                       _dt(case) if case["api"] == "noalloc" else None)
    if case["api"] == "dropin":
        return {"state": u.cpu().numpy(), "dts": np.array(dts)}
    return u
