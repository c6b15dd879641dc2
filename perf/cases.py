"""The work that a program using this framework has it do, as measured cases.

Every case advances a two-phase bubble cloud by a few LSRK3 steps through the
public entry points (the Python ``mpcf.Solver`` / ``WindowSolver`` /
``GPUlab`` and the C ABI calls beneath them that take device pointers):

- ``run``    a resident run: the state set from device arrays, ``steps`` steps
             replayed as a CUDA graph, the state read back into device arrays
             (an ensemble of domains when ``ndom`` > 1);
- ``step``   the command-line driver's loop: one step at a time with its dt
             and the device error word read back after each;
- ``lab``    the reference's integrator over the lab interface: the sound
             speed on the host, then three stages with the host's dt/h;
- ``host``   a state that lives in page-locked host memory, streamed through
             the GPU every step;
- ``window`` the same for a domain that passes through a few device slots.

``run``, ``step`` and ``lab`` start each pass from the prepared state; the two
streamed forms advance the host arrays further with every pass.
"""
import ctypes
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cubism-jr-gpu-mpcf_b200"))
import mpcf  # noqa: E402
from mpcf._lib import check, lib  # noqa: E402

CFL = 0.3
LSRK3 = ((0.0, 1.0 / 4), (-17.0 / 32, 8.0 / 9), (-32.0 / 27, 3.0 / 4))
EDGES = (32, 48, 64, 96, 128)
ABSORBING, REFLECTING = 0, 1
# Operations per cell and stage that the algorithm cannot do without: the
# reconstruction of both edges of a cell (7 quantities, 3 directions, ~73
# each), three face fluxes (~110 each), primitives, divergence and update.
FLOPS_PER_CELL_STAGE = 1950


def listed():
    return [
        # a short shock-tube-like run at the command line's smallest sizes,
        # its loop reading dt and the error word every step: launch latency
        dict(name="tube_64x8x8", kind="step", prec="fp32_ref", nx=64, ny=8, nz=8, ndom=1, bubbles=1, refl=0, tuned=False, steps=10),
        # one bubble in a 64^3 box, the smallest benchmark configuration,
        # tuned as the command line does
        dict(name="bubble_64", kind="step", prec="fp32_ref", nx=64, ny=64, nz=64, ndom=1, bubbles=1, refl=0, tuned=True, steps=10),
        # an odd-sized box between walls (rows of no 16-byte multiple), as
        # set up by a program that takes every default
        dict(name="walls_161x93x77", kind="run", prec="mixed", nx=161, ny=93, nz=77, ndom=1, bubbles=8, refl=63, tuned=False, steps=4),
        # the reference's integrator driving the lab interface (drop-in form)
        dict(name="lab_128", kind="lab", prec="fp32_ref", nx=128, ny=128, nz=128, ndom=1, bubbles=20, refl=0, tuned=False, steps=3),
        # the medium cloud in the fastest form, tuned
        dict(name="cloud_256_fp32", kind="run", prec="fp32", nx=256, ny=256, nz=256, ndom=1, bubbles=50, refl=0, tuned=True, steps=5),
        # the medium cloud in the bit-exact form, every default
        dict(name="cloud_256_ref", kind="run", prec="fp32_ref", nx=256, ny=256, nz=256, ndom=1, bubbles=50, refl=0, tuned=False, steps=2),
        # the headline: the large cloud, mixed precision, tuned, with the
        # conservation sums
        dict(name="cloud_512_mixed", kind="run", prec="mixed", nx=512, ny=512, nz=512, ndom=1, bubbles=200, refl=0, tuned=True, steps=4),
        # a parameter study: 64 domains of mixed sizes in one solver, tuned
        dict(name="ensemble_64", kind="run", prec="mixed", nx=0, ny=0, nz=0, ndom=64, bubbles=4, refl=0, tuned=True, steps=4),
        # double precision: the tuned form and the reference's expressions
        dict(name="cloud_192_fp64_fast", kind="run", prec="fp64_fast", nx=192, ny=192, nz=192, ndom=1, bubbles=30, refl=0, tuned=True, steps=3),
        dict(name="channel_fp64", kind="run", prec="fp64", nx=256, ny=96, nz=80, ndom=1, bubbles=10, refl=12, tuned=False, steps=2),
        # the state in host memory, streamed through the GPU every step
        dict(name="host_256_mixed", kind="host", prec="mixed", nx=256, ny=256, nz=256, ndom=1, bubbles=50, refl=0, tuned=False, steps=3),
        # a domain passing through device slots in chunks of planes
        dict(name="window_192_ref", kind="window", prec="fp32_ref", nx=192, ny=160, nz=192, ndom=1, bubbles=20, refl=0, tuned=False, steps=3),
    ]


def draw(rng):
    kind = rng.choice(("run", "run", "run", "step", "lab", "host", "window"))
    prec = rng.choice(("fp32_ref", "fp32", "mixed", "mixed", "fp64_fast", "fp64"))
    limit = 6.0e6 if prec.startswith("fp64") else 2.4e7
    while True:
        nx, ny, nz = (int(round(math.exp(rng.uniform(math.log(8), math.log(448))))) for _ in range(3))
        if nx * ny * nz <= limit:
            break
    if rng.random() < 0.5:      # half of the boxes have power-of-two-friendly rows
        nx = max(8, nx // 8 * 8)
    if kind == "window":
        nz = 16 * max(3, nz // 16)
    ndom = rng.choice((1, 1, 1, 12)) if kind == "run" and nx * ny * nz <= 1e6 else 1
    if ndom > 1:
        nx = ny = nz = 0
    return dict(kind=kind, prec=prec, nx=nx, ny=ny, nz=nz, ndom=ndom, bubbles=rng.randint(1, 20), refl=rng.choice((0, 0, 63, 12, rng.randint(0, 63))),
                tuned=kind in ("run", "step") and rng.random() < 0.5 and max(nx, 96) * max(ny, 96) * max(nz, 96) <= 8e6,
                steps=rng.choice((1, 2, 3)), layout=rng.randint(1, 10 ** 6))


def domains(case):
    """(nx, ny, nz) of every domain of a case (its sizes, not its inputs)."""
    if case["ndom"] == 1:
        return [(case["nx"], case["ny"], case["nz"])]
    r = random.Random(case.get("layout", 4))
    return [tuple(r.choice(EDGES) for _ in range(3)) for _ in range(case["ndom"])]


def real(case):
    return torch.float64 if case["prec"].startswith("fp64") else torch.float32


def faces(case):
    return tuple(REFLECTING if case["refl"] >> f & 1 else ABSORBING for f in range(6))


def cloud(dims, nb, seed, dtype, device):
    """Liquid (rho 1000, p 100, gamma 6.59, pc 4096) with gas bubbles, the
    interface smoothed over 1.5 cells, velocity noise of 1e-3: the conserved
    fields (rho, rho u, rho v, rho w, E, G, P) of one domain, x fastest."""
    nx, ny, nz = dims
    h = 1.0 / max(dims)
    ext = [n * h for n in dims]
    r = random.Random(seed)
    ax = [(torch.arange(n, device=device, dtype=torch.float64) + 0.5) * h for n in dims]
    phi = torch.full((nz, ny, nx), 20 * h, device=device, dtype=torch.float64)
    edge = min(ext)
    lo_r, hi_r = (0.08, 0.2) if nb <= 8 else (0.02, 0.06)
    for _ in range(nb):
        c = [r.uniform(0.2 * e, 0.8 * e) for e in ext]
        rad = r.uniform(lo_r, hi_r) * edge
        lo = [max(0, int((c[i] - rad) / h) - 12) for i in range(3)]
        hi = [min(dims[i], int((c[i] + rad) / h) + 13) for i in range(3)]
        d2 = [(ax[i][lo[i]:hi[i]] - c[i]) ** 2 for i in range(3)]
        d = (d2[2][:, None, None] + d2[1][None, :, None] + d2[0][None, None, :]).sqrt_().sub_(rad)
        box = phi[lo[2]:hi[2], lo[1]:hi[1], lo[0]:hi[0]]
        torch.minimum(box, d, out=box)
    a = phi.div_(1.5 * h).tanh_().mul_(-0.5).add_(0.5)       # gas fraction
    G = a * (1 / 0.4 - 1 / 5.59) + 1 / 5.59
    P = (1 - a) * (6.59 * 4096.0 / 5.59)
    rho = a * (1.0 - 1000.0) + 1000.0
    E = (a * (0.0234 - 100.0) + 100.0) * G + P
    del phi, a
    g = torch.Generator(device=device)
    g.manual_seed(seed)
    mom = []
    for _ in range(3):
        u = torch.rand(rho.shape, generator=g, device=device, dtype=torch.float64).mul_(2e-3).sub_(1e-3)
        E += 0.5 * rho * u * u
        mom.append((rho * u).to(dtype).reshape(-1))
    return [rho.to(dtype).reshape(-1)] + mom + [v.to(dtype).reshape(-1) for v in (E, G, P)]


def inputs(case, seed, device):
    """The 7 fields, the domains one after another in each."""
    parts = [cloud(d, case["bubbles"], 1000 * seed + i, real(case), device) for i, d in enumerate(domains(case))]
    return parts[0] if len(parts) == 1 else [torch.cat([p[q] for p in parts]) for q in range(7)]


def prepare(case, seed):
    dims = domains(case)
    init = inputs(case, seed, "cuda")
    if case["kind"] in ("host", "window"):
        host = [torch.empty(v.numel(), dtype=v.dtype, pin_memory=True) for v in init]
        for t, v in zip(host, init):
            t.copy_(v)
        if case["kind"] == "window":
            s = mpcf.WindowSolver(dims[0], 16, nslots=6, bc=faces(case), precision=case["prec"])
        else:
            s = mpcf.Solver(dims, bc=faces(case), precision=case["prec"])
        return dict(case=case, solver=s, keep=host, host=[t.numpy() for t in host])
    out = [torch.empty_like(v) for v in init]
    torch.cuda.synchronize()
    s = mpcf.Solver(dims, bc=faces(case), precision=case["prec"])
    at, src, dst = 0, [], []
    for nx, ny, nz in dims:
        src.append((ctypes.c_void_p * 7)(*[v[at:].data_ptr() for v in init]))
        dst.append((ctypes.c_void_p * 7)(*[v[at:].data_ptr() for v in out]))
        at += nx * ny * nz
    st = dict(case=case, solver=s, src=src, dst=dst, init=init, out=out)
    s.track_conservation(case["prec"] == "mixed")
    if case["tuned"]:
        load(st)
        s.autotune(reps=1)
    return st


def load(st):
    for d, p in enumerate(st["src"]):
        check(lib().mpcf_set_state(st["solver"]._h, d, p, None, 1))


def run(st):
    case, s = st["case"], st["solver"]
    kind, steps = case["kind"], case["steps"]
    if kind == "host":
        return st["host"], s.run_host(st["host"], steps, cfl=CFL)
    if kind == "window":
        return st["host"], s.run(st["host"], steps, cfl=CFL)
    load(st)
    if kind == "run":
        s.run(steps, cfl=CFL)
        said = s.conserved_sums() if case["prec"] == "mixed" else None
    elif kind == "step":
        said = []
        for _ in range(steps):
            said.append(s.step(cfl=CFL)[0])
            if s.error_word():
                raise RuntimeError("device error word")
    else:
        lab = mpcf.GPUlab(s)
        h = 1.0 / max(s.dims[0])
        said = [mpcf.lsrk3_step(lab, h, CFL) for _ in range(steps)]
    for d, p in enumerate(st["dst"]):
        check(lib().mpcf_get_state(s._h, d, p, None, 1))
    return st["out"], said


def work(case):
    n = sum(a * b * c for a, b, c in domains(case))
    size = 8 if case["prec"].startswith("fp64") else 4
    times = case["steps"] if case["kind"] in ("host", "window") else 1     # streamed states cross the bus every step
    return {"bytes": 2.0 * 7 * size * n * times, "flops": 3.0 * FLOPS_PER_CELL_STAGE * n * case["steps"]}


def tolerance(case):
    if case["prec"] == "fp32_ref":
        return "exact"          # this form's results are the reference's rounding, bit for bit
    if case["prec"] in ("fp32", "mixed"):
        # against 64 bits the momenta are 2e-4 to 4e-4 off (a small velocity
        # noise on a large pressure), every other field below 3e-7
        return {"rel": 1.2e-3, "max": 0.1}
    # against 64 bits the momenta are up to 2e-12 off
    return {"rel": 1e-11, "max": 1e-8}


# ---------------------------------------------------------------------------
# The same steps in plain torch, 64 bits.

def pad(v, axis, lo, hi, flip):
    """Three ghost layers on either side: the edge cell repeated, or mirrored
    (with the sign of `flip`) at a reflecting face."""
    n = v.shape[axis]
    i = torch.arange(-3, n + 3, device=v.device)
    left, right = i < 0, i >= n
    j = torch.where(left, -1 - i if lo else torch.zeros_like(i), torch.where(right, 2 * n - 1 - i if hi else torch.full_like(i, n - 1), i))
    out = v.index_select(axis, j.clamp_(0, n - 1))
    if flip and lo:
        out.narrow(axis, 0, 3).neg_()
    if flip and hi:
        out.narrow(axis, n + 3, 3).neg_()
    return out


def edges(v, axis):
    """WENO5 values at the right and left edge of every cell but the two
    outermost on each side, clipped to the cell and its two neighbours."""
    n = v.shape[axis] - 4
    y = [v.narrow(axis, k, n) for k in range(5)]
    k = [y[i] - 2 * y[i + 1] + y[i + 2] for i in range(3)]
    a = [y[0] - 4 * y[1] + 3 * y[2], y[1] - y[3], 3 * y[2] - 4 * y[3] + y[4]]
    g = [1 / (13 / 12 * k[i] ** 2 + a[i] ** 2 / 4 + 1e-6) ** 2 for i in range(3)]
    del k, a
    lo, hi = torch.minimum(torch.minimum(y[1], y[2]), y[3]), torch.maximum(torch.maximum(y[1], y[2]), y[3])
    r = (g[0] * (2 * y[0] - 7 * y[1] + 11 * y[2]) + 6 * g[1] * (-y[1] + 5 * y[2] + 2 * y[3]) + 3 * g[2] * (2 * y[2] + 5 * y[3] - y[4])) \
        / (6 * (g[0] + 6 * g[1] + 3 * g[2]))
    l = (g[2] * (2 * y[4] - 7 * y[3] + 11 * y[2]) + 6 * g[1] * (-y[3] + 5 * y[2] + 2 * y[1]) + 3 * g[0] * (2 * y[2] + 5 * y[1] - y[0])) \
        / (6 * (g[2] + 6 * g[1] + 3 * g[0]))
    return torch.minimum(torch.maximum(r, lo), hi), torch.minimum(torch.maximum(l, lo), hi)


def fluxes(m, p, nv):
    """HLLC fluxes of (rho, rho u, rho v, rho w, E, G, P) and the advecting
    velocity of faces between states m and p (rho, u, v, w, p, G, P)."""
    rm, rp, um, up, pm, pp, Gm, Gp, Pm, Pp = m[0], p[0], m[nv], p[nv], m[4], p[4], m[5], p[5], m[6], p[6]
    R = (rp / rm).sqrt()
    c2m, c2p = ((pm + Pm) / Gm + pm) / rm, ((pp + Pp) / Gp + pp) / rp
    d = ((c2m + R * c2p) / (1 + R) + 0.5 * R / (1 + R) ** 2 * (up - um) ** 2).sqrt()
    uu = (um + R * up) / (1 + R)
    sm, sp = torch.minimum(uu - d, um - c2m.sqrt()), torch.maximum(uu + d, up + c2p.sqrt())
    fm, fp = rm * (sm - um), rp * (sp - up)
    ss = (pp - pm + um * fm - up * fp) / (fm - fp)
    out = [0] * 8
    for q, u, s, sgn in ((m, um, sm.clamp(max=0), 1), (p, up, sp.clamp(min=0), -1)):
        w = 0.5 * (1 + sgn * torch.sign(ss))
        s0 = sm if sgn > 0 else sp
        chi = (s0 - u) / (s0 - ss)
        E = q[5] * q[4] + q[6] + 0.5 * q[0] * (q[1] ** 2 + q[2] ** 2 + q[3] ** 2)
        for k, v in ((0, q[0]), (1, q[0] * q[1]), (2, q[0] * q[2]), (3, q[0] * q[3]), (5, q[5]), (6, q[6])):
            star = q[0] * ss * chi if k == nv else v * chi
            out[k] = out[k] + w * (v * u + (q[4] if k == nv else 0) + s * (star - v))
        out[4] = out[4] + w * (u * (E + q[4]) + s * (chi * (E + (ss - u) * (q[0] * ss + q[4] / (s0 - u))) - E))
        out[7] = out[7] + w * (u + s * (chi - 1))
    return out


def primitives(U):
    u = [U[i] / U[0] for i in (1, 2, 3)]
    p = (U[4] - 0.5 * U[0] * (u[0] ** 2 + u[1] ** 2 + u[2] ** 2) - U[6]) / U[5]
    return [U[0]] + u + [p, U[5], U[6]]


def rhs(U, bc):
    q = primitives(U)
    div, sumG, sumP, divu = [0] * 7, 0, 0, 0
    for nv, axis in ((1, 2), (2, 1), (3, 0)):
        lo, hi = bc[2 * nv - 2], bc[2 * nv - 1]
        n = q[0].shape[axis]
        m, p = [], []
        for k in range(7):
            r, l = edges(pad(q[k], axis, lo, hi, k == nv), axis)     # cells -1 .. n
            m.append(r.narrow(axis, 0, n + 1))
            p.append(l.narrow(axis, 1, n + 1))
        f = fluxes(m, p, nv)
        for k in range(7):
            div[k] = div[k] + f[k].diff(dim=axis)
        divu = divu + f[7].diff(dim=axis)
        sumG = sumG + p[5].narrow(axis, 0, n) + m[5].narrow(axis, 1, n)
        sumP = sumP + p[6].narrow(axis, 0, n) + m[6].narrow(axis, 1, n)
    div[5] = div[5] - divu * sumG / 6
    div[6] = div[6] - divu * sumP / 6
    return div


def exact(case, seed):
    dims = domains(case)
    cells = sum(a * b * c for a, b, c in dims)
    if cells * case["steps"] > 9e7:
        return None
    device = "cuda" if torch.cuda.is_available() else "cpu"
    init, at, done, dts = [v.double() for v in inputs(case, seed, device)], 0, [], []
    for nx, ny, nz in dims:
        n = nx * ny * nz
        U = [v[at:at + n].reshape(nz, ny, nx) for v in init]
        at += n
        h, dom = 1.0 / max(nx, ny, nz), []
        for _ in range(case["steps"]):
            q = primitives(U)
            sos = torch.maximum(torch.maximum(q[1].abs(), q[2].abs()), q[3].abs()) + (((q[4] + q[6]) / q[5] + q[4]) / q[0]).sqrt()
            dt = CFL * h / float(sos.max())
            dom.append(dt)
            R = [0] * 7
            for a, b in LSRK3:
                L = rhs(U, faces(case))
                R = [a * R[k] - dt / h * L[k] for k in range(7)]
                U = [U[k] + b * R[k] for k in range(7)]
        done.append(U)
        dts.append(dom)
    out = [torch.cat([U[k].reshape(-1) for U in done]) for k in range(7)]
    if case["kind"] in ("host", "window"):
        return [v.cpu().numpy() for v in out], sum(dts[0])
    if case["kind"] == "run":
        if case["prec"] != "mixed":
            return out, None
        return out, np.array([[float(U[k].sum()) for k in range(5)] for U in done])
    return out, dts[0]
