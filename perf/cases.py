"""The calls whose speed counts: what a program that uses this package has it do.

A user holds a periodic box (or a batch of boxes) on the GPU, advances it by
the dt that the last step returned, and after a few steps takes the state out
on the device (for output, analysis or a halo exchange).  The cases below run
that over the package's range: the boxes of the request stream and of the
mixed batch (edges 32 to 192), the 64^3 double-precision parity box, the 256^3
and 512^3 driven-turbulence boxes, the four-scalar high-Mach box, odd edges, the
three Riemann solvers, 0 to 4 passive scalars, drive steps, and the
allocation-free step.  PPM reconstruction runs in double precision here: its
monotonicity switches are discontinuous, so single-precision results of two
correct programs differ by whole edge values where a switch flips and cannot
be compared cell by cell.

States are seeded turbulence: density 1 with smooth fluctuations, a solenoidal
velocity of the case's rms Mach number on the shells 1 <= |k| <= 2, a mean
field along a random direction plus a divergence-free fluctuation, and
smooth scalar concentrations.
"""
import ctypes
import math

import numpy as np
import torch

from isothermal_mhd_b200 import Batch, Box, _lib
from isothermal_mhd_b200.batch import make_config

COUR = 0.4
EDOT = 1.0e-3          # energy injection rate of a kick, the package's default
DT_TURB = 0.05
RIEMANN = {"roe": 1, "hlld": 2, "hlle": 3}


def _box(name, nx, ny, nz, bits, riemann, npass, mach, steps, recon="plm", drive=False):
    return {"name": name, "kind": "box", "nx": nx, "ny": ny, "nz": nz, "bits": bits, "riemann": riemann,
            "recon": recon, "npass": npass, "mach": mach, "steps": steps, "drive": drive}


def listed():
    return [
        # the most frequent request of the served stream, alone: latency of a step
        _box("box32_roe", 32, 32, 32, 32, "roe", 0, 1.0, 8),
        # the double-precision parity configuration
        _box("box64_f64_roe", 64, 64, 64, 64, "roe", 1, 0.5, 6),
        # an ordinary request
        _box("box96_hlld", 96, 96, 96, 32, "hlld", 0, 1.0, 8),
        # odd edges: no row tile divides them
        _box("box101x83x67_hlle", 101, 83, 67, 32, "hlle", 1, 1.0, 6),
        # the largest edge of the mixed batch, with a forcing kick
        _box("box128_driven", 128, 128, 128, 32, "roe", 2, 1.0, 6, drive=True),
        # double precision with PPM, the most expensive reconstruction
        _box("box96_f64_ppm", 96, 96, 96, 64, "hlld", 1, 0.7, 3, recon="ppm"),
        # allocation-free step on the caller's buffers
        {"name": "static64_hlld", "kind": "static", "nx": 64, "ny": 64, "nz": 64, "bits": 32, "riemann": "hlld",
         "recon": "plm", "npass": 2, "mach": 1.0, "steps": 4, "drive": False},
        # mixed boxes advanced together by graph replays, results to the host
        {"name": "batch10", "kind": "batch", "edges": "32,32,33,40,48,48,64,64,96,32", "bits": 32, "riemann": "roe",
         "recon": "plm", "npass": 0, "mach": 1.0, "steps": 48, "drive": False},
        # the 256^3 production box
        _box("box256_hlld", 256, 256, 256, 32, "hlld", 2, 1.5, 4),
        # four scalars in a high-Mach box with a weak field
        _box("box320_mach4", 320, 320, 320, 32, "hlld", 4, 4.0, 3),
        # the headline box
        _box("box512_roe", 512, 512, 512, 32, "roe", 2, 2.0, 2),
    ]


def draw(rng):
    bits = 64 if rng.random() < 0.25 else 32
    top = 112 if bits == 64 else 288
    geo = [int(round(math.exp(rng.uniform(math.log(24), math.log(top))))) for _ in range(3)]
    u = rng.random()
    if u < 0.12:       # a batch of boxes
        edges = sorted(rng.choice((24, 32, 40, 48, 57, 64, 80)) for _ in range(rng.randint(4, 10)))
        return {"kind": "batch", "edges": ",".join(map(str, edges)), "bits": 32,
                "riemann": rng.choice(("roe", "hlld", "hlle")), "recon": "plm", "npass": rng.choice((0, 1, 2)),
                "mach": round(rng.uniform(0.5, 1.5), 2), "steps": rng.randint(8, 40), "drive": False}
    if u < 0.24:       # the allocation-free step
        n = rng.randint(20, 56)
        return {"kind": "static", "nx": n, "ny": n, "nz": n, "bits": bits, "riemann": rng.choice(("roe", "hlld", "hlle")),
                "recon": "plm", "npass": rng.choice((0, 1, 2)), "mach": round(rng.uniform(0.5, 1.5), 2),
                "steps": rng.randint(2, 8), "drive": False}
    if u < 0.6:        # cubes and row lengths that are whole tiles are the common choice
        m = rng.choice((16, 32, 64))
        geo = [max(m, g // m * m) for g in geo]
        if rng.random() < 0.6:
            geo = [geo[0]] * 3
    recon = "ppm" if bits == 64 and rng.random() < 0.4 else "plm"
    c = _box("", geo[0], geo[1], geo[2], bits, rng.choice(("roe", "hlld", "hlle")), rng.choice((0, 0, 1, 2, 4)),
             round(rng.uniform(0.5, 1.5), 2), rng.randint(2, 5), recon=recon, drive=rng.random() < 0.25)
    del c["name"]
    return c


def work(case):
    """State read and written once a step (rho, m, face B, scalars) and the state taken out at the end; operations
    of the reference's formulas per cell and step."""
    if case["kind"] == "batch":
        cells = sum(int(e) ** 3 for e in case["edges"].split(","))
    else:
        cells = case["nx"] * case["ny"] * case["nz"]
    npass, esz = case["npass"], case["bits"] // 8
    ops = {"roe": 5647, "hlld": 3899, "hlle": 3459}[case["riemann"]] + 126 * npass + (830 if case["recon"] == "ppm" else 0)
    return {"bytes": float(cells * esz * (case["steps"] * 2 * (7 + npass) + 10 + npass)),
            "flops": float(ops) * cells * case["steps"]}


# ------------------------------------------------------------------ inputs
def _field(shape, rng, dev, comps=3):
    """Solenoidal field on the shells 1 <= |k| <= 2 with unit rms of its norm."""
    nz, ny, nx = shape
    x = [(torch.arange(n, dtype=torch.float64, device=dev) + 0.5) / n for n in (nx, ny, nz)]
    out = torch.zeros((comps, nz, ny, nx), dtype=torch.float64, device=dev)
    for kz in range(-2, 3):
        for ky in range(-2, 3):
            for kx in range(0, 3):
                k2 = kx * kx + ky * ky + kz * kz
                if not 1 <= k2 <= 4:
                    continue
                k = np.array([kx, ky, kz], dtype=np.float64)
                a = rng.standard_normal((2, 3))
                a = a - np.outer(a @ k / k2, k)
                p = 2 * math.pi * (kx * x[0][None, None, :] + ky * x[1][None, :, None] + kz * x[2][:, None, None])
                c, s = torch.cos(p), torch.sin(p)
                for d in range(comps):
                    out[d].add_(c, alpha=float(a[0, d])).sub_(s, alpha=float(a[1, d]))
    return out.mul_(1.0 / math.sqrt(float(out.square().sum(0).mean())))


def _state(shape, npass, mach, bits, seed, dev):
    """(10 + npass, nz, ny, nx): rho, momentum, cell-centred B, face B, scalars, in the box's precision."""
    rng = np.random.default_rng(seed)
    real = torch.float64 if bits == 64 else torch.float32
    nz, ny, nx = shape
    out = torch.empty((10 + npass,) + tuple(shape), dtype=real, device=dev)
    v = _field(shape, rng, dev)
    rho = 1.0 + 0.1 * v[0] / float(v[0].abs().max()) * min(mach, 1.0)
    out[0] = rho
    for d in range(3):
        out[1 + d] = rho * v[d] * mach
    del v, rho
    d0 = rng.standard_normal(3)
    d0 *= (0.3 if mach > 3 else 0.7) / np.linalg.norm(d0)
    a = _field(shape, rng, dev).mul_(0.02)
    n = max(shape)
    b = [None] * 3       # curl of the edge-centred potential: no discrete divergence
    for d in range(3):
        e, f = (d + 1) % 3, (d + 2) % 3
        b[d] = ((a[f] - torch.roll(a[f], 1, 2 - e)) - (a[e] - torch.roll(a[e], 1, 2 - f))) * n + float(d0[d])
    del a
    for d in range(3):
        out[7 + d] = b[d]
        out[4 + d] = 0.5 * (b[d] + torch.roll(b[d], 1, 2 - d))
    del b
    for p in range(npass):       # concentrations in [0, 1]
        if p % 3 == 0:
            g = _field(shape, rng, dev)
            g.div_(2 * float(g.abs().max())).add_(0.5)
        out[10 + p] = g[p % 3]
    return out


def _force(shape, bits, seed, dev):
    """The force field of a driven box, in the box's precision."""
    return _field(shape, np.random.default_rng(seed + 2), dev).to(torch.float64 if bits == 64 else torch.float32)


def _first_dt(u, dx):
    """COUR dx over the largest |v| + fast speed of the state."""
    top = 0.0
    for k in range(0, u.shape[1], 32):
        top = max(top, float(_cell_speed(u[:, k:k + 32].double()).max()))
    return COUR * dx / top


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    bits, npass, steps = case["bits"], case["npass"], case["steps"]
    if case["kind"] == "batch":
        edges = [int(e) for e in case["edges"].split(",")]
        cfgs = [make_config(n, precision=bits, riemann=case["riemann"], recon=case["recon"], npass=npass, cour=COUR)
                for n in edges]
        bt = Batch(cfgs)
        for i, n in enumerate(edges):
            u = _state((n, n, n), npass, case["mach"], bits, seed + 100 * i, dev)
            dt = _first_dt(u, 1.0 / n)
            h = u.double().cpu().numpy()
            bt.upload(i, h[:7], h[7:10], h[10:])
            bt.schedule(i, 1 << 40, dt0=dt)
        return {"kind": "batch", "batch": bt, "steps": steps, "n": len(edges)}
    shape = (case["nz"], case["ny"], case["nx"])
    u = _state(shape, npass, case["mach"], bits, seed, dev)
    dx = 1.0 / max(shape)
    dt = _first_dt(u, dx)
    if case["kind"] == "static":
        return {"kind": "static", "case": case, "in": u, "a": torch.empty_like(u), "b": torch.empty_like(u), "dt": dt}
    box = Box((case["nx"], case["ny"], case["nz"]), precision=bits, riemann=case["riemann"], recon=case["recon"],
              npass=npass, cour=COUR, edot=EDOT, dt_turb=DT_TURB, device=dev.index)
    if case["drive"]:
        box.set_force(_force(shape, bits, seed, dev).double().cpu().numpy())
    torch.cuda.current_stream().synchronize()      # the box copies on a stream of its own
    box.unpack_planes(0, shape[0], u.view(torch.uint8))
    return {"kind": "box", "box": box, "dt": dt, "steps": steps, "drive": case["drive"], "shape": shape,
            "out": u.view(torch.uint8), "real": u.dtype, "npass": npass}


# -------------------------------------------------------------------- pass
def _parts(u, dt, npass):
    out = {"rho": u[0], "mom": u[1:4], "b": u[4:7], "bface": u[7:10], "dt": dt}
    if npass:
        out["scalars"] = u[10:]
    return out


def run(state):
    if state["kind"] == "batch":
        bt = state["batch"]
        bt.run(state["steps"])
        out = []
        for i in range(state["n"]):
            q, b, p = bt.download(i)
            out.append({k: torch.from_numpy(v).float() for k, v in (("q", q), ("b", b), ("p", p)) if v is not None})
        return out
    if state["kind"] == "static":
        c, src, dt = state["case"], state["in"], state["dt"]
        got = ctypes.c_double()
        stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        for s in range(c["steps"]):
            dst = state["b"] if s % 2 else state["a"]
            _lib.check(_lib.lib().imhd_step_static(
                c["bits"], c["nx"], c["ny"], c["nz"], RIEMANN[c["riemann"]], c["npass"], 1.0, COUR,
                ctypes.c_void_p(src.data_ptr()), ctypes.c_void_p(dst.data_ptr()), dt, ctypes.byref(got), stream))
            src, dt = dst, got.value
        return _parts(src, dt, c["npass"])
    box, dt = state["box"], state["dt"]
    for s in range(state["steps"]):
        dt = box.step(dt, state["drive"] and s == 1)
    state["dt"] = dt
    nz, ny, nx = state["shape"]
    u = box.pack_planes(0, nz, state["out"]).view(state["real"]).view(10 + state["npass"], nz, ny, nx)
    return _parts(u, dt, state["npass"])


# ------------------------------------------- the same steps in 64 bits, plainly
def _at(a, axis, s):
    """a at the cell s further along x (0), y (1) or z (2)."""
    return torch.roll(a, -s, a.dim() - 1 - axis)


def _cell_speed(u):
    rho, asq, top = u[0], 1.0, None
    bsq = (u[4] ** 2 + u[5] ** 2 + u[6] ** 2) / rho
    for d in range(3):
        bt = bsq - u[4 + d] ** 2 / rho
        cf = torch.sqrt(0.5 * (asq + bsq + torch.sqrt((asq - bsq) ** 2 + 4 * asq * bt)))
        v = (u[1 + d] / rho).abs() + cf
        top = v if top is None else torch.maximum(top, v)
    return top


def _fast_slow(asq, ca2, bt2):
    dif = torch.sqrt((asq - ca2 - bt2) ** 2 + 4 * asq * bt2)
    cf2 = 0.5 * (asq + ca2 + bt2 + dif)
    return cf2, asq * ca2 / cf2, dif


def _flux(u, v):
    return torch.stack([u[1], u[1] * v[0] + u[0] + 0.5 * (u[5] ** 2 + u[6] ** 2 - u[4] ** 2),
                        u[1] * v[1] - u[4] * u[5], u[1] * v[2] - u[4] * u[6],
                        v[0] * u[5] - v[1] * u[4], v[0] * u[6] - v[2] * u[4]])


def _six(u):
    return torch.stack([u[0], u[1], u[2], u[3], u[5], u[6]])


def _beta(by, bz):
    bt = torch.sqrt(by ** 2 + bz ** 2)
    none, h = bt < 1e-20, torch.full_like(bt, math.sqrt(0.5))
    return torch.where(none, h, by / bt), torch.where(none, h, bz / bt)


def _roe(L, R):
    """Linearised flux about the mean state with an entropy fix of 0.3 on the fast and slow waves; sound speed 1."""
    vL, vR = L[1:4] / L[0], R[1:4] / R[0]
    rho = 0.5 * (L[0] + R[0])
    sr = torch.sqrt(rho)
    vx, vy, vz = 0.5 * (vL + vR)
    bx, by, bz = L[4] / sr, 0.5 * (L[5] + R[5]) / sr, 0.5 * (L[6] + R[6]) / sr
    bt2, ca2 = by ** 2 + bz ** 2, bx ** 2
    cf2, cs2, dif = _fast_slow(1.0, ca2, bt2)
    cf, cs, ca = torch.sqrt(cf2), torch.sqrt(cs2), bx.abs()
    big = 0.5 * ((1 - ca2).abs() + bt2 + dif)
    small = cf2 * bt2 / big
    af = torch.sqrt(torch.where(ca2 <= 1, big, small) / dif)
    as_ = torch.sqrt(torch.where(ca2 <= 1, small, big) / dif)
    gy, gz = _beta(by, bz)
    S = torch.copysign(torch.ones_like(bx), bx)
    d = _six(R) - _six(L)
    i1 = 0.5 / (af ** 2 + as_ ** 2 * cf2)
    i2 = 0.5 / (af ** 2 * cf + as_ ** 2 * cs * ca)
    vt, dmt, dbt = gy * vy + gz * vz, gy * d[2] + gz * d[3], gy * d[4] + gz * d[5]
    P = i1 * (af * d[0] + as_ * cf * sr * dbt)
    Q = i2 * (as_ * cs * S * (dmt - vt * d[0]) - af * (d[1] - vx * d[0]))
    U = 0.5 * S * (gz * d[2] - gy * d[3] - d[0] * (gz * vy - gy * vz))
    V = 0.5 * sr * (gz * d[4] - gy * d[5])
    p = i1 * (as_ * cf2 * d[0] - af * cf * sr * dbt)
    q = -i2 * (as_ * ca * (d[1] - vx * d[0]) + af * cf * S * (dmt - vt * d[0]))
    amp = [P + Q, U + V, p + q, p - q, V - U, P - Q]
    ev = [vx - cf, vx - ca, vx - cs, vx + cs, vx + ca, vx + cf]
    for k in range(6):
        a = ev[k].abs()
        amp[k] = amp[k] * (a if k in (1, 4) else torch.where(a >= 0.3, a, (a + 0.09) / 0.6))
    sf, df, ss, ds = amp[0] + amp[5], amp[0] - amp[5], amp[2] + amp[3], amp[3] - amp[2]
    sa, da = amp[1] + amp[4], amp[1] - amp[4]
    t = as_ * bx * df + af * S * ds
    w = as_ * cf / sr * sf - af / (sr * cf) * ss
    m = af * sf + as_ * ss
    diss = torch.stack([m, af * (amp[0] * ev[0] + amp[5] * ev[5]) + as_ * (amp[2] * ev[2] + amp[3] * ev[3]),
                        vy * m + gy * t + S * gz * da, vz * m + gz * t - S * gy * da,
                        gy * w + gz * sa / sr, gz * w - gy * sa / sr])
    return 0.5 * (_flux(L, vL) + _flux(R, vR) - diss), vx.abs() + cf


def _hll(L, R, double_star):
    vL, vR = L[1:4] / L[0], R[1:4] / R[0]
    M = 0.5 * (L + R)
    vm = M[1] / M[0]
    cL, cR, cm = (torch.sqrt(_fast_slow(1.0, w[4] ** 2 / w[0], (w[5] ** 2 + w[6] ** 2) / w[0])[0]) for w in (L, R, M))
    sL = torch.minimum(vL[0] - cL, vm - cm).clamp(max=0.0)
    sR = torch.maximum(vR[0] + cR, vm + cm).clamp(min=0.0)
    top = torch.maximum(torch.maximum(vL[0].abs() + cL, vR[0].abs() + cR), vm.abs() + cm)
    FL, FR, uL, uR = _flux(L, vL), _flux(R, vR), _six(L), _six(R)
    i = 1.0 / (sR - sL)
    hll = (sR * FL - sL * FR + sR * sL * (uR - uL)) * i
    if not double_star:
        return hll, top
    bx, rs, ms = L[4], (sR * uR[0] - sL * uL[0] - FR[0] + FL[0]) * i, (sR * uR[1] - sL * uL[1] - FR[1] + FL[1]) * i
    vs, sq = hll[0] / rs, torch.sqrt(rs)
    aL, aR = vs - bx.abs() / sq, vs + bx.abs() / sq

    def star(u, v, s):
        k = (s - aL) * (s - aR)
        near = ((s - aL).abs() < 1e-20) | ((s - aR).abs() < 1e-20)
        t1, t2 = bx * (vs - v[0]) / k, (u[0] * (s - v[0]) ** 2 - bx ** 2) / (rs * k)
        st = [rs * v[1] - t1 * u[4], rs * v[2] - t1 * u[5], t2 * u[4], t2 * u[5]]
        return torch.stack([rs, ms] + [torch.where(near, u[2 + m], st[m]) for m in range(4)])

    SL, SR = star(uL, vL, sL), star(uR, vR, sR)
    X = sq * torch.copysign(torch.ones_like(bx), bx)
    c = [0.5 * (SL[2 + m] + SR[2 + m] + X * (SR[4 + m] - SL[4 + m])) for m in range(2)]
    e = [0.5 * (SL[4 + m] + SR[4 + m] + (SR[2 + m] - SL[2 + m]) / X) for m in range(2)]
    mid = torch.stack([hll[0], hll[1], c[0] * vs - bx * e[0], c[1] * vs - bx * e[1],
                       vs * e[0] - c[0] * bx / rs, vs * e[1] - c[1] * bx / rs])
    F = torch.where(aR <= 0, FR + sR * (SR - uR), mid)
    F = torch.where(aL >= 0, FL + sL * (SL - uL), F)
    F = torch.where(sR <= 0, FR, F)
    return torch.where(sL >= 0, FL, F), top


def _riemann(L, R, name):
    return _roe(L, R) if name == "roe" else _hll(L, R, name == "hlld")


def _slope(wm, w, wp, wq, bn):
    """Limited characteristic slope (PLM), or the difference of the slopes of the next cell and this one (wq given)."""
    sr = torch.sqrt(w[0])
    bx, by, bz = bn / sr, w[4] / sr, w[5] / sr
    bt2 = by ** 2 + bz ** 2
    cf2, cs2, dif = _fast_slow(1.0, bx ** 2, bt2)
    af, as_ = torch.sqrt(((1 - cs2) / dif).clamp(min=0)), torch.sqrt(((cf2 - 1) / dif).clamp(min=0))
    none = dif < 1e-14
    af, as_ = torch.where(none, torch.ones_like(af), af), torch.where(none, torch.zeros_like(as_), as_)
    cf, cs = torch.sqrt(cf2), torch.sqrt(cs2)
    gy, gz = _beta(by, bz)
    S = torch.copysign(torch.ones_like(bx), bx)

    def left(d):
        vt, bt = gy * d[2] + gz * d[3], gy * d[4] + gz * d[5]
        P, Q = 0.5 * (af * d[0] / w[0] + as_ * bt / sr), 0.5 * (cs * as_ * S * vt - cf * af * d[1])
        p, q = 0.5 * (as_ * d[0] / w[0] - af * bt / sr), -0.5 * (cs * as_ * d[1] + cf * af * S * vt)
        U, V = 0.5 * (gy * d[3] - gz * d[2]), 0.5 * S / sr * (gy * d[5] - gz * d[4])
        return torch.stack([P + Q, U + V, p + q, p - q, V - U, P - Q])

    def mc(a, b):
        c = 0.5 * (a + b)
        m = torch.minimum(1.01 * torch.minimum(a.abs(), b.abs()), c.abs())
        return torch.where(a * b > 0, torch.copysign(m, c), torch.zeros_like(m))

    a = [left(w - wm), left(wp - w)]
    m = mc(a[0], a[1]) if wq is None else mc(a[1], left(wq - wp)) - mc(a[0], a[1])
    sf, df, ss, ds, sa, da = m[0] + m[5], m[5] - m[0], m[2] + m[3], m[3] - m[2], m[1] + m[4], m[4] - m[1]
    t, b = S * (cf * af * ds - cs * as_ * df), sr * (as_ * sf - af * ss)
    return torch.stack([w[0] * (af * sf + as_ * ss), cf * af * df + cs * as_ * ds, gy * t + gz * da, gz * t - gy * da,
                        gy * b - gz * S * sr * sa, gz * b + gy * S * sr * sa])


def _edges(wm, w, wp, dm, d):
    l, r = 0.5 * (wm + w) - dm / 6, 0.5 * (w + wp) - d / 6
    t1, t2, t3 = (r - w) * (w - l), 6 * (r - l) * (w - 0.5 * (l + r)), (r - l) ** 2
    flat, lo, hi = t1 <= 0, t2 > t3, t2 < -t3
    return (torch.where(flat, w, torch.where(lo, 3 * w - 2 * r, l)),
            torch.where(flat, w, torch.where(hi & ~lo, 3 * w - 2 * l, r)))


def _sweep(u, d, name, recon):
    """Fluxes through the upper faces along axis d and their largest speed per cell; recon None: first order."""
    i, j, k = d, (d + 1) % 3, (d + 2) % 3
    bn = u[7 + i]
    if recon is None:
        q = torch.stack([u[0], u[1 + i], u[1 + j], u[1 + k], bn, u[4 + j], u[4 + k]])
        r = _at(q, d, 1)
        r[4] = bn
        return _riemann(q, r, name)
    w = torch.stack([u[0], u[1 + i] / u[0], u[1 + j] / u[0], u[1 + k] / u[0], u[4 + j], u[4 + k]])
    wm, wp = _at(w, d, -1), _at(w, d, 1)
    if recon == "plm":
        s = _slope(wm, w, wp, None, bn)
        lo, hi = w - 0.5 * s, w + 0.5 * s
    else:
        s = _slope(wm, w, wp, _at(w, d, 2), bn)
        lo, hi = _edges(wm, w, wp, _at(s, d, -1), s)
    lo = _at(lo, d, 1)
    return _riemann(*(torch.stack([e[0], e[1] * e[0], e[2] * e[0], e[3] * e[0], bn, e[4], e[5]]) for e in (hi, lo)), name)


def _corner(u, F):
    """Edge EMFs from the face and cell EMFs, upwinded by the face velocity."""
    v = u[1:4] / u[0]
    out = []
    for c in range(3):
        a, b = (c + 1) % 3, (c + 2) % 3          # E_c = -(v_a B_b - v_b B_a)
        ec = v[b] * u[4 + a] - v[a] * u[4 + b]
        ea, eb = -F[a][4], F[b][5]               # the face EMFs are the fluxes of the transverse field
        va, vb = 0.5 * (v[a] + _at(v[a], a, 1)), 0.5 * (v[b] + _at(v[b], b, 1))

        def pick(s, x, y):
            return torch.where(s > 1e-20, x, torch.where(s < -1e-20, y, 0.5 * (x + y)))

        # along b, at the quarter points next to the edge, upwinded across a; and the other way round
        lo, hi = 2 * (eb - ec), 2 * (_at(ec, b, 1) - eb)
        x = pick(va, lo, _at(lo, a, 1)) - pick(va, hi, _at(hi, a, 1))
        lo, hi = 2 * (ea - ec), 2 * (_at(ec, a, 1) - ea)
        y = pick(vb, lo, _at(lo, b, 1)) - pick(vb, hi, _at(hi, b, 1))
        out.append(0.25 * (ea + _at(ea, b, 1) + eb + _at(eb, a, 1)) + 0.125 * (x + y))
    return out


def _update(u, F, E, c):
    new = torch.empty_like(u)
    flux = [torch.zeros_like(u[0]) for _ in range(4)]
    for d in range(3):
        for m, f in ((0, 0), (1 + d, 1), (1 + (d + 1) % 3, 2), (1 + (d + 2) % 3, 3)):
            flux[m] += F[d][f] - _at(F[d][f], d, -1)
    for m in range(4):
        new[m] = u[m] - c * flux[m]
    for d in range(3):
        a, b = (d + 1) % 3, (d + 2) % 3
        new[7 + d] = u[7 + d] - c * ((E[b] - _at(E[b], a, -1)) - (E[a] - _at(E[a], b, -1)))
        new[4 + d] = 0.5 * (new[7 + d] + _at(new[7 + d], d, -1))
    return new


def _advect(s, face, v, c, base, limited):
    """base - c v . (difference of the upwind face values of s)."""
    out = base.clone()
    for d in range(3):
        lo = hi = s
        if limited:
            x, y = s - _at(s, d, -1), _at(s, d, 1) - s
            g = 0.5 * (torch.copysign(torch.ones_like(x), x) + torch.copysign(torch.ones_like(y), y)) * torch.minimum(x.abs(), y.abs())
            lo, hi = s - 0.5 * g, s + 0.5 * g
        up, dn = face[d]
        f = torch.where(up >= 0, hi, _at(lo, d, 1)) - torch.where(dn >= 0, _at(hi, d, -1), lo)
        out -= c * v[d] * f
    return out


def _faces(v, ghost):
    """Velocity at the upper and lower faces; ghost: the velocity that a periodic image across the box's edge has."""
    out = []
    for d in range(3):
        ax, n = 2 - d, v[d].shape[2 - d]
        up, dn = _at(v[d], d, 1), _at(v[d], d, -1)
        up.select(ax, n - 1).copy_(ghost[d].select(ax, 0))
        dn.select(ax, 0).copy_(ghost[d].select(ax, n - 1))
        out.append((0.5 * (v[d] + up), 0.5 * (v[d] + dn)))
    return out


def _step(u, dt, dx, case, force):
    npass, c, top = case["npass"], dt / dx, 0.0
    F = []
    for d in range(3):
        f, s = _sweep(u, d, case["riemann"], None)
        F.append(f)
        top = max(top, float(s.max()))
    h = _update(u, F, _corner(u, F), 0.5 * c)
    F = []
    for d in range(3):
        f, s = _sweep(h, d, case["riemann"], case["recon"])
        F.append(f)
        top = max(top, float(s.max()))
    new = _update(u, F, _corner(h, F), c)
    del h, F
    kick, plain = 0.0, new[1:4]
    if force is not None:
        rho, dx3 = u[0], dx ** 3
        q1, q2 = 0.5 * float((rho * force.square().sum(0)).sum()), float((force * u[1:4]).sum())
        amp = 0.5 * (-q2 + math.sqrt(q2 * q2 + 4 * EDOT * DT_TURB / dx3 * q1)) / q1
        dm = amp * (rho * force - ((rho * force).sum((1, 2, 3)) * dx3).view(3, 1, 1, 1))
        plain = new[1:4].clone()
        new[1:4] += dm
        kick = float((dm.abs() / rho).max())
    if npass:
        v0 = u[1:4] / u[0]
        v, ghost = 0.5 * (v0 + new[1:4] / new[0]), 0.5 * (v0 + plain / new[0])
        f0, f1 = _faces(v0, v0), _faces(v, ghost)
        for p in range(10, 10 + npass):
            half = _advect(u[p], f0, v0, 0.5 * c, u[p], False)
            new[p] = _advect(half, f1, v, c, u[p], True)
    speed = max(float(_cell_speed(new).max()), top + kick)
    return new, (0.5 if force is not None else 1.0) * COUR * dx / speed


def _march(u, case, steps, force=None):
    dx = 1.0 / max(u.shape[1:])
    dt = _first_dt(u, dx)
    u = u.double()
    for s in range(steps):
        u, dt = _step(u, dt, dx, case, force if s == 1 else None)
    return u, dt


def exact(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device()) if torch.cuda.is_available() else torch.device("cpu")
    npass, bits = case["npass"], case["bits"]
    if case["kind"] == "batch":
        out = []
        for i, n in enumerate(int(e) for e in case["edges"].split(",")):
            u, _ = _march(_state((n, n, n), npass, case["mach"], bits, seed + 100 * i, dev), case, case["steps"])
            out.append({"q": u[:7].cpu(), "b": u[7:10].cpu()})
            if npass:
                out[-1]["p"] = u[10:].cpu()
        return out
    shape = (case["nz"], case["ny"], case["nx"])
    if shape[0] * shape[1] * shape[2] > 40_000_000:
        return None
    force = _force(shape, bits, seed, dev).double() if case["drive"] else None
    u, dt = _march(_state(shape, npass, case["mach"], bits, seed, dev), case, case["steps"], force)
    return _parts(u, dt, npass)
