"""The work that programs have this library do, as cases that can be timed and compared.

A case is a dict of plain values.  `prepare` makes what a program holds before the call (a lattice
handle with its configuration, a batch of replicas, a configuration on the device), `run` is one pass
through the public entry points, `exact` the same outputs in 64-bit arithmetic written in plain torch,
and `work` the bytes and operations a pass cannot do without.

Jobs
  chain       one measurement interval of a run: `sweeps` sweeps (heat-bath or Metropolis, then `n_or`
              over-relaxation passes each), `relax` further over-relaxation passes, one measurement
  batch       a batch of mixed replicas from their starts: seeding, `sweeps` sweeps with a measurement
              each, the series of every replica read back
  checkpoint  a configuration read in, re-projected and written out again, in device memory
  observe     energy and plaquette of a configuration that the caller holds on the device

Configurations are thermal-like: links that fluctuate about the identity as strongly as at the
case's beta (mean plaquette about 1 - 1/beta), seen in a random gauge.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import qcd_2d_gpu_b200 as q

BOUNDARY = {"periodic": 0, "pcc": 1, "pmc": 2}
AXIS = (2, 1, 0)  # dense fields are [t, x, y, ...]; directions are y, x, t
DEV = "cuda"


def chain(name, lt, lx, ly, beta, boundary, precision, algo="hb", n_or=0, sweeps=1, relax=0, upd=1, epsilon=0.1):
    c = {"job": "chain", "lt": lt, "lx": lx, "ly": ly, "beta": beta, "boundary": boundary, "precision": precision,
         "algo": algo, "n_or": n_or, "sweeps": sweeps, "relax": relax, "upd": upd, "epsilon": epsilon}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest calls: the first run of a new user and of every test, five sweeps between measurements
        chain("fp64 hb 16^3", 16, 16, 16, 6.0, "periodic", "fp64", sweeps=5),
        # Metropolis in the reference's precision, fixed-link boundary, four hits per link
        chain("fp64 metropolis 32x32x64", 32, 32, 64, 8.0, "pcc", "fp64", algo="metropolis", sweeps=2, upd=4,
              epsilon=0.2),
        # a small production lattice with over-relaxation, where launches count
        chain("fp32 hb+or 24x20x28", 24, 20, 28, 6.0, "pmc", "fp32", n_or=3, sweeps=2),
        # ragged extents: rows that fill no block, Lt without site pairs
        chain("fp32 hb+or 54x62x70", 54, 62, 70, 8.0, "pcc", "fp32", n_or=1, sweeps=1),
        # over-relaxation alone in the reference's precision, at a middle size
        chain("fp64 relax 48x64x80", 48, 64, 80, 8.0, "periodic", "fp64", sweeps=0, relax=3),
        # one interval of the accuracy study, both precisions
        chain("fp32 hb 128^3", 128, 128, 128, 8.0, "periodic", "fp32"),
        chain("fp64 hb 128^3", 128, 128, 128, 8.0, "pmc", "fp64"),
        # one interval of the large single lattice: 1 heat-bath + 3 over-relaxation passes, two sweeps
        chain("fp32 hb+or 384^3", 384, 384, 384, 10.0, "pmc", "fp32", n_or=3, sweeps=2),
        # the same kind of run in the reference's precision and without over-relaxation
        chain("fp64 hb 256^3", 256, 256, 256, 10.0, "pmc", "fp64", sweeps=2),
        # a parameter scan: 96 replicas of mixed sizes, couplings and boundaries
        {"name": "batch fp32 hb 96", "job": "batch", "replicas": 96, "most_t": 64, "most_y": 128, "sweeps": 50,
         "precision": "fp32", "shapes": 1234},
        # a saved configuration read back, re-projected and saved
        {"name": "checkpoint fp32 192^3", "job": "checkpoint", "lt": 192, "lx": 192, "ly": 192, "beta": 10.0,
         "boundary": "periodic", "precision": "fp32"},
        # measuring a configuration of another program
        {"name": "observe 160x144x176", "job": "observe", "lt": 160, "lx": 144, "ly": 176, "beta": 10.0,
         "boundary": "pmc"},
    ]


def _even(rng, lo, hi):
    return 2 * round(math.exp(rng.uniform(math.log(lo / 2), math.log(hi / 2))))


def draw(rng):
    job = rng.choices(("chain", "batch", "checkpoint", "observe"), (8, 1, 1, 1))[0]
    beta = round(rng.uniform(3.0, 12.0), 2)
    boundary = rng.choice(("periodic", "pcc", "pmc"))
    precision = rng.choice(("fp32", "fp64"))
    if job == "batch":
        return {"job": job, "replicas": rng.randint(2, 96), "most_t": _even(rng, 12, 64), "most_y": _even(rng, 12, 128),
                "sweeps": rng.randint(5, 40 if precision == "fp32" else 15), "precision": precision,
                "shapes": rng.randint(0, 9999)}
    if job == "checkpoint":
        lt, lx, ly = (_even(rng, 8, 256) for _ in range(3))
        return {"job": job, "lt": lt, "lx": lx, "ly": ly, "beta": beta, "boundary": boundary, "precision": precision}
    if job == "observe":
        lt, lx, ly = (_even(rng, 8, 256) for _ in range(3))
        return {"job": job, "lt": lt, "lx": lx, "ly": ly, "beta": beta, "boundary": boundary}
    algo = rng.choice(("hb", "hb", "hb", "metropolis"))
    most = 96 if algo == "metropolis" else 192 if precision == "fp64" else 300
    lt, lx, ly = (_even(rng, 8, most) for _ in range(3))
    n_or = rng.choice((0, 0, 1, 3))
    return chain("", lt, lx, ly, beta, boundary, precision, algo=algo, n_or=n_or, sweeps=rng.randint(1, 3),
                 relax=rng.choice((0, 0, 0, 1)), upd=rng.randint(1, 4) if algo == "metropolis" else 1,
                 epsilon=round(rng.uniform(0.05, 0.4), 3) if algo == "metropolis" else 0.1)


# ------------------------------------------------------------- inputs -----
def _mul(a, b):
    aw, ax, ay, az = a.unbind(-1)
    bw, bx, by, bz = b.unbind(-1)
    return torch.stack((aw * bw - ax * bx - ay * by - az * bz, ax * bw + aw * bx + ay * bz - az * by,
                        ay * bw + az * bx + aw * by - ax * bz, az * bw - ay * bx + aw * bz + ax * by), -1)


def _conj(a):
    return torch.cat((a[..., :1], -a[..., 1:]), -1)


def _unit(a):
    return a / a.norm(dim=-1, keepdim=True)


def _links(case, seed):
    """The case's configuration as three dense fields [t, x, y, 4] (links along y, x, t), in double."""
    g = torch.Generator(DEV)
    g.manual_seed(seed)
    shape = (case["lt"], case["lx"], case["ly"], 4)
    sigma = 1.0 / math.sqrt(6.0 * case["beta"])
    gauge = _unit(torch.randn(shape, generator=g, device=DEV, dtype=torch.float64))
    if case["boundary"] == "pcc":
        gauge[:, :, 0] = torch.tensor((1.0, 0, 0, 0), device=DEV, dtype=torch.float64)
    out = []
    for d in range(3):
        w = torch.randn(shape, generator=g, device=DEV, dtype=torch.float64).mul_(sigma)
        w[..., 0] = 1.0
        if case["boundary"] == "pcc" and d > 0:
            w[:, :, 0, 1:] = 0.0
        out.append(_mul(_mul(gauge, _unit(w)), _conj(gauge.roll(-1, AXIS[d]))))
    return out


def _parity(lt, lx):
    return (torch.arange(lt, device=DEV)[:, None] + torch.arange(lx, device=DEV)[None, :]) % 2


def _aos(links):
    """Dense fields to the layout at the boundary: V*12 doubles, even sites first, links in the order y, x, t."""
    lt, lx, ly = links[0].shape[:3]
    odd = _parity(lt, lx).bool()[:, :, None, None]
    out = torch.empty((2, lt, lx, ly // 2, 3, 4), device=DEV, dtype=torch.float64)
    for d, u in enumerate(links):
        u = u.view(lt, lx, ly // 2, 2, 4)
        out[0, ..., d, :] = torch.where(odd, u[..., 1, :], u[..., 0, :])
        out[1, ..., d, :] = torch.where(odd, u[..., 0, :], u[..., 1, :])
    return out.reshape(-1)


def _dense(aos, lt, lx, ly):
    """The inverse of _aos."""
    a = aos.view(2, lt, lx, ly // 2, 3, 4)
    odd = _parity(lt, lx).bool()[:, :, None, None]
    out = []
    for d in range(3):
        e, o = a[0, ..., d, :], a[1, ..., d, :]
        out.append(torch.stack((torch.where(odd, o, e), torch.where(odd, e, o)), 3).reshape(lt, lx, ly, 4))
    return out


class _Store:
    """The link store of a single-precision lattice, seen as an array on the device (keeps the lattice)."""

    def __init__(self, lattice):
        self.lattice = lattice
        ptr, size = lattice.link_store()
        self.__cuda_array_interface__ = {"shape": (size // 4,), "typestr": "<f4", "data": (ptr, False), "version": 3,
                                         "strides": None}


def _store_layout(aos, lt):
    """A configuration in the order of the single-precision link store (site pairs where Lt % 4 == 0)."""
    planes = aos.view(2, -1, 3, 4).permute(2, 0, 1, 3)  # direction, parity, site, component
    if lt % 4:
        return planes.reshape(-1)
    n = planes.shape[2] // 2
    return planes.reshape(6, 2, n, 4).permute(0, 2, 3, 1).reshape(-1)


def _replicas(case, seed):
    """Replicas as in a scan: shapes and couplings of the case, generators of the seed."""
    r = np.random.default_rng(case["shapes"])
    out, offset = [], 0
    for i in range(case["replicas"]):
        lt = int(r.choice(np.arange(8, case["most_t"] + 1, 2)))
        ly = int(r.choice(np.arange(8, case["most_y"] + 1, 2)))
        out.append(dict(lt=lt, lx=lt, ly=ly, beta=float(r.uniform(3.0, 12.0)), boundary=i % 3, hot=int(i % 2 == 0),
                        seed=seed, stream_offset=offset))
        offset += lt * lt * ly // 2
    return out


def _call(lattice, rc):
    if rc:
        raise q.QcdError(rc, q.load_library().qcd_last_error(lattice.handle).decode())


def prepare(case, seed):
    if case["job"] == "batch":
        b = q.Batch(_replicas(case, seed), algo="hb", precision=case["precision"],
                    renorm_every=1 if case["precision"] == "fp32" else 0)
        b.reserve(case["sweeps"])
        return {"case": case, "batch": b}
    aos = _aos(_links(case, seed))
    torch.cuda.synchronize()  # the handles launch on streams of their own
    state = {"case": case}
    if case["job"] == "observe":
        state.update(aos=aos, out=torch.zeros(2, device=DEV, dtype=torch.float64))
        return state
    lat = q.Lattice(case["lt"], case["lx"], case["ly"], case["beta"], algo=case.get("algo", "hb"),
                    boundary=case["boundary"], precision=case["precision"], epsilon=case.get("epsilon", 0.1),
                    upd=case.get("upd", 1), n_or=case.get("n_or", 0),
                    renorm_every=1 if case["precision"] == "fp32" else 0, seed=seed)
    state["lattice"] = lat
    if case["job"] == "checkpoint":
        state.update(aos=aos, out=torch.zeros_like(aos))
    else:
        _call(lat, q.load_library().qcd_load_config_device(lat.handle, aos.data_ptr()))
        torch.cuda.synchronize()
        if case["precision"] == "fp64":
            state["out"] = torch.zeros_like(aos)
    return state


# ---------------------------------------------------------------- run -----
def run(state):
    case, lib = state["case"], q.load_library()
    if case["job"] == "batch":
        b = state["batch"]
        b.init()
        b.run(case["sweeps"], measure_every=1)
        series = [b.series(i, case["sweeps"]) for i in range(case["replicas"])]
        return {"energy": np.stack([s[0] for s in series]), "plaquette": np.stack([s[1] for s in series])}
    if case["job"] == "observe":
        rc = lib.qcd_measure_aos_noalloc(state["aos"].data_ptr(), case["lt"], case["lx"], case["ly"],
                                         BOUNDARY[case["boundary"]], state["out"].data_ptr(),
                                         torch.cuda.current_stream().cuda_stream)
        if rc:
            raise q.QcdError(rc, "measure_aos_noalloc")
        return {"measured": state["out"]}
    lat = state["lattice"]
    if case["job"] == "checkpoint":
        _call(lat, lib.qcd_load_config_device(lat.handle, state["aos"].data_ptr()))
        lat.normalize()
        _call(lat, lib.qcd_store_config_device(lat.handle, state["out"].data_ptr()))
        return {"config": state["out"]}
    if case["sweeps"]:
        lat.sweep(case["sweeps"])
    if case["relax"]:
        lat.overrelax(case["relax"])
    energy, plaquette = lat.measure()
    if case["precision"] == "fp64":  # the configuration, as a program that analyses it on the device takes it
        _call(lat, lib.qcd_store_config_device(lat.handle, state["out"].data_ptr()))
        links = state["out"]
    else:  # the updated links where they lie
        links = torch.as_tensor(_Store(lat), device=DEV)
    return {"energy": energy, "plaquette": plaquette, "links": links}


def work(case):
    """One pass: links read once and written once; per update four staples of two products, and the update."""
    if case["job"] == "batch":
        v = sum(r["lt"] * r["lx"] * r["ly"] for r in _replicas(case, 0))
        size = 16 if case["precision"] == "fp32" else 32
        return {"bytes": 3.0 * v * size + 16.0 * case["replicas"] * case["sweeps"],
                "flops": 3.0 * v * case["sweeps"] * (320 + 140)}
    v = float(case["lt"]) * case["lx"] * case["ly"]
    if case["job"] == "observe":
        return {"bytes": 96 * v + 16, "flops": 3 * v * 63}
    size = 16 if case["precision"] == "fp32" else 32
    if case["job"] == "checkpoint":
        return {"bytes": 2 * 96 * v, "flops": 3 * v * 12}
    draws = case["sweeps"]
    relax = draws * case["n_or"] + case["relax"]
    rng = 24 * v if case["precision"] == "fp64" and draws else 0
    config = 96 * v if case["precision"] == "fp64" else 0
    per_draw = 320 if case["algo"] == "hb" else 240 + 60 * case["upd"]
    return {"bytes": 2 * 3 * v * size + rng + config, "flops": 3 * v * (draws * per_draw + relax * 270 + 47)}


# -------------------------------------------------------------- exact -----
M32 = 0xFFFFFFFF


def _mulhilo(m, a):
    lo = (a * m) & M32
    hi = ((a >> 16) * m + (((a & 0xFFFF) * m) >> 16)) >> 16
    return hi & M32, lo


def _philox(site, block, phase, seed):
    """Philox4x32-10 of the counters (site, block, phase) under the key `seed`: four words each."""
    x0, x1 = site, block
    x2, x3 = torch.full_like(site, phase & M32), torch.full_like(site, phase >> 32)
    k0, k1 = seed & M32, (seed >> 32) & M32
    for _ in range(10):
        h0, l0 = _mulhilo(0xD2511F53, x0)
        h1, l1 = _mulhilo(0xCD9E8D57, x2)
        x0, x1, x2, x3 = h1 ^ x1 ^ k0, l1, h0 ^ x3 ^ k1, l0
        k0, k1 = (k0 + 0x9E3779B9) & M32, (k1 + 0xBB67AE85) & M32
    return x0, x1, x2, x3


def _u24(w):
    return ((w >> 8) + 1).double() * 2.0 ** -24


def _staples(U, mu, boundary):
    A = torch.zeros_like(U[0])
    for nu in range(3):
        if nu == mu:
            continue
        m, n = AXIS[mu], AXIS[nu]
        fwd = _mul(_mul(U[nu].roll(-1, m), _conj(U[mu].roll(-1, n))), _conj(U[nu]))
        un = U[nu].roll(1, n)
        bwd = _mul(_mul(_conj(un.roll(-1, m)), _conj(U[mu].roll(1, n))), un)
        if boundary == "pmc" and nu == 0:  # no staple across the y boundary
            fwd[:, :, -1] = 0
            bwd[:, :, 0] = 0
        A += fwd + bwd
    return A


def _heatbath(A, beta, site, phase, seed):
    a = A.norm(dim=-1)
    inv = 0.5 / (a * beta)
    lf = torch.zeros_like(a)
    block = torch.zeros_like(site)
    todo = torch.arange(a.numel(), device=DEV)
    while todo.numel():
        r0, r1, r2, r3 = (_u24(w) for w in _philox(site[todo], block[todo], phase, seed))
        block[todo] += 1
        l = -(r0.log() + (2 * math.pi * r1).cos() ** 2 * r2.log()) * inv[todo]
        lf[todo] = l
        todo = todo[(1 - r3) ** 2 > 1 - l]
    w = _philox(site, block, phase, seed)
    ct, phi = 2 * _u24(w[0]) - 1, 2 * math.pi * _u24(w[1])
    n = 2 * (lf * (1 - lf)).clamp(min=0).sqrt()
    st = (1 - ct * ct).clamp(min=0).sqrt()
    X = torch.stack((1 - 2 * lf, n * ct, n * st * phi.cos(), n * st * phi.sin()), -1)
    return _mul(X, _conj(A / a[:, None]))


def _metropolis(A, U, beta, eps, upd, site, phase, seed):
    pos = torch.zeros_like(site)

    def word():
        w = torch.stack(_philox(site, pos // 4, phase, seed), -1).gather(-1, (pos % 4)[:, None])[:, 0]
        pos.add_(1)
        return w

    U = U.clone()
    for _ in range(upd):
        r = torch.stack([_u24(word()) - 0.5 for _ in range(3)], -1)
        r = eps * _unit(r)
        new = _mul(torch.cat((torch.full_like(r[:, :1], math.sqrt(1 - eps * eps)), r), -1), U)
        s = -beta * _mul(new - U, A)[:, 0]
        before = pos.clone()
        hi, lo = word(), word()
        u = (((hi << 21) | (lo >> 11)) + 1).double() * 2.0 ** -53
        pos = torch.where(s < 0, before, pos)  # the draw is taken only where the action grows
        U = torch.where(((s < 0) | ((-s).exp() > u))[:, None], new, U)
    return U


def _observables(U, boundary):
    def plaq(mu, nu):
        return _mul(_mul(_mul(U[mu], U[nu].roll(-1, AXIS[mu])), _conj(U[mu].roll(-1, AXIS[nu]))), _conj(U[nu]))[..., 0]

    a, b, c = 1 - plaq(0, 1), 1 - plaq(0, 2), 1 - plaq(1, 2)
    if boundary == "pmc":
        a[:, :, -1] = 0
        b[:, :, -1] = 0
    return float((-c).mean()), float(1 - (a + b + c).mean() / 3)


def _exact_chain(case, seed):
    lt, lx, ly = case["lt"], case["lx"], case["ly"]
    single, boundary = case["precision"] == "fp32", case["boundary"]
    beta, eps = float(np.float32(case["beta"])), float(np.float32(case.get("epsilon", 0.1)))
    U = _links(case, seed)
    if single:
        U = [u.float().double() for u in U]
    odd = (_parity(lt, lx)[:, :, None] + torch.arange(ly, device=DEV)) % 2
    t, x, y = (torch.arange(n, device=DEV) for n in (lt, lx, ly))
    ident = y[None, None, :] // 2 + (ly // 2) * (x[None, :, None] + lx * t[:, None, None])
    passes = (["draw"] + ["relax"] * case["n_or"]) * case["sweeps"]
    last = {case["n_or"] + i * (1 + case["n_or"]) for i in range(case["sweeps"])}  # re-projected, single precision
    passes += ["relax"] * case["relax"]
    drawn = 0
    for i, kind in enumerate(passes):
        for mu in range(3):
            for par in range(2):
                A = _staples(U, mu, boundary)
                at = odd == par
                if boundary == "pcc" and mu > 0:
                    at[:, :, 0] = False
                A, old, site, phase = A[at], U[mu][at], ident[at], 6 * drawn + 2 * mu + par
                if kind == "relax":
                    ratio = 2 * _mul(A, old)[:, :1] / A.square().sum(-1, keepdim=True)
                    new = ratio * _conj(A) - old
                elif case["algo"] == "hb":
                    new = _heatbath(A, beta, site, phase, seed)
                else:
                    new = _metropolis(A, old, beta, eps, case["upd"], site, phase, seed)
                U[mu][at] = _unit(new) if single and i in last else new
        drawn += kind == "draw"
    energy, plaquette = _observables(U, boundary)
    aos = _aos(U)
    return {"energy": energy, "plaquette": plaquette, "links": _store_layout(aos, lt) if single else aos}


def exact(case, seed):
    if case["job"] == "batch":
        return None  # the starts are draws of cuRAND's generator
    if case["job"] == "observe":
        return {"measured": torch.tensor(_observables(_links(case, seed), case["boundary"]), dtype=torch.float64)}
    if case["job"] == "checkpoint":
        aos = _aos(_links(case, seed))
        if case["precision"] == "fp32":
            aos = aos.float().double()
        return {"config": _unit(aos.view(-1, 4)).reshape(-1)}
    if case["precision"] == "fp64" and case["sweeps"]:
        return None  # draws of cuRAND's generator
    if case["lt"] * case["lx"] * case["ly"] * (case["sweeps"] * (1 + case["n_or"]) + case["relax"]) > 6e7:
        return None  # takes too long
    return _exact_chain(case, seed)
