"""Performance cases of the framework: what its users run, through the public
Python entry points, over the sizes its own configurations, tests and benchmark
use.

Paths (the case's "path"):
  job      HYP x1, APE x n, the on-axis W(R,T) table of one device-resident
           configuration (the reference app's loop): the table
  smear    HYP, APE, and the smeared links packed into the caller's device
           buffer, as a time-slab program hands them on: the links
  adjoint  adjoint-representation W(R,T) of smeared links: the table
  gevp     W(R,T) between two smearing levels of one configuration: the table
  offaxis  off-axis loops, merged by size, of smeared links
  spatial  spatial Wilson loops with two-dimensional APE smearing
  polyakov Polyakov loop and its correlator up to a distance
  batch    many uneven configurations as one batch: every job's table
  host     the reference's function calls on a host configuration (each call
           uploads and downloads it): the smeared links and the table
"""
from __future__ import annotations

import itertools
import math
import random

import numpy as np
import torch

from general_code_b200 import lattice as gl
from general_code_b200.batch import Batch, Job
from general_code_b200.lattice import Lattice, LatticeData

HYP = (1.0, 0.75, 0.6)
APE = 0.5
EPS = {2: 0.3, 3: 0.25}  # width of the synthetic links, as in the benchmark


def _case(name, path, nc, prec, dims, **kw):
    c = {"name": name, "path": path, "nc": nc, "prec": prec, "lx": dims[0], "ly": dims[1],
         "lz": dims[2], "lt": dims[3]}
    c.update(kw)
    return c


def listed():
    return [
        # the reference's CPU-sized configuration: launches and latency
        _case("job_su2_16_fp64", "job", 2, "fp64", (16, 16, 16, 16), hyp=1, ape=10, r=8, t=8),
        # the ordinary SU(3) configuration in the reference's precision
        _case("job_su3_24_fp64", "job", 3, "fp64", (24, 24, 24, 24), hyp=1, ape=20, r=12, t=12),
        # the benchmark's default workload, the largest SU(3) configuration
        _case("job_su3_32_mixed", "job", 3, "mixed", (32, 32, 32, 32), hyp=1, ape=40, r=16,
              t=16),
        # the largest SU(2) configuration
        _case("job_su2_48_mixed", "job", 2, "mixed", (48, 48, 48, 48), hyp=1, ape=10, r=24,
              t=24),
        # unequal extents that fit no tile (a time extent that 4 does not divide)
        _case("job_su3_ragged_mixed", "job", 3, "mixed", (18, 20, 22, 26), hyp=1, ape=15, r=9,
              t=13),
        # smearing whose links are handed on in device memory
        _case("smear_su3_24x48_mixed", "smear", 3, "mixed", (24, 24, 24, 48), hyp=1, ape=10),
        # two smearing levels in one variational basis
        _case("gevp_su3_24_fp64", "gevp", 3, "fp64", (24, 24, 24, 24), ape=4, ape2=8, r=6, t=6),
        # loops along every spatial direction (the static potential at non-integer distances)
        _case("offaxis_su3_24_mixed", "offaxis", 3, "mixed", (24, 24, 24, 24), ape=6, r=6, t=6),
        # the spatial string tension
        _case("spatial_su3_24_fp64", "spatial", 3, "fp64", (24, 24, 24, 24), r=6, t=6, ape=10,
              every=3),
        # the finite-temperature lattice of Polyakov correlators
        _case("polyakov_su3_32x8_fp64", "polyakov", 3, "fp64", (32, 32, 32, 8), d=8, singlet=1),
        # an ensemble of uneven lattices of both groups
        _case("batch_uneven_mixed", "batch", 0, "mixed", (0, 0, 0, 0), jobs=16, mix=5),
        # a program of the reference on its own host arrays
        _case("host_su3_16_fp64", "host", 3, "fp64", (16, 16, 16, 16), ape=3, r=8, t=8),
    ]


def _extent(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["job"] * 6 + ["smear"] * 2 + ["adjoint", "gevp", "offaxis", "spatial",
                                                     "polyakov", "batch", "host"])
    nc = rng.choice([2, 3])
    prec = "fp64" if path == "host" else rng.choice(["fp64", "mixed"])
    if path == "batch":
        return {"path": path, "nc": 0, "prec": prec, "lx": 0, "ly": 0, "lz": 0, "lt": 0,
                "jobs": rng.randint(4, 12), "mix": rng.randint(0, 10 ** 6)}
    # unequal and odd extents in half of the draws, L^3 x Lt in the others
    hi = {"job": 44 if nc == 2 else 26, "smear": 40 if nc == 2 else 28, "offaxis": 16,
          "spatial": 22, "host": 16}.get(path, 24)
    ls = _extent(rng, 8, hi)
    lt = _extent(rng, 6, min(48, int(1.4 * hi)))
    dims = [ls, ls, ls, lt]
    if rng.random() < 0.5:
        dims = [max(4, ls + rng.randint(-3, 3)) for _ in range(3)] + [lt]
    c = {"path": path, "nc": nc, "prec": prec, "lx": dims[0], "ly": dims[1], "lz": dims[2],
         "lt": dims[3]}
    rr, tt = max(2, min(dims[:3]) // 2), max(2, lt // 2)
    if path == "job":
        c.update(hyp=1, ape=rng.randint(5, 40 if nc == 3 else 20), r=rr, t=tt)
    elif path == "smear":
        c.update(hyp=rng.randint(0, 1), ape=rng.randint(1, 20))
    elif path == "adjoint":
        c.update(ape=rng.randint(1, 8), r=min(rr, 8), t=min(tt, 8))
    elif path == "gevp":
        c.update(ape=rng.randint(1, 4), ape2=rng.randint(5, 10), r=min(rr, 8), t=min(tt, 8))
    elif path == "offaxis":
        c.update(ape=rng.randint(1, 8), r=rng.randint(2, 5), t=min(tt, 6))
    elif path == "spatial":
        c.update(r=min(rr, 6), t=min(rr, 6), ape=rng.randint(2, 10), every=rng.randint(1, 4))
    elif path == "polyakov":
        c.update(d=rng.randint(2, min(dims[:3]) // 2), singlet=rng.randint(0, 1))
    else:
        c.update(ape=rng.randint(1, 4), r=rr, t=tt)
    return c


def _dims(c):
    return (c["lx"], c["ly"], c["lz"], c["lt"])


def _batch_jobs(c):
    """The batch's jobs: sizes, groups and step counts spread as an ensemble's are."""
    sizes = [(8, 8, 8, 8), (12, 12, 12, 12), (16, 16, 16, 16), (16, 16, 16, 32),
             (24, 24, 24, 24), (24, 24, 24, 48)]
    rng = random.Random(c["mix"])
    jobs = []
    for k in range(c["jobs"]):
        dims = rng.choice(sizes)
        jobs.append((dims, 2 + k % 2, rng.randint(5, 30), dims[0] // 2, dims[0] // 2))
    return jobs


# ------------------------------------------------------------------- inputs
def _mm(a, b):
    """Products of small matrices (..., n, n)."""
    n = a.shape[-1]
    r = a[..., :, 0:1] * b[..., 0:1, :]
    for k in range(1, n):
        r += a[..., :, k:k + 1] * b[..., k:k + 1, :]
    return r


def _dag(a):
    return a.conj().transpose(-1, -2)


def _shift(f, d, n=1):
    """f at x + n d; f is [t][z][y][x]..."""
    return torch.roll(f, -n, dims=3 - d)


def _special(a):
    """Gram-Schmidt of (..., n, n) into SU(n)."""
    r0 = a[..., 0, :]
    r0 = r0 / r0.abs().square().sum(-1, keepdim=True).sqrt()
    if a.shape[-1] == 2:
        return torch.stack([r0, torch.stack([-r0[..., 1].conj(), r0[..., 0].conj()], -1)], -2)
    r1 = a[..., 1, :]
    r1 = r1 - (r0.conj() * r1).sum(-1, keepdim=True) * r0
    r1 = r1 / r1.abs().square().sum(-1, keepdim=True).sqrt()
    return torch.stack([r0, r1, torch.linalg.cross(r0, r1, dim=-1).conj()], -2)


def _matrices(dims, nc, seed):
    """Links U[mu][t][z][y][x] of a seeded configuration, complex128: each link
    near the unit matrix, then a random gauge transformation."""
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    shape = (dims[3], dims[2], dims[1], dims[0], nc, nc)

    def noise():
        return torch.view_as_complex(torch.randn(*shape, 2, generator=gen, device="cuda",
                                                 dtype=torch.float64))
    g = _special(noise())
    eye = torch.eye(nc, dtype=torch.complex128, device="cuda")
    out = []
    for mu in range(4):
        z = noise()
        u = _special(eye + 0.5j * EPS[nc] * (z + _dag(z)))
        out.append(_mm(_mm(g, u), _dag(_shift(g, mu))))
    return out


def _to_host(u):
    """The reference's host layout: (4 V, 18) row-major, or (4 V, 4) quaternions."""
    a = torch.stack(u, 4)  # [t][z][y][x][mu][i][j]
    nc = a.shape[-1]
    if nc == 3:
        return torch.view_as_real(a).reshape(-1, 18).cpu().numpy()
    q = torch.stack([a[..., 0, 0].real, a[..., 0, 1].imag, a[..., 0, 1].real,
                     a[..., 0, 0].imag], -1)
    return q.reshape(-1, 4).cpu().numpy()


def _host_links(dims, nc, seed):
    return _to_host(_matrices(dims, nc, seed))


def prepare(case, seed):
    c, path = case, case["path"]
    dims, nc, prec = _dims(c), c["nc"], c["prec"]
    if path == "batch":
        jobs = _batch_jobs(c)
        b = Batch([Job(dims=d, nc=n, ape_steps=a, r_max=r, t_max=t) for d, n, a, r, t in jobs],
                  prec)
        for k, j in enumerate(jobs):
            b.upload(k, _host_links(j[0], j[1], 1000 * seed + k))
        return {"case": c, "batch": b}
    links = _host_links(dims, nc, seed)
    if path == "host":
        return {"case": c, "raw": links, "conf": LatticeData(dims, nc, links.copy())}
    s = {"case": c, "lat": Lattice(dims, nc, prec)}
    lat = s["lat"]
    if path in ("job", "smear"):
        # the raw configuration stays on the device; each pass smears a copy of it
        s["raw"] = Lattice(dims, nc, prec)
        s["raw"].upload(links)
        s["raw"].synchronize()
        if path == "smear":
            n = lat.slice_bytes(dims[3])
            dt, size = (torch.float64, 8) if prec == "fp64" else (torch.float32, 4)
            s["out"] = torch.empty(n // size, dtype=dt, device="cuda")
        return s
    lat.upload(links)
    if path in ("adjoint", "gevp", "offaxis"):
        lat.hyp(*HYP, 1)
        lat.ape(APE, c["ape"])
    if path == "gevp":
        s["second"] = Lattice(dims, nc, prec)
        s["second"].copy_from(lat)
        s["second"].ape(APE, c["ape2"])
        s["second"].synchronize()
    lat.synchronize()
    return s


def _values(case, a):
    """Loop averages in the type they are computed in: the mixed form's are
    sums of FP32 traces of FP32 links."""
    return np.asarray(a, dtype=np.float64 if case["prec"] == "fp64" else np.float32)


def run(state):
    c, path = state["case"], state["case"]["path"]
    if path == "batch":
        b = state["batch"]
        b.run()
        b.synchronize()
        return [_values(c, b.wilson(k)) for k in range(c["jobs"])]
    if path == "host":
        conf = state["conf"]
        conf.array[...] = state["raw"]
        gl.smearing_HYP(conf, *HYP)
        for _ in range(c["ape"]):
            gl.smearing_APE(conf, APE)
        w = gl.wilson_loop(conf, 1, c["r"], 1, c["t"])
        return {"links": conf.array, "w": np.array([w[k] for k in sorted(w)])}
    lat = state["lat"]
    if path in ("job", "smear"):
        lat.copy_from(state["raw"])
        if c["hyp"]:
            lat.hyp(*HYP, c["hyp"])
        lat.ape(APE, c["ape"])
        if path == "job":
            return _values(c, lat.wilson_loop(1, c["r"], 1, c["t"]))
        lat.pack_slices(0, c["lt"], state["out"].data_ptr())
        return state["out"]
    if path == "adjoint":
        return _values(c, lat.wilson_loop_adjoint(1, c["r"], 1, c["t"]))
    if path == "gevp":
        return _values(c, lat.wilson_gevp(state["second"], 1, c["r"], 1, c["t"]))
    if path == "offaxis":
        w = lat.wilson_offaxis_result(1, c["r"], 1, c["t"])
        return {"keys": np.array(sorted(w)), "w": _values(c, [w[k] for k in sorted(w)])}
    if path == "spatial":
        w = lat.wilson_spatial_3d(1, c["r"], 1, c["t"], APE, 1, c["ape"], c["every"])
        return {"keys": np.array(sorted(w), dtype=np.int64),
                "w": _values(c, [w[k] for k in sorted(w)])}
    return {"loop": _values(c, lat.polyakov_loop()),
            "correlator": _values(c, lat.polyakov_correlator(c["d"], bool(c["singlet"])))}


# ------------------------------------------------------------ the work needed
def _link_bytes(nc, prec):
    return {(3, "fp64"): 144, (3, "mixed"): 48, (2, "fp64"): 32, (2, "mixed"): 16}[(nc, prec)]


def _smear_flops(v, nc, hyp, ape):
    mm, proj = (198, 600) if nc == 3 else (28, 11)
    return v * (hyp * (96 * mm + 16 * proj) + ape * 3 * (8 * mm + proj))


def _table_flops(v, nc, r, t, lines=2):
    # space lines by one product per step, loops by one trace each
    mm, dot = (198, 36) if nc == 3 else (28, 8)
    return v * 3 * (lines * r * mm + r * t * dot)


def work(case):
    c, path = case, case["path"]
    if path == "batch":
        by = fl = 0
        for d, n, a, r, t in _batch_jobs(c):
            v = math.prod(d)
            by += 4 * v * _link_bytes(n, c["prec"]) + 8 * r * t
            fl += _smear_flops(v, n, 1, a) + _table_flops(v, n, r, t)
        return {"bytes": by, "flops": fl}
    nc, prec = c["nc"], c["prec"]
    v = math.prod(_dims(c))
    b = _link_bytes(nc, prec) * v
    mm, dot = (198, 36) if nc == 3 else (28, 8)
    if path == "job":
        return {"bytes": 4 * b + 8 * c["r"] * c["t"],
                "flops": _smear_flops(v, nc, c["hyp"], c["ape"]) +
                _table_flops(v, nc, c["r"], c["t"])}
    if path == "smear":
        return {"bytes": 8 * b, "flops": _smear_flops(v, nc, c["hyp"], c["ape"])}
    if path == "adjoint":
        return {"bytes": 4 * b + 8 * c["r"] * c["t"],
                "flops": _table_flops(v, nc, c["r"], 2 * c["t"])}
    if path == "gevp":
        return {"bytes": 7 * b + 8 * c["r"] * c["t"],
                "flops": _table_flops(v, nc, c["r"], 2 * c["t"], 4)}
    if path == "offaxis":
        lines = _offaxis_lines(c["r"])
        links = sum(max(1, len(p) // m) for p, _, _, m in lines)
        return {"bytes": 4 * b + 8 * len(lines) * c["t"],
                "flops": v * (links * mm + len(lines) * c["t"] * dot)}
    if path == "spatial":
        n = 1 + len([s for s in range(1, c["ape"] + 1) if (s - 1) % c["every"] == 0
                     and c["every"] >= 1])
        return {"bytes": 3 * b + 8 * n * c["r"] * c["t"],
                "flops": v * (n * 6 * (c["r"] * mm + c["r"] * c["t"] * dot) +
                              c["ape"] * 6 * (4 * mm + (600 if nc == 3 else 11)))}
    if path == "polyakov":
        vs = v // c["lt"]
        return {"bytes": b + 8 * (2 * c["d"] + 1) ** 3,
                "flops": v * mm + vs * len(_offsets(c["d"])) * (dot if c["singlet"] else 8)}
    host = 4 * v * (18 if nc == 3 else 4) * 8
    return {"bytes": host * (2 * (1 + c["ape"]) + 1),
            "flops": _smear_flops(v, nc, 1, c["ape"]) + _table_flops(v, nc, c["r"], c["t"])}


# -------------------------------------------------- the values in 64 bits
def _project(a):
    """SU(3): six steps A <- 3/2 A - 1/2 A A^dag A, A <- (1 - (det A - 1)/3) A;
    SU(2): a / |a|."""
    if a.shape[-1] == 2:
        d = (a[..., 0, 0] * a[..., 1, 1] - a[..., 0, 1] * a[..., 1, 0]).real
        return a / d.sqrt()[..., None, None]
    for _ in range(6):
        a = 1.5 * a - 0.5 * _mm(_mm(a, _dag(a)), a)
        m = [[a[..., i, j] for j in range(3)] for i in range(3)]
        det = (m[0][0] * (m[1][1] * m[2][2] - m[1][2] * m[2][1])
               - m[0][1] * (m[1][0] * m[2][2] - m[1][2] * m[2][0])
               + m[0][2] * (m[1][0] * m[2][1] - m[1][1] * m[2][0]))
        a = (1 - (det - 1) / 3)[..., None, None] * a
    return a


def _staples(fm, fn, mu, nu):
    """Upper and lower staple of the links fm (along mu) with sides fn (along nu)."""
    up = _mm(_mm(fn, _shift(fm, nu)), _dag(_shift(fn, mu)))
    low = _mm(_mm(_dag(fn), fm), _shift(fn, mu))
    return up + _shift(low, nu, -1)


def _exact_ape(u, steps):
    u = list(u)
    for _ in range(steps):
        new = []
        for mu in range(3):
            s = (1 - APE) * u[mu]
            for nu in range(3):
                if nu != mu:
                    s = s + APE / 4 * _staples(u[mu], u[nu], mu, nu)
            new.append(_project(s))
        u[:3] = new
    return u


def _exact_hyp(u):
    a1, a2, a3 = HYP
    one = {}  # (mu, direction of the staples)
    for mu in range(4):
        for eta in range(3):
            if eta != mu:
                one[mu, eta] = _project((1 - a3) * u[mu] + a3 / 2 * _staples(u[mu], u[eta], mu,
                                                                            eta))
    two = {}
    for nu in range(3):
        for mu, skip in ((3, nu), (nu, 3)):  # V_t without nu, V_nu without t
            s = (1 - a2) * u[mu]
            for rho in range(3):
                if rho != nu:
                    eta = 3 - nu - rho  # the direction neither link is decorated against
                    s = s + a2 / 4 * _staples(one[mu, eta], one[rho, eta], mu, rho)
            two[mu, skip] = _project(s)
    s = (1 - a1) * u[3]
    for nu in range(3):
        s = s + a1 / 6 * _staples(two[3, nu], two[nu, 3], 3, nu)
    return list(u[:3]) + [_project(s)]


def _re_tr(a, b):
    """Sum of Re Tr(a b^dag)."""
    return (torch.view_as_real(a) * torch.view_as_real(b)).sum()


def _lines(f, d, n):
    """Straight lines of 1..n links along d."""
    out = [f]
    for k in range(1, n):
        out.append(_mm(out[-1], _shift(f, d, k)))
    return out


def _exact_table(u, r, t, kind="fundamental", u2=None):
    v, nc = u[0][..., 0, 0].numel(), u[0].shape[-1]
    time = _lines(u[3], 3, t)
    w = torch.zeros(t, r, dtype=torch.float64, device="cuda")
    for nu in range(3):
        pairs = [(_lines(u[nu], nu, r),) * 2]
        if u2 is not None:
            second = _lines(u2[nu], nu, r)
            pairs = [(pairs[0][0], second), (second, pairs[0][0])]
        for k in range(r):
            for i in range(t):
                far = _shift(time[i], nu, k + 1)
                for top, bottom in pairs:
                    a = _mm(time[i], _shift(top[k], 3, i + 1))
                    b = _mm(bottom[k], far)
                    if kind == "adjoint":
                        tr = (a * b.conj()).sum((-1, -2))
                        w[i, k] += (tr.abs().square() - 1).sum()
                    else:
                        w[i, k] += _re_tr(a, b) / nc
    return (w / (3 * v * len(pairs))).cpu().numpy()


def _packed(u, prec):
    """Links as the device form packs them: per direction planes of 16 bytes per site."""
    out = []
    for f in u:
        nc = f.shape[-1]
        if nc == 3:
            x = torch.view_as_real(f).reshape(-1, 18)
            x = x[:, :12].reshape(-1, 3, 4) if prec == "mixed" else x.reshape(-1, 9, 2)
        else:
            x = torch.stack([f[..., 0, 0].real, f[..., 0, 1].imag, f[..., 0, 1].real,
                             f[..., 0, 0].imag], -1).reshape(-1, 4)
            x = x.reshape(-1, 1, 4) if prec == "mixed" else x.reshape(-1, 2, 2)
        out.append(x.transpose(0, 1).reshape(-1))
    return torch.cat(out)


def _offaxis_lines(r_max):
    """[(steps, displacement, (direction, multiple), multiple)] of every line of
    the merged off-axis table: directions up to 4 in the first octant, one per
    slope, as staircases in all permuted and reflected orientations."""
    dirs = []
    for d in itertools.product(range(1, 5), range(5), range(5)):
        if d[0] >= d[1] >= d[2] and not any(e[0] * d[1] == e[1] * d[0] and
                                            e[0] * d[2] == e[2] * d[0] for e in dirs):
            dirs.append(d)
    lines = []
    for d in dirs:
        size = math.sqrt(sum(x * x for x in d))
        base, e1, e2 = [], -d[1], -d[2]
        for _ in range(d[0]):
            e1 += 2 * d[1]
            e2 += 2 * d[2]
            if e1 >= d[0]:
                base.append(1)
                e1 -= 2 * d[0]
            if e2 >= d[0]:
                base.append(2)
                e2 -= 2 * d[0]
            base.append(0)
        zeros = d.count(0)
        perms = [(0, 1, 2), (1, 0, 2), (2, 0, 1)] if zeros == 2 else \
            list(itertools.permutations(range(3)))
        flips = {0: [(1, 1, 1), (1, 1, -1), (1, -1, 1), (1, -1, -1), (1, 1, 1)],
                 1: [(1, 1, 1), (-1, 1, 1)], 2: [(1, 1, 1)]}[zeros]
        # the range [1, r_max], widened by 0.1, in multiples of the direction
        lo = _round_half_away((1 - 0.1) / size + 0.5)
        hi = _round_half_away((r_max + 0.1) / size - 0.5)
        for p in perms:
            for f in flips:
                steps = [(p[b], f[p[b]]) for b in base]
                end = [0, 0, 0]
                for ax, sg in steps:
                    end[ax] += sg
                for m in range(lo, hi + 1):
                    lines.append((steps * m, tuple(m * e for e in end), (d, m), m))
    return lines


def _round_half_away(x):
    return int(math.floor(x + 0.5))


def _exact_offaxis(u, r_max, t):
    nc, v = u[0].shape[-1], u[0][..., 0, 0].numel()
    time = _lines(u[3], 3, t)
    lines = _offaxis_lines(r_max)
    vals, cache = {}, {}
    for steps, end, group, m in lines:
        key = tuple(steps)
        if key in cache:
            got = cache[key]
        else:
            s, at = None, [0, 0, 0]
            for ax, sg in steps:
                if sg < 0:
                    at[ax] -= 1
                f = u[ax]
                for d in range(3):
                    if at[d]:
                        f = _shift(f, d, at[d])
                f = f if sg > 0 else _dag(f)
                s = f if s is None else _mm(s, f)
                if sg > 0:
                    at[ax] += 1
            got = torch.zeros(t, dtype=torch.float64, device="cuda")
            for i in range(t):
                far = time[i]
                for d in range(3):
                    if end[d]:
                        far = _shift(far, d, end[d])
                got[i] = _re_tr(_mm(time[i], _shift(s, 3, i + 1)), _mm(s, far)) / nc / v
            cache[key] = got
        vals.setdefault(group, []).append(got)
    entries = []  # [W, T, size, statistics], in the order of the directions
    for (d, m), g in vals.items():
        mean = torch.stack(g).sum(0).cpu() / len(g)
        size = math.sqrt(sum(x * x for x in d)) * m
        entries += [[float(mean[i]), i + 1, size, len(g)] for i in range(t)]
    # entries of equal size and T merge, the later one into the earlier
    i = 0
    while i < len(entries):
        j = 0
        while j < len(entries):
            if i != j and i < len(entries) and entries[i][1:3] == entries[j][1:3]:
                a, b = entries[i], entries[j]
                a[0] = (a[0] * a[3] + b[0] * b[3]) / (a[3] + b[3])
                del entries[j]
            j += 1
        i += 1
    w = {(e[1], e[2]): e[0] for e in entries}
    return {"keys": None, "w": np.array([w[k] for k in sorted(w)])}


def _exact_plane(f, ax):
    """One two-dimensional APE step of the fields f[0], f[1] along the axes ax."""
    a, b = ax
    return [_project((1 - APE) * f[0] + APE / 2 * _staples(f[0], f[1], a, b)),
            _project((1 - APE) * f[1] + APE / 2 * _staples(f[1], f[0], b, a))]


def _exact_spatial(u, c):
    nc, v = u[0].shape[-1], u[0][..., 0, 0].numel()
    measured = [0] + [s for s in range(1, c["ape"] + 1) if (s - 1) % c["every"] == 0
                      and c["every"] >= 1]
    w = {}
    for ax in ((0, 1), (0, 2), (1, 2)):
        mu = 3 - ax[0] - ax[1]
        time = _lines(u[mu], mu, c["t"])
        f = [u[ax[0]], u[ax[1]]]
        for sm in range(c["ape"] + 1):
            if sm in measured:
                for k in range(2):
                    for r, s in enumerate(_lines(f[k], ax[k], c["r"]), 1):
                        for i in range(c["t"]):
                            a = _mm(time[i], _shift(s, mu, i + 1))
                            b = _mm(s, _shift(time[i], ax[k], r))
                            key = (sm, i + 1, r)
                            w[key] = w.get(key, 0) + _re_tr(a, b) / (6 * nc * v)
            if sm < c["ape"]:
                f = _exact_plane(f, ax)
    return {"keys": None, "w": np.array([float(w[k]) for k in sorted(w)])}


def _offsets(d):
    """Offsets of the correlator: one of (x, y, z), (-x, y, z) where y and z are not 0."""
    return [(x, y, z) for z in range(-d, d + 1) for y in range(-d, d + 1)
            for x in range(0 if y and z else -d, d + 1) if math.sqrt(x * x + y * y + z * z) <= d]


def _exact_polyakov(u, c):
    p = _lines(u[3], 3, c["lt"])[-1][0]  # [z][y][x]
    nc, vs, d = p.shape[-1], p[..., 0, 0].numel(), c["d"]
    tr = p.diagonal(dim1=-2, dim2=-1).sum(-1) / nc
    out = np.zeros((2 * d + 1) ** 3)
    vals = []
    for x, y, z in _offsets(d):
        if c["singlet"]:
            q = torch.roll(p, (-z, -y, -x), dims=(0, 1, 2))
            vals.append(_re_tr(p, q) / nc / vs)
        else:
            q = torch.roll(tr, (-z, -y, -x), dims=(0, 1, 2))
            vals.append((tr * q.conj()).real.sum() / vs)
    n = 2 * d + 1
    at = [(z + d) * n * n + (y + d) * n + x + d for x, y, z in _offsets(d)]
    out[at] = torch.stack(vals).cpu().numpy()
    return {"loop": float(tr.real.mean()), "correlator": out}


def exact(case, seed):
    c, path = case, case["path"]
    if path == "batch":
        out = []
        for k, (dims, nc, ape, r, t) in enumerate(_batch_jobs(c)):
            u = _exact_ape(_exact_hyp(_matrices(dims, nc, 1000 * seed + k)), ape)
            out.append(_exact_table(u, r, t))
        return out
    u = _matrices(_dims(c), c["nc"], seed)
    if path in ("job", "smear"):
        u = _exact_ape(_exact_hyp(u) if c["hyp"] else u, c["ape"])
        return _exact_table(u, c["r"], c["t"]) if path == "job" else _packed(u, c["prec"])
    if path == "host":
        u = _exact_ape(_exact_hyp(u), c["ape"])
        w = _exact_table(u, c["r"], c["t"])
        return {"links": _to_host(u), "w": w.reshape(-1)}
    if path in ("adjoint", "gevp", "offaxis"):
        u = _exact_ape(_exact_hyp(u), c["ape"])
    if path == "adjoint":
        return _exact_table(u, c["r"], c["t"], "adjoint")
    if path == "gevp":
        return _exact_table(u, c["r"], c["t"], u2=_exact_ape(u, c["ape2"]))
    if path == "offaxis":
        return _exact_offaxis(u, c["r"], c["t"])
    if path == "spatial":
        return _exact_spatial(u, c)
    return _exact_polyakov(u, c)
