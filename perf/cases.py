"""Performance cases of the su2 hot path, through the Python mirror of the C ABI.

A case is a dict of plain values; its "kind" names the work:

  hmc            SU(2) HMC trajectories, then the field downloaded (a save point)
  batch          an uneven ensemble of SU(2) chains advanced together, every chain downloaded
  metropolis     checkerboard Metropolis sweeps, then the field downloaded
  flow           a Wilson-flow measurement: the records of gradient_flow
  flow_gradient  t^2 E_p(t) after some flow steps and its derivative with respect to the links
  solve          one U(1) staggered solve (CG, mixed CG on D D^+, BiCGStab on D)
  fermion_hmc    U(1) HMC trajectories with the staggered det(D D^+) monomial
  measure        the observables measured between trajectories

Fields are drawn near the plaquette that the workloads run at (about 0.64).  What a context
with FP32 links computes is returned as FP32 numbers, which is what it holds.  Delta H is a
small difference of the large H terms, which are returned instead.
"""
import math

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

from su2_b200.batch import chain_batch
from su2_b200.lattice import gaugeconfig

F64 = torch.float64
SPREAD = 0.3  # of the imaginary parts of a start link; plaquette about 0.64


def listed():
    return [
        # the smallest lattice in everyday use: algorithm checks and tuning runs, where the
        # latency of the launches is the cost
        dict(name="hmc_8x8x8x8_fp64", kind="hmc", Lx=8, Ly=8, Lz=8, Lt=8, nd=4, beta=2.3,
             precision="fp64", integrator="leapfrog", n=10, traj=10, accept=True),
        # the production workload, in the precision it is run in; the first trajectories of a
        # run are always accepted (acceptreject off)
        dict(name="hmc_32x32x32x32_mixed", kind="hmc", Lx=32, Ly=32, Lz=32, Lt=32, nd=4,
             beta=2.4, precision="mixed", integrator="omf2", n=16, traj=4, accept=False),
        # the same in FP64, the reference's precision
        dict(name="hmc_32x32x32x32_fp64", kind="hmc", Lx=32, Ly=32, Lz=32, Lt=32, nd=4,
             beta=2.4, precision="fp64", integrator="omf2", n=16, traj=4, accept=False),
        # three dimensions, extents that are no powers of two
        dict(name="hmc_48x40x36_d3_fp64", kind="hmc", Lx=48, Ly=40, Lz=1, Lt=36, nd=3, beta=2.4,
             precision="fp64", integrator="omf2", n=10, traj=8, accept=True),
        # a parameter scan: many small chains of uneven sizes in one handle
        dict(name="batch_40_chains_mixed", kind="batch", chains=40, shapes=1, precision="mixed",
             n=10, traj=6),
        # Metropolis updates of the production lattice between two measurements
        dict(name="metropolis_32x32x32x32_fp64", kind="metropolis", Lx=32, Ly=32, Lz=32, Lt=32,
             nd=4, beta=2.4, precision="fp64", delta=0.15, hits=8, sweeps=10),
        # a two-dimensional lattice, the reference's known-answer runs: launches count here
        dict(name="metropolis_100x100_d2_fp64", kind="metropolis", Lx=100, Ly=1, Lz=1, Lt=100,
             nd=2, beta=2.0, precision="fp64", delta=0.3, hits=10, sweeps=20),
        # scale setting on a thermalised field
        dict(name="flow_24x24x24x24_fp64", kind="flow", Lx=24, Ly=24, Lz=24, Lt=24, nd=4,
             beta=2.4, precision="fp64", eps=0.01, records=20),
        # gradients of the flowed energy
        dict(name="flow_gradient_24x24x24x24_mixed", kind="flow_gradient", Lx=24, Ly=24, Lz=24,
             Lt=24, nd=4, beta=2.4, precision="mixed", eps=0.01, steps=20),
        # one inversion of the Schwinger-model workload
        dict(name="solve_256x256_cg_fp64", kind="solve", Lx=256, Lt=256, beta=4.0, mass=0.05,
             solver="CG", tol=1e-12),
        # dynamical staggered fermions
        dict(name="fermion_hmc_64x64", kind="fermion_hmc", Lx=64, Lt=64, beta=4.0, mass=0.1, n=6,
             traj=1),
        # what is measured after every trajectory, on a medium lattice
        dict(name="measure_16x16x16x16_fp64", kind="measure", Lx=16, Ly=16, Lz=16, Lt=16, nd=4,
             beta=2.4, precision="fp64", loop=4),
    ]


def draw(rng):
    def extent(lo, hi):  # an even extent, spread over its logarithm
        return 2 * round(math.exp(rng.uniform(math.log(lo / 2), math.log(hi / 2))))

    def lattice(nd, lo, hi):
        e = [extent(lo, hi) for _ in range(nd)]
        return dict(Lt=e[0], Lx=e[1], Ly=e[2] if nd > 2 else 1, Lz=e[3] if nd > 3 else 1, nd=nd)

    kind = rng.choice(["hmc", "hmc", "hmc", "batch", "metropolis", "metropolis", "flow",
                       "flow_gradient", "solve", "solve", "fermion_hmc", "measure"])
    precision = rng.choice(["fp64", "mixed"])
    beta = round(rng.uniform(2.2, 2.5), 3)
    if kind == "batch":
        return dict(kind=kind, chains=rng.randint(4, 40), shapes=rng.randrange(1 << 20),
                    precision=precision, n=rng.randint(5, 12), traj=2)
    if kind == "solve":
        return dict(kind=kind, Lx=extent(32, 256), Lt=extent(32, 256), beta=4.0,
                    mass=round(rng.uniform(0.05, 0.2), 3),
                    solver=rng.choice(["CG", "CG_mixed", "BiCGStab"]), tol=1e-12)
    if kind == "fermion_hmc":
        return dict(kind=kind, Lx=extent(16, 64), Lt=extent(16, 64), beta=4.0,
                    mass=round(rng.uniform(0.1, 0.3), 3), n=rng.randint(4, 6), traj=1)
    nd = rng.choice([3, 4, 4, 4])
    c = dict(kind=kind, **lattice(nd, 8, 48 if nd == 3 else 28), beta=beta, precision=precision)
    if kind == "hmc":
        integrator = rng.choice(["leapfrog", "omf2", "omf2"])
        c.update(integrator=integrator, n=rng.randint(6, 16), traj=rng.randint(2, 4),
                 accept=False)
    elif kind == "metropolis":
        # FP32 links take one decision in ten million another way when their staples round
        # another way: few updates keep two runs comparable
        mixed = precision == "mixed"
        c.update(delta=round(rng.uniform(0.1, 0.3), 3), hits=rng.randint(2, 10),
                 sweeps=1 if mixed else rng.randint(2, 10))
    elif kind == "flow":
        c.update(eps=rng.choice([0.01, 0.02]), records=rng.randint(5, 20))
    elif kind == "flow_gradient":
        c.update(eps=rng.choice([0.01, 0.02]), steps=rng.randint(5, 20))
    else:
        c.update(loop=rng.randint(2, 4))
    return c


# ---- inputs ------------------------------------------------------------------------------

def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _generator(seed):
    return torch.Generator(device=_device()).manual_seed(int(seed))


def _dims(c):
    return c["Lx"], c.get("Ly", 1), c.get("Lz", 1), c["Lt"]


def _sites(c):
    Lx, Ly, Lz, Lt = _dims(c)
    return Lx * Ly * Lz * Lt


def _su2_links(n, g):
    q = torch.randn(n, 4, generator=g, device=g.device, dtype=F64) * SPREAD
    q[:, 0] = 1.0
    return q / q.norm(dim=1, keepdim=True)


def _su2_field(c, seed):
    return _su2_links(_sites(c) * c["nd"], _generator(seed)).reshape(-1)


def _u1_field(c, seed):
    g = _generator(seed)
    return torch.randn(_sites(c) * 2, generator=g, device=g.device, dtype=F64) * 0.5


def _source(c, seed):
    g = _generator(seed + 1000003)
    return torch.randn(2 * _sites(c), generator=g, device=g.device, dtype=F64)


def _chains(c, seed):
    """The ensemble's chains: d = 4 with extents 4..12 and d = 3 with extents 8..24."""
    rng = np.random.default_rng(c["shapes"])
    out = []
    for i in range(c["chains"]):
        if rng.random() < 0.6:
            e, nd = 2 * rng.integers(2, 7, 4), 4
        else:
            e, nd = 2 * rng.integers(4, 13, 4), 3
            e[2] = 1
        out.append(dict(dims=tuple(int(v) for v in e), ndims=nd, beta=2.0 + 0.02 * i,
                        seed=seed + i))
    return out


def _buffer(n):
    return torch.empty(n, dtype=F64, pin_memory=torch.cuda.is_available())


def prepare(case, seed):
    c, kind = case, case["kind"]
    st = dict(c, seed=seed, count=0)
    if kind == "batch":
        chains = _chains(c, seed)
        b = chain_batch(chains, precision=c["precision"])
        g = _generator(seed)
        for i in range(len(chains)):
            b.upload(i, _su2_links(b.n_links(i), g).reshape(-1).cpu().numpy())
        b.autotune()
        st["lattice"] = b
        return st
    if kind in ("solve", "fermion_hmc"):
        precision = "mixed" if c.get("solver") == "CG_mixed" else "fp64"
        u = gaugeconfig(*_dims(c), 2, c["beta"], group="u1", precision=precision)
        u.upload(_u1_field(c, seed).cpu().numpy())
        if kind == "solve":
            st["b"] = _source(c, seed).cpu().numpy()
    else:
        u = gaugeconfig(*_dims(c), c["nd"], c["beta"], precision=c["precision"])
        u.upload(_su2_field(c, seed).cpu().numpy())
        if kind != "measure":
            u.autotune()  # once per run, as the driver's shim does after its upload
    st["lattice"] = u
    if kind in ("hmc", "metropolis", "fermion_hmc"):
        n = u.n_links * u.link_reals
        st["links"] = _buffer(n)  # the host copy that a save point writes to
        if c.get("precision") == "mixed":
            st["links32"] = torch.empty(n, dtype=torch.float32)
    return st


# ---- one pass ----------------------------------------------------------------------------

def _links(st):
    st["lattice"].download(st["links"].numpy())
    if "links32" in st:
        return st["links32"].copy_(st["links"])
    return st["links"]


def _numbers(st, rows):
    return np.asarray(rows, dtype=np.float32 if st.get("precision") == "mixed" else np.float64)


def _trajectories(st, u, **kw):
    H, accepted = [], []
    for _ in range(st["traj"]):
        r = u.md_update(n_steps=st["n"], tau=1.0, seed=st["seed"], traj=st["count"], **kw)
        st["count"] += 1
        H.append([*r.H_old, *r.H_new, r.plaquette])
        accepted.append(int(r.accepted))
    return dict(H=_numbers(st, H), accepted=np.asarray(accepted))


def run(state):
    st, u, kind = state, state["lattice"], state["kind"]
    if kind == "hmc":
        out = _trajectories(st, u, integrator=st["integrator"], accept_reject=st["accept"])
        return dict(out, links=_links(st))
    if kind == "fermion_hmc":
        out = _trajectories(st, u, integrator="omf2", fermion_mass=st["mass"], cg_tol=1e-10)
        return dict(out, links=_links(st))
    if kind == "batch":
        H, accepted = [], []
        for _ in range(st["traj"]):
            rs = u.md_update("leapfrog", st["n"], 1.0, traj=st["count"])
            st["count"] += 1
            H.append([[*r.H_old, *r.H_new, r.plaquette] for r in rs])
            accepted.append([int(r.accepted) for r in rs])
        links = [u.download(i) for i in range(st["chains"])]
        if st["precision"] == "mixed":
            links = [x.astype(np.float32) for x in links]
        return dict(H=_numbers(st, H), accepted=np.asarray(accepted), links=links)
    if kind == "metropolis":
        rates = []
        for _ in range(st["sweeps"]):
            rates.append(u.sweep(st["delta"], st["hits"], st["seed"], st["count"]))
            st["count"] += 1
        return dict(rates=np.asarray(rates), links=_links(st))
    if kind == "flow":
        # 2 steps per record; the end point half a step off the grid, clear of rounding
        tmax = (2 * st["records"] - 0.5) * st["eps"]
        return _numbers(st, u.gradient_flow(tmax, st["eps"], max_rows=st["records"] + 1))
    if kind == "flow_gradient":
        O, grad = u.flow_objective(st["eps"], st["steps"])
        return dict(objective=_numbers(st, [O]), grad=_numbers(st, grad))
    if kind == "solve":
        r = u.solve(st["b"], st["mass"], tol=st["tol"], solver=st["solver"], tol_mode="rel")
        return dict(x=r.x, converged=r.converged)
    E, Q = u.energy_density()
    return dict(plaquette=u.gauge_energy(), spatial=u.gauge_energy(True), E=E, Q=Q,
                polyakov=u.polyakov_loop_spatial_average(),
                loop=u.wilsonloop(st["loop"], st["loop"]))


# ---- what a pass cannot do without -------------------------------------------------------

def _force_work(V, nd, reals):
    """One fused force step: links in and out, momenta in and out; the 2(d-1) staples of each
    link (two quaternion products each), the force product, exp and the link product."""
    links = V * nd
    return links * (8 + 6) * reals, links * (2 * (nd - 1) * 64 + 64 + 40)


def _omf2_forces(c):
    return 2 * c["n"] + 1 if c.get("integrator", "omf2") == "omf2" else c["n"] + 1


def work(case):
    c, kind = case, case["kind"]
    if kind == "batch":
        by = fl = 0
        for ch in _chains(c, 0):
            Lx, Ly, Lz, Lt = ch["dims"]
            V = Lx * Ly * Lz * Lt
            b, f = _force_work(V, ch["ndims"], 4 if c["precision"] == "mixed" else 8)
            by += b * (c["n"] + 1) * c["traj"] + 32 * V * ch["ndims"]
            fl += f * (c["n"] + 1) * c["traj"]
        return dict(bytes=by, flops=fl)
    V = _sites(c)
    if kind == "solve":
        # source, links and solution once; per iteration two applications of the hopping term
        # (16 complex multiply-adds a site) and the vector updates
        iterations = 4.5 / c["mass"] * math.log(1 / c["tol"]) / 2.3
        return dict(bytes=V * (16 + 16 + 16), flops=V * iterations * 180)
    if kind == "fermion_hmc":
        iterations = 4.5 / c["mass"] * 6
        return dict(bytes=V * (2 * 16 + 48), flops=V * iterations * 180 * _omf2_forces(c))
    nd, reals = c["nd"], 4 if c["precision"] == "mixed" else 8
    by, fl = _force_work(V, nd, reals)
    host = V * nd * 32
    if kind == "hmc":
        k = c["traj"] * _omf2_forces(c)
        return dict(bytes=k * by + host, flops=k * fl)
    if kind == "metropolis":
        # every pass over one direction and parity reads the field and writes its links
        per = V * nd * 4 * reals * 2
        hit = V * nd * (2 * (nd - 1) * 64 + c["hits"] * 120)
        return dict(bytes=c["sweeps"] * per + host, flops=c["sweeps"] * hit)
    plaq = V * nd * (nd - 1) / 2 * 100
    clover = V * nd * (nd - 1) / 2 * 4 * 100
    if kind == "flow":
        steps = 2 * c["records"]
        return dict(bytes=3 * steps * by + c["records"] * 2 * V * nd * 4 * reals,
                    flops=3 * steps * fl + c["records"] * (plaq + clover))
    if kind == "flow_gradient":
        # forward once, every stage again in the backward sweep, its adjoint twice a force
        k = 3 * c["steps"]
        return dict(bytes=3 * k * by + V * nd * 24, flops=4 * k * fl)
    loops = V * (nd - 1) * 4 * c["loop"] * 28
    return dict(bytes=5 * V * nd * 4 * reals, flops=2 * plaq + clover + loops)


# ---- the same in 64 bits with torch alone ------------------------------------------------
# An SU(2) field is a list over directions of lists of four tensors [T, X, Y, Z]: a link is
# [[a, b], [-b*, a*]] with (Re a, Im a, Re b, Im b).

def _mul(u, v):
    return [u[0] * v[0] - u[1] * v[1] - u[2] * v[2] - u[3] * v[3],
            u[0] * v[1] + u[1] * v[0] + u[2] * v[3] - u[3] * v[2],
            u[0] * v[2] - u[1] * v[3] + u[2] * v[0] + u[3] * v[1],
            u[0] * v[3] + u[1] * v[2] - u[2] * v[1] + u[3] * v[0]]


def _dag(u):
    return [u[0], -u[1], -u[2], -u[3]]


def _shift(u, mu, s):
    """u at x + s mu."""
    return [torch.roll(a, -s, mu) for a in u]


def _unpack(flat, dims, nd):
    Lx, Ly, Lz, Lt = dims
    a = flat.reshape(Lt, Lx, Ly, Lz, nd, -1)
    return [[a[..., mu, k].contiguous() for k in range(a.shape[-1])] for mu in range(nd)]


def _pack(U):
    return torch.stack([torch.stack(u, -1) for u in U], -2).reshape(-1)


def _restore(U):
    out = []
    for u in U:
        r = torch.sqrt(sum(a * a for a in u))
        out.append([a / r for a in u])
    return out


def _exp(x):
    """exp of the algebra element with components x (each a tensor)."""
    t = torch.sqrt(sum(a * a for a in x))
    s = torch.sinc(t / math.pi)
    return [torch.cos(t), s * x[2], s * x[1], s * x[0]]


def _staples(U, mu, site=None):
    nd, K = len(U), None
    for nu in range(nd):
        if nu == mu:
            continue
        up = _mul(_mul(_shift(U[nu], mu, 1), _dag(_shift(U[mu], nu, 1))), _dag(U[nu]))
        dn = _shift(_mul(_mul(_dag(_shift(U[nu], mu, 1)), _dag(U[mu])), U[nu]), nu, -1)
        both = [a + b for a, b in zip(up, dn)]
        K = both if K is None else [a + b for a, b in zip(K, both)]
    return K


def _force(U, f):
    out = []
    for mu in range(len(U)):
        w = _mul(U[mu], _staples(U, mu))
        out.append([2 * f * w[3], 2 * f * w[2], 2 * f * w[1]])
    return out


def _plaquettes(U):
    """ReTr summed over sites: all planes, and the planes without direction 0."""
    full = spatial = 0.0
    for mu in range(len(U) - 1):
        for nu in range(mu + 1, len(U)):
            w = _mul(_mul(U[mu], _shift(U[nu], mu, 1)),
                     _dag(_mul(U[nu], _shift(U[mu], nu, 1))))
            s = 2 * w[0].sum()
            full = full + s
            if mu:
                spatial = spatial + s
    return full, spatial


def _clover(U):
    """(E over all planes, E over spatial planes, Q) of the clover definition, per site."""
    nd, V = len(U), U[0][0].numel()
    G, e, es = {}, 0.0, 0.0
    for mu in range(nd - 1):
        for nu in range(mu + 1, nd):
            a, b = U[mu], U[nu]
            p = _mul(_mul(a, _shift(b, mu, 1)), _dag(_mul(b, _shift(a, nu, 1))))
            # the other leaves are the plaquettes of the other corners, carried to x
            q = _shift(_mul(_mul(_dag(a), p), a), mu, -1)
            r = _shift(_mul(_mul(_dag(b), p), b), nu, -1)
            g = [w + x + y + z for w, x, y, z in zip(p, q, r, _corner(a, b, p, mu, nu))]
            g[0] = torch.zeros_like(g[0])
            G[mu, nu] = g
            t = 2 * (-(g[1] ** 2 + g[2] ** 2 + g[3] ** 2)).sum()
            e = e + t
            if mu:
                es = es + t
    Q = 0.0
    if nd == 4:
        def tr(x, y):
            return 2 * (-(x[1] * y[1] + x[2] * y[2] + x[3] * y[3])).sum()
        Q = 2 * (tr(G[0, 1], G[2, 3]) - tr(G[0, 2], G[1, 3]) + tr(G[0, 3], G[1, 2]))
    E, Es = -e / V / 16, -es / V / 16
    return float(E), float(Es), float(-4 * Q / (32 * math.pi ** 2) / 16)


def _corner(a, b, p, mu, nu):
    """The leaf U_mu(x-mu)^+ U_nu(x-mu-nu)^+ U_mu(x-mu-nu) U_nu(x-nu)."""
    am, bn = _shift(a, mu, -1), _shift(b, nu, -1)
    amn, bmn = _shift(am, nu, -1), _shift(bn, mu, -1)
    return _mul(_mul(_dag(am), _dag(bmn)), _mul(amn, bn))


# Philox4x32-10 in int64 tensors
_M32 = 0xFFFFFFFF


def _philox(c0, c1, c2, c3, seed):
    k0, k1 = seed & _M32, (seed >> 32) & _M32
    c1, c2, c3 = (torch.full_like(c0, v) if not torch.is_tensor(v) else v for v in (c1, c2, c3))

    def wide(m, c):  # 32 x 32 -> (high, low)
        lo, hi = c & 0xFFFF, c >> 16
        a, b = m * lo, m * hi
        t = (a >> 16) + (b & 0xFFFF)
        return ((b >> 16) + (t >> 16)) & _M32, (a + (b << 16)) & _M32

    for _ in range(10):
        h0, l0 = wide(0xD2511F53, c0)
        h1, l1 = wide(0xCD9E8D57, c2)
        c0, c1, c2, c3 = h1 ^ c1 ^ k0, l1, h0 ^ c3 ^ k1, l0
        k0, k1 = (k0 + 0x9E3779B9) & _M32, (k1 + 0xBB67AE85) & _M32
    return c0, c1, c2, c3


def _u53(hi, lo):
    return (((hi << 21) ^ (lo >> 11)).to(F64) + 1.0) * 2.0 ** -53


def _normals(index, draw_, step, tag, seed):
    r = _philox(index, draw_, step, tag, seed)
    rad = torch.sqrt(-2 * torch.log(_u53(r[0], r[1])))
    a = 2 * math.pi * _u53(r[2], r[3])
    return rad * torch.cos(a), rad * torch.sin(a)


def _momenta(dims, nd, comps, seed, traj):
    Lx, Ly, Lz, Lt = dims
    V = Lx * Ly * Lz * Lt
    lex = torch.arange(V, device=_device(), dtype=torch.int64)
    P = []
    for mu in range(nd):
        n0, n1 = _normals(lex * nd + mu, 0, traj, 0x4D4F4D31, seed)
        n = [n0]
        if comps == 3:
            n += [n1, _normals(lex * nd + mu, 1, traj, 0x4D4F4D31, seed)[0]]
        P.append([a.reshape(Lt, Lx, Ly, Lz) for a in n])
    return P


def _accepts(dH, traj, seed):
    if dH <= 0:
        return True
    z = torch.zeros(1, dtype=torch.int64)
    r = _philox(z, 0, traj, 0x41434331, seed)
    return float(_u53(r[0], r[1])) - 2.0 ** -53 <= math.exp(-dH)


def _schedule(integrator, n):
    """(momentum coefficient, gauge coefficient) of each fused step; the last has no gauge."""
    dt = 1.0 / n
    if integrator == "leapfrog":
        m, g = [dt / 2] + [dt] * (n - 1) + [dt / 2], dt
    else:
        lam = 0.1938
        m, g = [lam * dt], 0.5 * dt
        for _ in range(n - 1):
            m += [(1 - 2 * lam) * dt, 2 * lam * dt]
        m += [(1 - 2 * lam) * dt, lam * dt]
    return [(c, g if i + 1 < len(m) else None) for i, c in enumerate(m)]


def _kinetic(P):
    return 0.5 * float(sum((a * a).sum() for p in P for a in p))


def _su2_trajectory(U, dims, beta, seed, traj, integrator, n, accept):
    P = _momenta(dims, len(U), 3, seed, traj)
    plaq = float(_plaquettes(U)[0])
    old = [_kinetic(P), -beta / 2 * plaq, 0.0]
    W = U
    for cm, cg in _schedule(integrator, n):
        F = _force(W, beta / 2)
        P = [[a - cm * b for a, b in zip(p, f)] for p, f in zip(P, F)]
        if cg is not None:
            W = [_mul(_exp([cg * a for a in p]), w) for p, w in zip(P, W)]
    W = _restore(W)
    plaq_new = float(_plaquettes(W)[0])
    new = [_kinetic(P), -beta / 2 * plaq_new, 0.0]
    ok = not accept or _accepts(sum(new) - sum(old), traj, seed)
    return (W if ok else U), [*old, *new, plaq_new if ok else plaq], int(ok)


def _exact_hmc(c, seed):
    U, H, acc = _unpack(_su2_field(c, seed), _dims(c), c["nd"]), [], []
    for t in range(c["traj"]):
        U, h, a = _su2_trajectory(U, _dims(c), c["beta"], seed, t, c["integrator"], c["n"],
                                  c["accept"])
        H.append(h)
        acc.append(a)
    return dict(H=np.asarray(H), accepted=None, links=_pack(U))


def _exact_batch(c, seed):
    g, H, links = _generator(seed), [], []
    for ch in _chains(c, seed):
        Lx, Ly, Lz, Lt = ch["dims"]
        U = _unpack(_su2_links(Lx * Ly * Lz * Lt * ch["ndims"], g).reshape(-1), ch["dims"],
                    ch["ndims"])
        rows = []
        for t in range(c["traj"]):
            U, h, _ = _su2_trajectory(U, ch["dims"], ch["beta"], ch["seed"], t, "leapfrog",
                                      c["n"], True)
            rows.append(h)
        H.append(rows)
        links.append(_pack(U))
    return dict(H=np.asarray(H).transpose(1, 0, 2).copy(), accepted=None, links=links)


def _exact_metropolis(c, seed):
    if c["precision"] == "mixed":
        return None  # its accept decisions are those of FP32 proposals
    dims, nd, V = _dims(c), c["nd"], _sites(c)
    Lx, Ly, Lz, Lt = dims
    U = _unpack(_su2_field(c, seed), dims, nd)
    lex = torch.arange(V, device=_device(), dtype=torch.int64).reshape(Lt, Lx, Ly, Lz)
    par = sum(torch.meshgrid(*[torch.arange(L, device=_device()) for L in (Lt, Lx, Ly, Lz)],
                             indexing="ij")) % 2
    rates = []
    for sweep in range(c["sweeps"]):
        count, temporal = 0, 0
        for mu in range(nd):
            for p in range(2):
                at = (par == p).reshape(-1).nonzero()[:, 0]
                K = [a.reshape(-1)[at] for a in _staples(U, mu)]
                u = [a.reshape(-1)[at] for a in U[mu]]
                link = lex.reshape(-1)[at] * nd + mu
                for hit in range(c["hits"]):
                    r = [x.to(F64) * 2.0 ** -32
                         for x in _philox(link, hit, sweep, 0x4D455431, seed)]
                    al, z, th = 2 * math.pi * c["delta"] * r[0], 2 * r[1] - 1, 2 * math.pi * r[2]
                    rho = torch.sqrt(1 - z * z)
                    sa = torch.sin(al)
                    v = _mul(u, [torch.cos(al), sa * z, sa * rho * torch.sin(th),
                                 sa * rho * torch.cos(th)])
                    dS = c["beta"] / 2 * 2 * (_mul(u, K)[0] - _mul(v, K)[0])
                    ok = (dS < 0) | (r[3] < torch.exp(-dS))
                    u = [torch.where(ok, a, b) for a, b in zip(_restore([v])[0], u)]
                    k = int(ok.sum())
                    count += k
                    temporal += k if mu == 0 else 0
                for a, b in zip(U[mu], u):
                    a.view(-1)[at] = b
        rates.append([count / c["hits"] / (V * nd), temporal / c["hits"] / V])
    return dict(rates=np.asarray(rates), links=_pack(U))


_Z = (-17 / 36, 8 / 9, -3 / 4)
_E = (-36 / 4 / 17, 1.0, -1.0)


def _flow_stage(W, Z, eps, f):
    F = _force(W, 2 * _Z[f])
    Z = F if Z is None else [[a + b for a, b in zip(z, x)] for z, x in zip(Z, F)]
    W = [_mul(_exp([-eps * _E[f] * a for a in z]), w) for z, w in zip(Z, W)]
    return W, Z


def _exact_flow(c, seed):
    nd, V = c["nd"], _sites(c)
    W, rows = _unpack(_su2_field(c, seed), _dims(c), nd), []
    for k in range(2 * c["records"]):
        Z = None
        for f in range(3):
            W, Z = _flow_stage(W, Z, c["eps"], f)
        if k % 2 == 0:
            P, Ps = (float(v) / (2 * V) for v in _plaquettes(W))
            E, Es, Q = _clover(W)
            nf, ns = nd * (nd - 1) / 2, (nd - 1) * (nd - 2) / 2
            Ep, Eps = nf - P, ns - Ps
            rows.append([(k + 1) * c["eps"], math.sqrt((Ep - Eps) / (nd - 1) / (Eps / ns)), P, Ps,
                         Ep, Eps, E, Es, Q])
    return np.asarray(rows)


def _exact_flow_gradient(c, seed):
    nd, V = c["nd"], _sites(c)
    U = [[a.requires_grad_() for a in u] for u in _unpack(_su2_field(c, seed), _dims(c), nd)]

    def stage(f, *flat):
        W = [list(flat[4 * m:4 * m + 4]) for m in range(nd)]
        z = flat[4 * nd:]
        Z = [list(z[3 * m:3 * m + 3]) for m in range(nd)] if z else None
        W, Z = _flow_stage(W, Z, c["eps"], f)
        return tuple(a for w in W for a in w) + tuple(a for z in Z for a in z)

    flat = tuple(a for u in U for a in u)
    for _ in range(c["steps"]):
        for f in range(3):
            flat = checkpoint(stage, f, *(flat if f else flat[:4 * nd]), use_reentrant=False)
    W = [list(flat[4 * m:4 * m + 4]) for m in range(nd)]
    t = c["steps"] * c["eps"]
    O = t * t * (nd * (nd - 1) / 2 - _plaquettes(W)[0] / (2 * V))
    O.backward()
    grad = []
    with torch.no_grad():
        for u in U:
            row = []
            for k in (3, 2, 1):  # the generator of each component of the algebra
                e = [torch.zeros_like(u[0]) for _ in range(4)]
                e[k] += 1
                row.append(sum(a.grad * b for a, b in zip(u, _mul(e, u))))
            grad.append(row)
        return dict(objective=np.asarray([float(O)]), grad=_pack(grad))


def _staggered(c, th):
    """psi -> hop(psi) and the plaquette force's pieces on angles th[mu][T, X]."""
    ph = [torch.polar(torch.ones_like(a), a) for a in th]
    eta = [torch.ones_like(th[0]), torch.ones_like(th[0])]
    eta[1][1::2] = -1

    def hop(v):
        o = 0
        for mu in range(2):
            o = o + 0.5 * eta[mu] * (ph[mu] * torch.roll(v, -1, mu)
                                     - torch.roll(ph[mu].conj() * v, 1, mu))
        return o

    return hop, ph, eta


def _invert(hop, m, b, tol=1e-14):
    """(D D^+)^-1 b by CG with restarts on the true residual."""
    def A(v):
        w = m * v - hop(v)
        return m * w + hop(w)

    x, best = torch.zeros_like(b), None
    bn = float(b.abs().square().sum().sqrt())
    for _ in range(3):
        r = b - A(x)
        p, rr = r, r.abs().square().sum()
        for k in range(8000):
            w = m * p - hop(p)
            q = m * w + hop(w)
            al = rr / w.abs().square().sum()
            x, r = x + al * p, r - al * q
            new = r.abs().square().sum()
            if k % 20 == 0 and float(new) <= (tol * bn) ** 2:
                break
            p, rr = r + (new / rr) * p, new
        best = float((b - A(x)).abs().square().sum().sqrt()) / bn
        if best < 4 * tol:
            break
    return x


def _u1_angles(flat, c):
    a = flat.reshape(c["Lt"], c["Lx"], 2)
    return [a[..., 0].contiguous(), a[..., 1].contiguous()]


def _exact_solve(c, seed):
    hop, _, _ = _staggered(c, _u1_angles(_u1_field(c, seed), c))
    b = torch.view_as_complex(_source(c, seed).reshape(c["Lt"], c["Lx"], 2))
    m = c["mass"]
    x = _invert(hop, m, b)
    if c["solver"] == "BiCGStab":  # D x = b: x = D^+ (D D^+)^-1 b
        x = m * x - hop(x)
    return dict(x=torch.view_as_real(x).reshape(-1), converged=None)


def _u1_plaquettes(th):
    return torch.cos(th[0] + torch.roll(th[1], -1, 0) - torch.roll(th[0], -1, 1) - th[1])


def _exact_fermion_hmc(c, seed):
    m, beta, dims = c["mass"], c["beta"], _dims(c)
    th, H = _u1_angles(_u1_field(c, seed), c), []
    V = _sites(c)
    lex = torch.arange(V, device=_device(), dtype=torch.int64)
    for traj in range(c["traj"]):
        P = [p[0].reshape(c["Lt"], c["Lx"]) for p in _momenta(dims, 2, 1, seed, traj)]
        R = (_normals(lex, 0, traj, 0x50465331, seed)[0] * math.sqrt(0.5)).reshape(c["Lt"], c["Lx"])
        hop, _, _ = _staggered(c, th)
        R = R.to(torch.complex128)
        phi = m * R + hop(R)
        plaq = float(_u1_plaquettes(th).sum())
        old = [0.5 * float(sum((p * p).sum() for p in P)), -beta * plaq,
               float(R.abs().square().sum())]
        w = th
        for cm, cg in _schedule("omf2", c["n"]):
            hop, ph, eta = _staggered(c, w)
            chi = _invert(hop, m, phi)
            chi1 = m * chi - hop(chi)
            s = torch.sin(w[0] + torch.roll(w[1], -1, 0) - torch.roll(w[0], -1, 1) - w[1])
            F = [beta * (s - torch.roll(s, 1, 1)), beta * (torch.roll(s, 1, 0) - s)]
            for mu in range(2):
                vp = 0.5j * eta[mu] * ph[mu] * torch.roll(chi1, -1, mu)
                vx = 0.5j * eta[mu] * ph[mu].conj() * chi1
                d = chi.conj() * vp + torch.roll(chi, -1, mu).conj() * vx
                F[mu] = F[mu] - 2 * d.real
            P = [p - cm * f for p, f in zip(P, F)]
            if cg is not None:
                w = [a + cg * p for a, p in zip(w, P)]
        hop, _, _ = _staggered(c, w)
        plaq_new = float(_u1_plaquettes(w).sum())
        new = [0.5 * float(sum((p * p).sum() for p in P)), -beta * plaq_new,
               float((phi.conj() * _invert(hop, m, phi)).real.sum())]
        ok = _accepts(sum(new) - sum(old), traj, seed)
        th = w if ok else th
        H.append([*old, *new, plaq_new if ok else plaq])
    return dict(H=np.asarray(H), accepted=None, links=torch.stack(th, -1).reshape(-1))


def _exact_measure(c, seed):
    nd, V = c["nd"], _sites(c)
    U = _unpack(_su2_field(c, seed), _dims(c), nd)
    P, Ps = _plaquettes(U)
    E, _, Q = _clover(U)
    line = [a[0] for a in U[0]]
    for t in range(1, c["Lt"]):
        line = _mul(line, [a[t] for a in U[0]])
    loops, n = 0.0, c["loop"]

    def straight(mu):
        w = U[mu]
        for k in range(1, n):
            w = _mul(w, _shift(U[mu], mu, k))
        return w

    t = straight(0)
    for mu in range(1, nd):
        s = straight(mu)
        w = _mul(_mul(t, _shift(s, 0, n)), _dag(_mul(s, _shift(t, mu, n))))
        loops = loops + 2 * w[0].sum()
    return dict(plaquette=float(P), spatial=float(Ps), E=E, Q=Q,
                polyakov=2 * float(line[0].sum()) / V, loop=float(loops) / (V * 2 * nd))


def exact(case, seed):
    with torch.enable_grad() if case["kind"] == "flow_gradient" else torch.no_grad():
        return dict(hmc=_exact_hmc, batch=_exact_batch, metropolis=_exact_metropolis,
                    flow=_exact_flow, flow_gradient=_exact_flow_gradient, solve=_exact_solve,
                    fermion_hmc=_exact_fermion_hmc, measure=_exact_measure)[case["kind"]](case,
                                                                                         seed)
