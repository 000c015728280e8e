"""The work that users of this library have it do, as cases that can be timed and compared.

Six kinds of work, each a call sequence of a lattice program through the public entry points:

* ``update``   a generation run: rounds of heatbath and overrelaxation sweeps, the plaquette, and
  the configuration taken out (lt_download_links into the program's pinned buffer, as before
  writing it to disk);
* ``flow``     a gradient flow (Wilson, Luescher-Weisz or Zeuthen force) of a configuration with
  the plaquette, the clover charge and the energy density every few steps;
* ``hmc``      the molecular dynamics of an HMC trajectory, Hamiltonian before and after;
* ``metad``    the same with the metadynamics bias on the smeared clover charge;
* ``analysis`` a stored configuration uploaded and put through the reference driver's measurement
  bundle on several levels of Euler flow;
* ``ensemble`` rounds of sweeps on many small lattices of different extents at once.

Inputs are drawn on the GPU from the seed: links g(x) exp(i s H) g(x+mu)^dag with Gaussian H and
random gauge rotations g, at the spread s where the plaquette is that of a thermalised
configuration at beta = 6 (0.59), and Gaussian momenta.  They do not come from the library's own
heatbath, so they stay the same whatever its kernels do.

Sweeps are chaotic: a difference of one rounding grows two- to fourfold with every sweep (measured:
1e-7 in a link is 1e-3 after eight overrelaxation sweeps in FP32, 2e-16 is of order one after forty
sweeps in FP64), and an FP32 heatbath proposal within rounding of the accept threshold is
taken by one correct implementation and refused by another.  With the Wilson action, where a staple
is six fixed products summed in a fixed order, a seeded chain is therefore reproduced bit for bit.
With the rectangle actions, whose longer paths can be multiplied out in many orders, passes are kept
short enough to be compared, and the heatbath runs in FP64 (the reference's own precision).
"""
import math

import numpy as np
import torch

import lettuce_b200 as lt

BETA = 6.0
SPREAD = 0.445
LW = (1.0 + 8.0 / 12.0, -1.0 / 12.0)
IWASAKI = (1.0 + 8.0 * 0.331, -0.331)
RHO = 0.12


# ---------------------------------------------------------------- the cases
def _case(name, kind, ext, prec, **more):
    return {"name": name, "kind": kind, "nt": ext[0], "nx": ext[1], "ny": ext[2], "nz": ext[3], "prec": prec, **more}


def listed():
    return [
        # the plain method of the reference at its smallest size: 20 rounds on an 8^4 lattice
        # in FP64; 800 dependent launches of 2048 links, all latency
        _case("update_small_fp64", "update", (8, 8, 8, 8), "fp64", action="wilson", colours=2, rounds=20, n_hb=1, n_or=4),
        # the bulk workload: 10 rounds of 1 heatbath + 4 overrelaxation sweeps at 32^4 on the
        # compressed links (the bench's lattice and storage)
        _case("update_bulk_fp32_12", "update", (32, 32, 32, 32), "fp32_12", action="wilson", colours=2, rounds=10, n_hb=1, n_or=4),
        # the same in the reference's precision on an ordinary finite-temperature-like box
        _case("update_fp64", "update", (16, 24, 24, 24), "fp64", action="wilson", colours=2, rounds=8, n_hb=1, n_or=4),
        # the reference driver's own update loop: Checkerboard4 with the Symanzik action, FP64
        _case("update_lw_fp64", "update", (16, 16, 16, 16), "fp64", action="lw", colours=4, rounds=4, n_hb=1, n_or=4),
        # flow to t = 2 with the charge every 0.1 on the small lattice, FP64
        _case("flow_small_fp64", "flow", (8, 8, 8, 8), "fp64", action="wilson", eps=0.01, n_meas=20, every=10),
        # the bulk flow: 40 RK3 steps at 32^4 on the compressed links
        _case("flow_bulk_fp32_12", "flow", (32, 32, 32, 32), "fp32_12", action="wilson", eps=0.01, n_meas=4, every=10),
        # the improved flow on the way to t0, measured after every step as the scale setting does
        _case("flow_zeuthen_fp32_12", "flow", (48, 24, 24, 24), "fp32_12", action="zeuthen", eps=0.01, n_meas=8, every=1),
        # one long trajectory's dynamics of the large HMC run: 48^4, tau = 2 in 40 Omelyan steps
        _case("hmc_large_fp32_12", "hmc", (48, 48, 48, 48), "fp32_12", action="wilson", integrator="OMF_2", tau=2.0, n_step=40),
        # HMC with the improved action on an ordinary lattice, the reference driver's integrator
        _case("hmc_lw_fp32", "hmc", (24, 20, 20, 20), "fp32", action="lw", integrator="OMF_4", tau=0.5, n_step=4),
        # metadynamics: 16^4, four stout levels, tau = 1 in 10 Omelyan steps (21 adjoint forces)
        _case("metad_fp32_12", "metad", (16, 16, 16, 16), "fp32_12", integrator="OMF_2", tau=1.0, n_step=10, n_stout=4),
        # measurements on a stored 32 x 24^3 configuration and two levels of Euler flow above it
        _case("analysis_fp64", "analysis", (32, 24, 24, 24), "fp64", n_smear=2, smear_skip=10, eps=0.02),
        # tempering streams of 12^4 with independent chains of uneven extents beside them
        _case("ensemble_fp32_12", "ensemble", (12, 12, 12, 12), "fp32_12", n_streams=8, n_chains=40, pick=5, rounds=10),
    ]


def _extents(rng, lo, hi, step=2):
    """Four extents, multiples of `step`, whose volume is log-uniform over [lo^4, hi^4]."""
    base = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    while True:
        e = [max(4, step * round(base * 2.0 ** rng.uniform(-0.45, 0.45) / step)) for _ in range(4)]
        if lo ** 4 / 2 <= math.prod(e) <= hi ** 4:
            return e


def draw(rng):
    kind = rng.choice(["update", "update", "flow", "flow", "hmc", "metad", "analysis", "ensemble"])
    if kind == "update":
        colours = rng.choice([2, 2, 4])
        action = "wilson" if colours == 2 else rng.choice(["wilson", "lw", "iwasaki"])
        prec = rng.choice(["fp64", "fp32", "fp32_12"])
        rect = action != "wilson"
        n_hb = 0 if rect and prec != "fp64" else rng.choice([0, 1, 1, 2])
        e = _extents(rng, 4, 24 if rect else 32, 4 if colours == 4 else 2)
        n_or = rng.randint(0 if n_hb else 1, 4 if prec == "fp64" or not rect else 2)
        most = 10 if not rect else 3 if n_hb else 1
        c = _case("", kind, e, prec, action=action, colours=colours, rounds=rng.randint(1, most), n_hb=n_hb, n_or=n_or)
    elif kind == "flow":
        action = rng.choice(["wilson", "wilson", "lw", "zeuthen"])
        prec = rng.choice(["fp64", "fp32", "fp32_12", "fp32_12"])
        e = _extents(rng, 6, 32 if action == "wilson" else 24)
        every = rng.randint(1, 8)
        c = _case("", kind, e, prec, action=action, eps=rng.choice([0.005, 0.01, 0.02]), n_meas=rng.randint(1, 4), every=every)
    elif kind == "hmc":
        action = rng.choice(["wilson", "lw", "iwasaki"])
        prec = rng.choice(["fp64", "fp32", "fp32_12"])
        e = _extents(rng, 6, 32 if action == "wilson" else 20)
        c = _case("", kind, e, prec, action=action, integrator=rng.choice(["Leapfrog", "OMF_2", "OMF_4"]),
                  tau=rng.choice([0.25, 0.5]), n_step=rng.randint(3, 6))
    elif kind == "metad":
        e = _extents(rng, 6, 16)
        c = _case("", kind, e, rng.choice(["fp64", "fp32", "fp32_12"]), integrator=rng.choice(["Leapfrog", "OMF_2"]),
                  tau=0.25, n_step=rng.randint(2, 5), n_stout=rng.randint(1, 6))
    elif kind == "analysis":
        e = _extents(rng, 8, 28)
        c = _case("", kind, e, rng.choice(["fp64", "fp32", "fp32_12"]), n_smear=rng.randint(0, 3),
                  smear_skip=rng.randint(1, 10), eps=rng.choice([0.01, 0.02]))
    else:
        l = rng.choice([6, 8, 10, 12])
        c = _case("", kind, (l, l, l, l), rng.choice(["fp32", "fp32_12", "fp64"]), n_streams=rng.randint(1, 8),
                  n_chains=rng.randint(2, 24), pick=rng.randrange(1000), rounds=rng.randint(1, 6))
    del c["name"]
    return c


def _ext(case):
    return case["nt"], case["nx"], case["ny"], case["nz"]


def _ensemble_extents(case):
    """The streams' common extents, then chains with extents from {8, 10, 12, 14, 16}."""
    r = np.random.RandomState(case["pick"])
    return [_ext(case)] * case["n_streams"] + [(int(l),) * 4 for l in r.choice([8, 10, 12, 14, 16], case["n_chains"])]


# ---------------------------------------------------------------- inputs
_LAMBDA = None


def _generators():
    """The eight SU(3) generators lambda_a / 2 on the GPU."""
    global _LAMBDA
    if _LAMBDA is None:
        g = np.zeros((8, 3, 3), complex)
        g[0][0, 1] = g[0][1, 0] = 1
        g[1][0, 1], g[1][1, 0] = -1j, 1j
        g[2][0, 0], g[2][1, 1] = 1, -1
        g[3][0, 2] = g[3][2, 0] = 1
        g[4][0, 2], g[4][2, 0] = -1j, 1j
        g[5][1, 2] = g[5][2, 1] = 1
        g[6][1, 2], g[6][2, 1] = -1j, 1j
        g[7] = np.diag([1, 1, -2]) / math.sqrt(3)
        _LAMBDA = torch.from_numpy(g / 2).cuda()
    return _LAMBDA


def _mm(a, b):
    """Products of batches of 3x3 complex matrices, summed in ascending inner index."""
    r = a[..., :, 0:1] * b[..., 0:1, :]
    r += a[..., :, 1:2] * b[..., 1:2, :]
    r += a[..., :, 2:3] * b[..., 2:3, :]
    return r


def _dag(a):
    return a.conj().transpose(-1, -2)


def _expm(x):
    """exp of anti-Hermitian 3x3 matrices of norm up to about one: 20 Taylor terms."""
    one = torch.eye(3, dtype=x.dtype, device=x.device)
    r = one + x / 20
    for n in range(19, 0, -1):
        r = one + _mm(x, r) / n
    return r


def _gaussian_algebra(gen, ext):
    """i phi_a lambda_a / 2 with unit Gaussians phi, one per site."""
    phi = torch.randn((*ext, 8), generator=gen, device="cuda", dtype=torch.float64)
    return 1j * torch.einsum("...a,aij->...ij", phi.to(torch.complex128), _generators())


def _random_links(ext, seed):
    """Four fields [T, X, Y, Z, 3, 3] of links with a thermalised plaquette in a random gauge."""
    gen = torch.Generator("cuda").manual_seed(int(seed))
    g = torch.view_as_complex(torch.randn((*ext, 3, 3, 2), generator=gen, device="cuda", dtype=torch.float64))
    a = g[..., 0, :] / g[..., 0, :].norm(dim=-1, keepdim=True)
    b = g[..., 1, :] - (a.conj() * g[..., 1, :]).sum(-1, keepdim=True) * a
    b = b / b.norm(dim=-1, keepdim=True)
    g = torch.stack([a, b, torch.linalg.cross(a, b).conj()], dim=-2)
    return [_mm(_mm(g, _expm(SPREAD * _gaussian_algebra(gen, ext))), _dag(torch.roll(g, -1, d))) for d in range(4)]


def _random_momenta(ext, seed):
    gen = torch.Generator("cuda").manual_seed(int(seed) + 7_000_003)
    return [_gaussian_algebra(gen, ext) for _ in range(4)]


def _to_host(fields):
    """Fields by direction -> pinned host array double[V][4][3][3][2]."""
    a = torch.view_as_real(torch.stack(fields, dim=4)).reshape(-1, 4, 3, 3, 2)
    h = torch.empty(a.shape, dtype=torch.float64, pin_memory=True)
    return h.copy_(a)


def _to_fields(host, ext):
    a = torch.view_as_complex(torch.as_tensor(host).cuda().reshape(*ext, 4, 3, 3, 2))
    return [a[..., d, :, :].contiguous() for d in range(4)]


# ---------------------------------------------------------------- what a program keeps
def _action(name):
    return {"wilson": lt.WilsonAction, "lw": lt.LuescherWeiszAction, "iwasaki": lt.IwasakiAction}[name](BETA)


def _bias_grid():
    """A filled bias potential: 3200 bins over [-32, 32] with wells at the integers."""
    q = np.linspace(-32.0, 32.0, 3201)
    return 2.0 * (1.0 - np.cos(2.0 * np.pi * q)) + 0.05 * q * q


def _field(ext, prec, host):
    u = lt.GaugeField(ext, prec)
    u.upload(host.numpy())
    return u


def prepare(case, seed):
    ext, kind, prec = _ext(case), case["kind"], case["prec"]
    s = {"case": dict(case), "ext": ext}
    if kind == "ensemble":
        sizes = _ensemble_extents(case)
        s["U"] = [_field(e, prec, _to_host(_random_links(e, seed + 1000 * k))) for k, e in enumerate(sizes)]
        s["out"] = [torch.empty((math.prod(e), 4, 3, 3, 2), dtype=torch.float64, pin_memory=True) for e in sizes]
        s["ensemble"] = lt.Ensemble(s["U"], np.linspace(5.8, 6.2, len(sizes)), seed=seed % 1000 + 1)
        return s
    host = _to_host(_random_links(ext, seed))
    if kind == "analysis":
        s["host"] = host
        s["U"] = lt.GaugeField(ext, prec)
        return s
    s["U"] = _field(ext, prec, host)
    s["out"] = host   # the program's pinned buffer: its input, then what it takes out
    if kind == "update":
        s["counter"], s["seed"] = 0, seed % 1000 + 1
    elif kind == "flow":
        action = lt.ZeuthenFlow() if case["action"] == "zeuthen" else _action(case["action"])
        s["V"] = lt.GaugeField(ext, prec)
        s["kernel"] = lt.GradientFlowKernel(s["U"], s["V"], lt.RK3, action, case["eps"])
    else:
        integ = getattr(lt.Integrators.HMC, case["integrator"])
        if kind == "hmc":
            s["kernel"] = lt.HMCKernel(s["U"], _action(case["action"]), case["tau"], integrator=integ)
        else:
            bias = lt.MetaBiasPotential(-32, 32, 3200, 0.05, 0.08, 10, 1000)
            bias.set_grid(_bias_grid())
            s["kernel"] = lt.HMCMetaDKernel(s["U"], bias, lt.WilsonAction(BETA), case["tau"], RHO, case["n_stout"],
                                            integrator=integ)
        s["kernel"].SetMomenta(_to_host(_random_momenta(ext, seed)).numpy())
    return s


def _take(u, out):
    """The links into the program's pinned buffer (lt_download_links of the C ABI)."""
    if lt.lib().lt_download_links(u.handle, out.numpy()):
        raise RuntimeError(lt.lib().lt_last_error().decode())
    return out


def run(s):
    case, kind, u = s["case"], s["case"]["kind"], s["U"]
    if kind == "update":
        n = (case["rounds"], case["n_hb"], case["n_or"], s["seed"], s["counter"])
        if case["colours"] == 2:
            s["counter"] = lt.UpdateSweeps(u, BETA, *n)
        else:
            s["counter"] = lt.UpdateSweeps4(u, BETA, *n, action=_action(case["action"]))
        return {"plaquette": lt.PlaquetteSum(u), "links": _take(u, s["out"])}
    if kind == "flow":
        p, q, e = s["kernel"].Measure(case["n_meas"], case["every"])
        return {"plaquette": p, "charge": q, "energy": e, "links": _take(s["V"], s["out"])}
    if kind in ("hmc", "metad"):
        h = s["kernel"].Integrate(case["n_step"])
        return {"hamiltonian": np.array(h), "links": _take(u, s["out"])}
    if kind == "analysis":
        u.upload(s["host"].numpy())
        levels = lt.Observables(u, BETA, case["n_smear"], case["smear_skip"], case["eps"])
        for d in levels:
            d["Polyakov_loop"] = np.array([d["Polyakov_loop"].real, d["Polyakov_loop"].imag])
        # one array per observable over the levels, as a program tabulates them
        return {k: np.array([d[k] for d in levels]) for k in levels[0]}
    s["ensemble"].sweeps(case["rounds"])
    return [_take(g, o) for g, o in zip(u, s["out"])]


# ---------------------------------------------------------------- work and tolerances
def work(case):
    """Bytes: each launch-sized step (a sub-sweep, a flow stage, a kick, a drift) reads its
    fields once and writes its result once, and the configuration crosses to the host.  Flops: 198 per
    3x3 complex product, the products each step is defined by."""
    kind, prec = case["kind"], case["prec"]
    b = {"fp64": 144, "fp32": 72, "fp32_12": 48}[prec]
    a = 64 if prec == "fp64" else 32
    V = sum(math.prod(e) for e in _ensemble_extents(case)) if kind == "ensemble" else math.prod(_ext(case))
    links = 4 * V
    host = 4 * V * 144
    rect = case.get("action") in ("lw", "iwasaki", "zeuthen")
    staple = 2500 + (10000 if rect else 0)
    if kind == "update":
        n = case["rounds"] * (case["n_hb"] + case["n_or"]) * links
        per = (9 if case["colours"] == 2 else 17) * b
        return {"bytes": n * per + V * 4 * b + host, "flops": n * (staple + 1400)}
    if kind == "ensemble":
        n = case["rounds"] * 5 * links
        return {"bytes": n * 9 * b + host, "flops": n * (staple + 1400)}
    if kind == "flow":
        n = case["n_meas"] * case["every"]
        return {"bytes": n * links * (6 * b + 4 * a) + case["n_meas"] * 2 * links * b + host,
                "flops": 3 * n * links * (staple + 900) + case["n_meas"] * V * 16000}
    if kind in ("hmc", "metad"):
        kicks = {"Leapfrog": 1, "OMF_2": 2, "OMF_4": 6}[case["integrator"]] * case["n_step"] + 1
        drifts = {"Leapfrog": 1, "OMF_2": 2, "OMF_4": 5}[case["integrator"]] * case["n_step"]
        by = kicks * links * (b + 2 * a) + drifts * links * (2 * b + a) + 2 * links * (b + a) + host
        fl = kicks * links * (staple + 250) + drifts * links * 700
        if kind == "metad":
            by += kicks * links * (6.9 * case["n_stout"] + 3.5) * b
            fl += kicks * links * (14000 + 14000 * case["n_stout"])
        return {"bytes": by, "flops": fl}
    levels = case["n_smear"] + 1
    return {"bytes": host + levels * 9 * links * b + case["n_smear"] * case["smear_skip"] * links * 2 * b,
            "flops": levels * V * 50000 + case["n_smear"] * case["smear_skip"] * links * (staple + 900)}


def tolerance(case):
    """Measured: inputs changed by one rounding, two passes, and the distance from exact(); about
    four times what was seen.  Wilson sweeps: bit for bit (see above)."""
    kind, fp64 = case["kind"], case["prec"] == "fp64"
    if kind == "ensemble" or (kind == "update" and case["action"] == "wilson"):
        return "exact"
    if kind == "update":
        if case["n_hb"]:   # 2e-6 and 2e-5 after forty Luescher-Weisz sweeps
            return {"rel": 1e-5, "max": 1e-3}
        # 3e-7 and 6e-6 after one FP32 sweep, growing 3.5-fold a sweep; 7e-12 after eight in FP64
        return {"rel": 1e-9, "max": 1e-7} if fp64 else {"rel": 2e-4, "max": 2e-2}
    if kind in ("flow", "analysis"):
        # the charge, a sum with cancellations: 4e-6 in FP32 where it is large, more where it is
        # small; 1e-14 in FP64; links 4e-7 and 3e-15
        return {"rel": 1e-11, "max": 1e-10} if fp64 else {"rel": 1e-4, "max": 4e-3}
    # links 4e-7 (largest entry 3e-6) in FP32, 1e-15 in FP64; forces of the smeared charge more
    return {"rel": 1e-11, "max": 1e-10} if fp64 else {"rel": 5e-6, "max": 1e-4}


# ---------------------------------------------------------------- the same in 64 bits
def _sh(f, d, n=1):
    return torch.roll(f, -n, d)


def _staple_plaq(U, mu):
    st = torch.zeros_like(U[mu])
    for nu in range(4):
        if nu == mu:
            continue
        st += _mm(_mm(U[nu], _sh(U[mu], nu)), _dag(_sh(U[nu], mu)))
        st += _sh(_mm(_mm(_dag(U[nu]), U[mu]), _sh(U[nu], mu)), nu, -1)
    return st


def _staple_rect(U, mu):
    """The 1x2 and 2x1 loops through the link, with two-link products D."""
    D = [_mm(U[d], _sh(U[d], d)) for d in range(4)]
    st = torch.zeros_like(U[mu])
    for nu in range(4):
        if nu == mu:
            continue
        st += _mm(_mm(D[nu], _sh(U[mu], nu, 2)), _dag(_sh(D[nu], mu)))
        st += _sh(_mm(_mm(_dag(D[nu]), U[mu]), _sh(D[nu], mu)), nu, -2)
        e = _mm(_mm(U[nu], _sh(D[mu], nu)), _dag(_sh(U[nu], mu, 2)))
        e += _sh(_mm(_mm(_dag(U[nu]), D[mu]), _sh(U[nu], mu, 2)), nu, -1)
        st += _mm(e, _dag(_sh(U[mu], mu))) + _sh(_mm(_dag(U[mu]), e), mu, -1)
    return st


def _staple(U, mu, coef):
    if coef is None:
        return _staple_plaq(U, mu)
    return coef[0] * _staple_plaq(U, mu) + coef[1] * _staple_rect(U, mu)


def _algebra(m):
    m = 0.5 * (m - _dag(m))
    tr = torch.diagonal(m, dim1=-2, dim2=-1).sum(-1) / 3.0
    return m - tr[..., None, None] * torch.eye(3, dtype=m.dtype, device=m.device)


def _force(U, coef):
    return [_algebra(_mm(_staple(U, mu, coef), _dag(U[mu]))) for mu in range(4)]


def _zeuthen_force(U):
    X = _force(U, LW)
    F = []
    for mu in range(4):
        up = _mm(_mm(U[mu], _sh(X[mu], mu)), _dag(U[mu]))
        dn = _sh(_mm(_mm(_dag(U[mu]), X[mu]), U[mu]), mu, -1)
        F.append(X[mu] + (up + dn - 2.0 * X[mu]) / 12.0)
    return F


def _coef(name):
    return {"wilson": None, "lw": LW, "iwasaki": IWASAKI}[name]


def _retr(m):
    return torch.diagonal(m, dim1=-2, dim2=-1).sum(-1).real


def _planes():
    return [(mu, nu) for mu in range(4) for nu in range(mu + 1, 4)]


def _plaquette(U, mu, nu):
    return _mm(_mm(U[mu], _sh(U[nu], mu)), _dag(_mm(U[nu], _sh(U[mu], nu))))


def _plaquette_sum(U):
    return float(sum(_retr(_plaquette(U, mu, nu)).sum() for mu, nu in _planes()))


def _rect_sum(U):
    r = 0.0
    for mu, nu in _planes():
        for a, b in ((mu, nu), (nu, mu)):
            d = _mm(U[a], _sh(U[a], a))
            r += float(_retr(_mm(_mm(d, _sh(U[b], a, 2)), _dag(_mm(U[b], _sh(d, b))))).sum())
    return r


def _clover(U, mu, nu):
    """C - C^dag of the four-leaf clover."""
    p = _plaquette(U, mu, nu)
    g = p + _sh(_mm(_mm(_dag(U[nu]), p), U[nu]), nu, -1)
    c = g + _sh(_mm(_mm(_dag(U[mu]), g), U[mu]), mu, -1)
    return c - _dag(c)


def _clover_densities(U):
    F = {p: _clover(U, *p) for p in _planes()}
    tr = lambda a, b: _retr(_mm(F[a], F[b]))  # noqa: E731
    q = tr((0, 1), (2, 3)) - tr((0, 2), (1, 3)) + tr((0, 3), (1, 2))
    e = 0.0
    for f in F.values():
        t = torch.diagonal(f, dim1=-2, dim2=-1).sum(-1).imag / 3.0
        e = e + (f.abs() ** 2).sum((-1, -2)) - 3.0 * t * t
    return -q / (256.0 * math.pi ** 2), e / 64.0


def _exact_flow(case, U):
    b = {0: (0.0, 1.0, 0.25), 1: (-17.0 / 36.0, 8.0 / 9.0, 1.0), 2: (-1.0, 0.75, 1.0)}
    p, q, e = [], [], []
    for _ in range(case["n_meas"]):
        for _ in range(case["every"]):
            Z = [torch.zeros_like(u) for u in U]
            for j in range(3):
                F = _zeuthen_force(U) if case["action"] == "zeuthen" else _force(U, _coef(case["action"]))
                Z = [b[j][0] * z + b[j][1] * case["eps"] * f for z, f in zip(Z, F)]
                U = [_mm(_expm(b[j][2] * z), u) for z, u in zip(Z, U)]
        dq, de = _clover_densities(U)
        p.append(_plaquette_sum(U))
        q.append(float(dq.sum()))
        e.append(float(de.mean()))
    return {"plaquette": np.array(p), "charge": np.array(q), "energy": np.array(e), "links": _to_host(U)}


def _smeared_charge(U, n_stout):
    for _ in range(n_stout):
        U = [_mm(_expm(RHO * f), u) for f, u in zip(_force(U, None), U)]
    return _clover_densities(U)[0].sum()


def _bias_value(q):
    grid, x = _bias_grid(), (q + 32.0) / 0.02
    i = math.floor(x)
    return grid[i] * (1.0 - (x - i)) + grid[i + 1] * (x - i)


def _exact_md(case, U, P):
    coef = _coef(case.get("action", "wilson"))
    V = math.prod(U[0].shape[:4])

    def bias_force(U):
        U = [u.clone().requires_grad_() for u in U]
        q = _smeared_charge(U, case["n_stout"])
        g = torch.autograd.grad(q, U)
        q = float(q)
        d = (_bias_value(q + 0.01) - _bias_value(q - 0.01)) / 0.02
        return [0.5 * d * _algebra(_mm(u.detach(), _dag(x))) for u, x in zip(U, g)]

    def energy():
        cp, cr = coef or (1.0, 0.0)
        s = BETA * cp * (6.0 * V - _plaquette_sum(U) / 3.0)
        if coef:
            s += BETA * cr * (12.0 * V - _rect_sum(U) / 3.0)
        s += sum(float((p.abs() ** 2).sum()) for p in P)
        if case["kind"] == "metad":
            with torch.no_grad():
                s += _bias_value(float(_smeared_charge(U, case["n_stout"])))
        return s

    def kick(x):
        F = [BETA / 6.0 * f for f in _force(U, coef)]
        if case["kind"] == "metad":
            F = [f + g for f, g in zip(F, bias_force(U))]
        for p, f in zip(P, F):
            p += x * f

    def drift(x):
        for d in range(4):
            U[d] = _mm(_expm(x * P[d]), U[d])

    n, h0 = case["n_step"], energy()
    e = case["tau"] / n
    for k in range(n):   # kicks at the ends of neighbouring steps evaluate the same force
        if case["integrator"] == "Leapfrog":
            steps = [(kick, 0.5), (drift, 1.0), (kick, 0.5)]
        elif case["integrator"] == "OMF_2":
            l2 = 0.1931833275037836
            steps = [(kick, l2), (drift, 0.5), (kick, 1.0 - 2.0 * l2), (drift, 0.5), (kick, l2)]
        else:
            a4, b4, g4, d4 = 0.08398315262876693, 0.2539785108410595, 0.6822365335719091, -0.03230286765269967
            m4, n4 = 0.5 - g4 - a4, 1.0 - 2.0 * (d4 + b4)
            steps = [(kick, a4), (drift, b4), (kick, g4), (drift, d4), (kick, m4), (drift, n4),
                     (kick, m4), (drift, d4), (kick, g4), (drift, b4), (kick, a4)]
        for f, x in steps:
            f(x * e)
    return {"hamiltonian": np.array([h0, energy()]), "links": _to_host(U)}


def _measure(U):
    V, nt = math.prod(U[0].shape[:4]), U[0].shape[0]
    q, e = _clover_densities(U)
    q_t, e_t = q.sum((1, 2, 3)).cpu().numpy(), (e.sum((1, 2, 3)) / V).cpu().numpy()
    plaq = _plaquette_sum(U)
    loops = {}
    C, n = [u.clone() for u in U], 1
    for L in (2, 4, 8):
        while n < L:
            C = [_mm(c, _sh(c, d, n)) for d, c in enumerate(C)]
            n *= 2
        w = sum(float(_retr(_mm(_mm(C[a], _sh(C[b], a, L)), _dag(_mm(C[b], _sh(C[a], b, L))))).sum()) for a, b in _planes())
        loops[L] = 1.0 - w / (18.0 * V)
    poly = U[0][0]
    for t in range(1, nt):
        poly = _mm(poly, U[0][t])
    poly = torch.diagonal(poly, dim1=-2, dim2=-1).sum(-1).mean()
    G = {p: _plaquette(U, *p) for p in _planes()}
    G = {p: g - _dag(g) for p, g in G.items()}
    tr = lambda a, b: float(_retr(_mm(G[a], G[b])).sum())  # noqa: E731
    qp = -(tr((0, 1), (2, 3)) - tr((0, 2), (1, 3)) + tr((0, 3), (1, 2))) / (16.0 * math.pi ** 2)
    lw = LW[0] * (6.0 * V - plaq / 3.0) + LW[1] * (12.0 * V - _rect_sum(U) / 3.0)
    return {"Wilson_Action": 1.0 - plaq / V / 18.0, "Improved_Action": lw / (6.0 * V), "Plaquette": plaq / V,
            "E_plaq": 36.0 - 2.0 * plaq / V, "E_clov": float(e_t.sum()), "E_clov_timeslice": e_t,
            "Wilson_loop(L=2)": loops[2], "Wilson_loop(L=4)": loops[4], "Wilson_loop(L=8)": loops[8],
            "Polyakov_loop": np.array([poly.real.item(), poly.imag.item()]), "TopChargeClov": float(q_t.sum()),
            "TopChargeClov_timeslice": q_t, "TopChargePlaq": qp}


def _exact_analysis(case, U):
    levels = [_measure(U)]
    for _ in range(case["n_smear"]):
        for _ in range(case["smear_skip"]):
            U = [_mm(_expm(case["eps"] * f), u) for f, u in zip(_force(U, None), U)]
        levels.append(_measure(U))
    return {k: np.array([d[k] for d in levels]) for k in levels[0]}


def _reflect(u, st):
    """The three SU(2) subgroup reflections of a link against its staple."""
    w = _mm(u, _dag(st))
    for a, b in ((0, 1), (0, 2), (1, 2)):
        x = 0.5 * (w[..., a, a] + w[..., b, b].conj())
        y = 0.5 * (w[..., a, b] - w[..., b, a].conj())
        n = torch.rsqrt(x.abs() ** 2 + y.abs() ** 2)
        x, y = n * x, n * y
        h, k = (x * x - y * y.conj()).conj(), -(x * y + y * x.conj())
        for m in (u, w):
            ra, rb = m[..., a, :].clone(), m[..., b, :].clone()
            m[..., a, :] = h[..., None] * ra + k[..., None] * rb
            m[..., b, :] = h.conj()[..., None] * rb - k.conj()[..., None] * ra
    return u


def _exact_overrelax(case, U):
    ext = U[0].shape[:4]
    x = torch.meshgrid(*[torch.arange(n, device="cuda") for n in ext], indexing="ij")
    total = x[0] + x[1] + x[2] + x[3]
    coef = _coef(case["action"])
    for _ in range(case["rounds"] * case["n_or"]):
        for mu in range(4):
            colour = total % 2 if case["colours"] == 2 else (total + x[mu]) % 4
            for sub in range(case["colours"]):
                at = colour == sub
                U[mu][at] = _reflect(U[mu][at], _staple(U, mu, coef)[at])
    return {"plaquette": _plaquette_sum(U), "links": _to_host(U)}


def exact(case, seed):
    """What run() returns, in complex128 torch on the library's input rounded as it is stored.
    None for heatbath sweeps, whose links follow the library's own random streams, and where
    this would take long."""
    ext, kind = _ext(case), case["kind"]
    V = math.prod(ext)
    if kind == "ensemble" or (kind == "update" and case["n_hb"] > 0):
        return None
    if kind == "update":
        steps = 40 * case["rounds"] * case["n_or"] * (1 if case["action"] == "wilson" else 3) * case["colours"]
    elif kind == "flow":
        steps = 150 * case["n_meas"] * case["every"] * (1 if case["action"] == "wilson" else 3)
    elif kind == "analysis":
        steps = 150 * (1 + case["n_smear"] * case["smear_skip"])
    else:
        steps = 200 * case["n_step"] * (3 if case["integrator"] == "OMF_4" else 1) * (4 * (1 + case["n_stout"]) if kind == "metad" else 2)
    if V * steps > 1.2e10:
        return None
    # the rows that the storage keeps, rounded to it, the third row rebuilt from them in 64 bits
    U = _random_links(ext, seed)
    if case["prec"] != "fp64":
        U = [u.to(torch.complex64).to(torch.complex128) for u in U]
    if case["prec"] == "fp32_12":
        for u in U:
            u[..., 2, :] = torch.linalg.cross(u[..., 0, :], u[..., 1, :]).conj()
    if kind == "flow":
        return _exact_flow(case, U)
    if kind == "analysis":
        return _exact_analysis(case, U)
    if kind == "update":
        return _exact_overrelax(case, U)
    P = _random_momenta(ext, seed)
    if case["prec"] != "fp64":
        P = [p.to(torch.complex64).to(torch.complex128) for p in P]
    return _exact_md(case, U, P)
