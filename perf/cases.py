"""Timed cases of the lensing-map library: the calls a user's program makes, with seeded inputs.

listed() names the cases, draw(rng) gives further ones from the same ranges.  prepare(case, seed) makes what a
program has in hand before the call (resident catalogues, output planes, a batch), run(state) makes one pass
through the public entry points, work(case) counts what the pass cannot do without and exact(case, seed) gives
the same outputs from plain FP64 torch arithmetic.

Fields of a case
  op         deflection | hessian | potential | lens | mass | posterior | chi2
  precision  fp64 | fp64fast | fp32c
  nx, ny     grid (chi2: nx x nx; posterior: the largest grid side, mass: nx x nx)
  halos      halos of the catalogue, `clusters` of them of cluster scale
  mix        0: cut dPIE only; 1: SIS, PIEMD and cut dPIE halos together
  half       half width of the field (arcsec)
  maps       the Hessian or lens maps asked for, comma separated
  sets       posterior sets, or chi2 models
  systems    image systems (chi2)
"""
import importlib.util
import math
import pathlib
import sys

import numpy as np
import torch

ROOT = pathlib.Path(__file__).resolve().parent.parent


def _package():
    """The package directory has a hyphen in its name: imported by its path, as the tests and the benchmark do."""
    if "lenstool_hpc_b200" not in sys.modules:
        d = ROOT / "lenstool-hpc_b200"
        spec = importlib.util.spec_from_file_location("lenstool_hpc_b200", d / "__init__.py",
                                                      submodule_search_locations=[str(d)])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["lenstool_hpc_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["lenstool_hpc_b200"]


def _case(name, op, precision, nx, ny, halos, clusters=2, mix=0, half=100., maps="", sets=0, systems=0):
    c = dict(op=op, precision=precision, nx=nx, ny=ny, halos=halos, clusters=clusters, mix=mix, half=half, maps=maps,
             sets=sets, systems=systems)
    return dict(name=name, **c) if name else c


def listed():
    return [
        # a small field of the 90-halo model: the four raw Hessian planes in the default precision, a call whose
        # cost is latency and a handful of blocks
        _case("hessian_90h_128", "hessian", "fp64", 128, 128, 90, 1, half=50., maps="hess_a,hess_b,hess_c,hess_d"),
        # the reference's own calling sequence: a host catalogue in, a mass map in host memory out, halos on several
        # lens planes (Kmap weights)
        _case("mass_host_90h_500", "mass", "fp64", 500, 500, 90, 1, half=50., maps="mass"),
        # the deflection benchmark: 200 halos on 1024^2 in the default precision
        _case("deflection_200h_1024", "deflection", "fp64", 1024, 1024, 200),
        # a ragged field with every profile type
        _case("deflection_mix_350h_1501x777", "deflection", "fp64", 1501, 777, 350, 3, mix=1, half=130.),
        # the potential map of an ordinary model
        _case("potential_200h_512", "potential", "fp64", 512, 512, 200),
        # convergence, shear and magnification of a rich cluster in the default precision
        _case("hessian_1000h_1024", "hessian", "fp64", 1024, 1024, 1000, 4, half=150., maps="kappa,gamma1,gamma2,mu"),
        # convergence, shear and potential in the fast FP64 arithmetic, odd sizes
        _case("lens_fast_500h_1199x901", "lens", "fp64fast", 1199, 901, 500, 3, half=120., maps="kappa,gamma1,gamma2,psi"),
        # the headline workload: every lens map of the 1000-halo field on 4096^2
        _case("lens_1000h_4096", "lens", "fp32c", 4096, 4096, 1000, 4, half=150., maps="kappa,gamma1,gamma2,mu,psi"),
        # the same call on a small ragged cut-out
        _case("lens_200h_301x257", "lens", "fp32c", 301, 257, 200, maps="kappa,gamma1,gamma2,mu,psi"),
        # a large deflection grid in the mixed precision (ray shooting)
        _case("deflection_fp32c_1000h_2048", "deflection", "fp32c", 2048, 2048, 1000, 4, half=150.),
        # posterior maps: rows of a chain applied to resident catalogues, then every set's convergence and
        # magnification in one batch (the tiles the serving loop runs too)
        _case("posterior_24x200h_1024", "posterior", "fp32c", 1024, 1024, 200, sets=24, maps="kappa,mu"),
        # one step of a sampler: the chi2 of perturbed models against 40 systems of multiple images
        _case("chi2_4x200h_2048", "chi2", "fp64", 2048, 2048, 200, sets=4, systems=40),
    ]


# rough picoseconds per halo and pixel, to keep the drawn cases below the largest listed one
_PS = {("deflection", "fp64"): 20., ("deflection", "fp64fast"): 13., ("deflection", "fp32c"): 5.,
       ("hessian", "fp64"): 33., ("hessian", "fp64fast"): 10., ("hessian", "fp32c"): 4.,
       ("potential", "fp64"): 90., ("potential", "fp64fast"): 18., ("potential", "fp32c"): 7.,
       ("lens", "fp64"): 122., ("lens", "fp64fast"): 26., ("lens", "fp32c"): 7.,
       ("mass", "fp64"): 33., ("posterior", "fp32c"): 10., ("chi2", "fp64"): 25., ("chi2", "fp32c"): 7.}


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["deflection", "deflection", "hessian", "hessian", "potential", "lens", "lens", "mass", "posterior",
                     "chi2"])
    if op == "mass":
        precision = "fp64"
    elif op == "posterior":
        precision = "fp32c"
    elif op == "chi2":
        precision = rng.choice(["fp64", "fp64", "fp32c"])
    else:
        precision = rng.choice(["fp64", "fp64", "fp32c", "fp32c", "fp64fast"])
    while True:
        halos = _log_int(rng, 40, 2500)
        nx = _log_int(rng, 100, 3000)
        if op == "mass":
            nx = _log_int(rng, 100, 900)
        elif op == "posterior":
            nx = _log_int(rng, 200, 1100)
        elif op == "chi2":
            nx = _log_int(rng, 500, 2100)
        ny = nx if op in ("mass", "posterior", "chi2") else max(33, min(3000, int(nx * math.exp(rng.uniform(-0.7, 0.7)))))
        sets = rng.randint(3, 30) if op == "posterior" else rng.randint(1, 6) if op == "chi2" else 0
        pixels = nx * ny * (0.6 * sets if op == "posterior" else max(1, sets))
        if pixels * halos * _PS[op, precision] * 1e-12 < 0.07:
            break
    maps = ""
    if op == "hessian":
        maps = rng.choice(["kappa,gamma1,gamma2", "hess_a,hess_b,hess_c,hess_d", "shear1", "ampli5", "kappa"])
        if precision != "fp64fast" and rng.random() < 0.5:
            maps = rng.choice(["kappa,gamma1,gamma2,mu", "ampli1", "kappa,mu"])
    elif op == "lens":
        maps = "kappa,gamma1,gamma2,psi" if precision == "fp64fast" else "kappa,gamma1,gamma2,mu,psi"
    elif op == "mass":
        maps = "mass"
    elif op == "posterior":
        maps = "kappa,mu"
    return _case("", op, precision, nx, ny, halos, max(1, min(6, halos // 90)),
                 mix=0 if op in ("posterior", "chi2") else int(rng.random() < 0.3),
                 half=round(rng.uniform(60., 160.), 3), maps=maps, sets=sets,
                 systems=rng.randint(8, 60) if op == "chi2" else 0)


# ---- inputs ---------------------------------------------------------------------------------------------------


def _halos(case, seed):
    """The physical parameters of a cluster + galaxy model (the distributions of the package's own generator):
    {type, x, y, sigma, e, theta, rcore, rcut, plane}, sorted by type and lens plane."""
    rng = np.random.Generator(np.random.PCG64([seed, case["halos"], case["nx"]]))
    nc = case["clusters"]
    ng = case["halos"] - nc
    d = {
        "sigma": np.concatenate([rng.uniform(800., 1200., nc), np.exp(rng.uniform(math.log(80.), math.log(300.), ng))]),
        "rcore": np.concatenate([rng.uniform(5., 15., nc), rng.uniform(0.05, 0.2, ng)]),
        "rcut": np.concatenate([np.full(nc, 800.), rng.uniform(5., 50., ng)]),
        "e": np.concatenate([rng.uniform(0.01, 0.6, nc), rng.uniform(0.01, 0.5, ng)]),
        "theta": rng.uniform(0., math.pi, nc + ng),
        "x": np.concatenate([rng.uniform(-20., 20., nc), rng.uniform(-90., 90., ng)]),
        "y": np.concatenate([rng.uniform(-20., 20., nc), rng.uniform(-90., 90., ng)]),
    }
    t = np.full(nc + ng, 81, np.int32)
    if case["mix"]:
        t = rng.choice(np.array([5, 8, 81, 81], np.int32), nc + ng)
    plane = np.sort(rng.integers(0, 3, nc + ng)) if case["op"] == "mass" else np.zeros(nc + ng, np.int64)
    order = np.lexsort((plane, t))
    d = {k: v[order] for k, v in d.items()}
    d["type"], d["plane"] = t[order], plane[order]
    return d


def _catalog(lt, d):
    c = lt.catalog.make_catalog(d["type"], d["x"], d["y"], d["sigma"], d["e"], d["theta"], d["rcore"], d["rcut"],
                                dlsds=np.array([0.55, 0.7, 0.85])[d["plane"]])
    return c


def _efficiency(seed):
    """D_LS/D_OS of the source plane."""
    return 0.55 + 0.3 * float(np.random.Generator(np.random.PCG64([seed, 77])).random())


def _grid(lt, case, nx=None, ny=None):
    h = case["half"]
    nx, ny = nx or case["nx"], ny or case["ny"]
    return lt.Grid(-h, h, -h * ny / nx, h * ny / nx, nx, ny)


def _posterior_inputs(case, seed):
    """The model, its grid sides and its rows: 5% Gaussian perturbations of every halo's parameters (columns x, y,
    mass ellipticity, angle in degrees, core radius, velocity dispersion, cut radius, halo by halo)."""
    d = _halos(case, seed)
    rng = np.random.Generator(np.random.PCG64([seed, 5]))
    k, n = case["sets"], case["halos"]
    sides = [max(64, int(case["nx"] * (0.25, 0.5, 1.0)[(i * i + i // 3) % 3])) for i in range(k)]
    j = lambda a: a[None, :] * (1. + 0.05 * rng.standard_normal((k, n)))  # noqa: E731
    p = {"x": d["x"] + 0.05 * (np.abs(d["x"]) + 1.) * rng.standard_normal((k, n)),
         "y": d["y"] + 0.05 * (np.abs(d["y"]) + 1.) * rng.standard_normal((k, n)),
         "e": np.clip(j(d["e"]), 0.005, 0.9), "theta": np.degrees(j(d["theta"])), "rcore": np.abs(j(d["rcore"])),
         "sigma": np.abs(j(d["sigma"])), "rcut": np.abs(j(d["rcut"]))}
    rows = np.stack([p[f] for f in ("x", "y", "e", "theta", "rcore", "sigma", "rcut")], axis=2).reshape(k, 7 * n)
    return d, sides, rows, p


def _chi2_systems(lt, case, seed, d, D, device):
    """Observed systems: sources near the largest halo; their images are the local minima of the source-plane
    distance on a coarse grid through the true model, with 0.05" noise (1 to 5 images each)."""
    n, h = 320, min(case["half"], 60.)
    g = torch.linspace(-h, h, n, dtype=torch.float64, device=device)
    px, py = g.repeat(n), g.repeat_interleave(n)
    s = _sums(_profiles(d), px, py, ("alpha",))
    bx, by = (px - D * s["ax"]).reshape(n, n), (py - D * s["ay"]).reshape(n, n)
    rng = np.random.Generator(np.random.PCG64([seed, 9]))
    i = int(np.argmax(d["sigma"]))
    ci = int(np.clip(round((d["x"][i] + h) / (2 * h) * (n - 1)), 0, n - 1))
    cj = int(np.clip(round((d["y"][i] + h) / (2 * h) * (n - 1)), 0, n - 1))
    c0, c1 = float(bx[cj, ci]), float(by[cj, ci])
    nimg, xs, ys = [], [], []
    for _ in range(case["systems"]):
        r, t = 10. * math.sqrt(rng.random()), 2. * math.pi * rng.random()
        q = (bx - (c0 + r * math.cos(t))) ** 2 + (by - (c1 + r * math.sin(t))) ** 2
        low = -torch.nn.functional.max_pool2d(-q[None, None], 3, 1, 1)[0, 0]
        at = torch.nonzero((q == low) & (q < 1.), as_tuple=False)[:5].cpu().numpy()
        if len(at) == 0:
            at = np.array([[cj, ci]])
        nimg.append(len(at))
        xs.append(-h + at[:, 1] * (2 * h / (n - 1)) + 0.05 * rng.standard_normal(len(at)))
        ys.append(-h + at[:, 0] * (2 * h / (n - 1)) + 0.05 * rng.standard_normal(len(at)))
    from lenstool_hpc_b200.images import ImageSystems
    return ImageSystems(np.asarray(nimg, np.int32), np.concatenate(xs), np.concatenate(ys),
                        D * rng.uniform(0.9, 1.1, case["systems"])).contiguous()


class State:
    pass


def prepare(case, seed):
    lt = _package()
    ctx = lt.default_context()
    s = State()
    s.case, s.lt, s.ctx = case, lt, ctx
    s.D = _efficiency(seed)
    plane = lambda ny, nx: torch.empty((ny, nx), dtype=torch.float64, device="cuda")  # noqa: E731
    op = case["op"]
    if op == "mass":
        s.lens = _catalog(lt, _halos(case, seed))
        h = case["half"]
        s.frame = {"xmin": -h, "xmax": h, "ymin": -h, "ymax": h}
    elif op == "posterior":
        from lenstool_hpc_b200 import bayes as B
        d, sides, rows, _ = _posterior_inputs(case, seed)
        params = lt.catalog.HaloParameters(d["type"], d["x"], d["y"], d["sigma"], d["e"], d["theta"], d["rcore"], d["rcut"])
        model = B.model_from_parameters(params)
        cols = [(f, i) for i in range(case["halos"]) for f in (B.X, B.Y, B.EMASS, B.THETA, B.RCORE, B.VDISP, B.RCUT)]
        base = _catalog(lt, d)
        s.cats = [ctx.upload(base) for _ in range(case["sets"])]
        s.post = ctx.bayes(model, cols)
        s.rows = torch.tensor(rows, device="cuda")
        s.out = [{m: plane(n, n) for m in case["maps"].split(",")} for n in sides]
        s.batch = ctx.batch([lt.Request(c, _grid(lt, case, n, n), o, dlsds=s.D)
                             for c, n, o in zip(s.cats, sides, s.out)], precision=case["precision"])
    elif op == "chi2":
        d = _halos(case, seed)
        s.systems = _chi2_systems(lt, case, seed, d, s.D, "cuda")
        rng = np.random.Generator(np.random.PCG64([seed, 3]))
        base = _catalog(lt, d)
        s.cats = [ctx.upload(lt.catalog.perturb_catalog(base, rng)) for _ in range(case["sets"])]
        h = case["half"]
        s.frame = (-h, h, -h, h)
    else:
        s.grid = _grid(lt, case)
        s.cat = ctx.upload(_catalog(lt, _halos(case, seed)))
        names = {"deflection": ["ax", "ay"], "potential": ["psi"]}.get(op) or case["maps"].split(",")
        s.out = {m: plane(s.grid.ny, s.grid.nx) for m in names}
    return s


def run(s):
    case, ctx = s.case, s.ctx
    op, precision = case["op"], case["precision"]
    if op == "deflection":
        ctx.gradient_grid(s.cat, s.grid, precision=precision, out=(s.out["ax"], s.out["ay"]))
    elif op == "potential":
        ctx.potential_grid(s.cat, s.grid, precision=precision, scale=s.D, out=s.out["psi"])
    elif op == "hessian":
        ctx.hessian_maps(s.cat, s.grid, list(s.out), precision=precision, dlsds=s.D, out=list(s.out.values()))
    elif op == "lens":
        ctx.lens_maps(s.cat, s.grid, precision=precision, dlsds=s.D, out=s.out)
    elif op == "mass":
        return s.lt.map_grid_mass_GPU(1, s.lt.cosmo.Cosmology(), s.frame, s.lens, case["nx"], 0.35, 1.5)
    elif op == "posterior":
        s.post.apply(s.rows, s.cats)
        s.batch.launch()
    elif op == "chi2":
        chi, found = ctx.chi2(s.cats, s.frame, case["nx"], s.systems, precision=precision)
        return {"chi2": chi, "images": found}
    return s.out


def work(case):
    """Bytes: the halo parameters read once, the output planes written once.  Flops: one evaluation of the profile
    per halo and pixel, in the shortest closed form of each quantity (+, -, *, /, sqrt and a logarithm or arc
    tangent count one each)."""
    per = {"deflection": 46., "potential": 62., "hessian": 47., "mass": 50., "posterior": 47., "chi2": 46.}
    op, n = case["op"], case["halos"]
    pair = per.get(op) or (71. if "psi" in case["maps"] else 47.)
    if op == "posterior":
        pixels = case["sets"] * (1. / 16 + 1. / 4 + 1.) / 3. * case["nx"] * case["ny"]
    else:
        pixels = float(case["nx"] * case["ny"]) * max(1, case["sets"])
    planes = {"deflection": 2, "potential": 1, "chi2": 0}.get(op)
    planes = len(case["maps"].split(",")) if planes is None else planes
    return {"bytes": 8. * planes * pixels + 72. * n * max(1, case["sets"]) + 24. * 4 * case["systems"],
            "flops": pair * n * pixels}


# ---- the same outputs in plain FP64 torch ------------------------------------------------------------------------


def _profiles(d):
    """Per halo: type, centre, cos, sin, ellipticity of the potential, impact parameter, radii, weight."""
    pi_c2 = 7.209970e-06
    out = []
    for i in range(len(d["x"])):
        t, e, s = int(d["type"][i]), float(d["e"][i]), float(d["sigma"][i])
        eps = e / 3 if t == 5 else (1. - math.sqrt(1. - e * e)) / e
        out.append((t, float(d["x"][i]), float(d["y"][i]), math.cos(d["theta"][i]), math.sin(d["theta"][i]), eps,
                    (4. if t == 5 else 6.) * pi_c2 * s * s, float(d["rcore"][i]), float(d["rcut"][i]),
                    (0.55, 0.7, 0.85)[int(d["plane"][i])]))
    return out


def _ellipse(u, v, eps, A, r, want, acc, sign):
    """Adds sign x one isothermal ellipse of core radius r (halo frame): axis ratio q = (1 - eps)/(1 + eps)."""
    q = (1. - eps) / (1. + eps)
    k = 2. * math.sqrt(eps) / (1. + eps)
    s = (1. + eps) * r
    uu, vv = u * u, v * v
    psi = torch.sqrt(q * q * (s * s + uu) + vv)
    if "hess" in want:
        D = (1. + q * q) * s * s + 2. * s * psi + uu + vv
        E = (sign * A / 2.) / psi
        acc["k"] += E
        E /= D
        acc["g1"] += E * ((q * q - 1.) * s * s + vv - uu)
        acc["g2"] -= 2. * E * u * v
    if "alpha" in want or "psi" in want:
        au = (A / k) * torch.atan(k * u / (psi + s))
        av = (A / k) * torch.atanh(k * v / (psi + q * q * s))
        if "alpha" in want:
            acc["u"] += sign * au
            acc["v"] += sign * av
        if "psi" in want:
            t = (uu + vv + 2. * s * (q * q * uu + vv) / (psi + q * s)) / (4. * r * r)
            acc["p"] += sign * (u * au + v * av - (A * s / 2.) * torch.log1p(t))


def _sums(profiles, px, py, want, weighted=False):
    """Sums over the halos at the points (px, py): convergence and shear, deflection, potential (unscaled)."""
    out = {k: torch.zeros_like(px) for k in ("k", "g1", "g2", "ax", "ay", "psi")}
    for t, x0, y0, c, s, eps, b0, rc, rcut, w in profiles:
        x, y = px - x0, py - y0
        u, v = x * c + y * s, y * c - x * s
        a = {k: torch.zeros_like(px) for k in (("k", "g1", "g2") if "hess" in want else ()) +
             (("u", "v") if "alpha" in want else ()) + (("p",) if "psi" in want else ())}
        if t == 5:
            R = torch.sqrt((1. - eps) * u * u + (1. + eps) * v * v)
            if "hess" in want:
                kk = 0.5 * b0 * (1. - eps * eps) / (R * R * R)
                a["k"], a["g1"], a["g2"] = kk * (u * u + v * v), kk * (v * v - u * u), -2. * kk * u * v
            if "alpha" in want:
                a["u"], a["v"] = b0 * (1. - eps) * u / R, b0 * (1. + eps) * v / R
            if "psi" in want:
                a["p"] = b0 * R
        else:
            A = b0 * (1. - eps) * (rcut / (rcut - rc) if t == 81 else 1.)
            _ellipse(u, v, eps, A, rc, want, a, 1.)
            if t == 81:
                _ellipse(u, v, eps, A, rcut, want, a, -1.)
        f = w if weighted else 1.
        if "hess" in want:
            c2, s2 = c * c - s * s, 2. * s * c
            out["k"] += f * a["k"]
            out["g1"] += f * (a["g1"] * c2 - a["g2"] * s2)
            out["g2"] += f * (a["g1"] * s2 + a["g2"] * c2)
        if "alpha" in want:
            out["ax"] += a["u"] * c - a["v"] * s
            out["ay"] += a["u"] * s + a["v"] * c
        if "psi" in want:
            out["psi"] += a["p"]
    return out


def _map(kind, h, D):
    """One map of the sums h."""
    k, g1, g2 = h["k"], h["g1"], h["g2"]
    g = torch.sqrt(g1 * g1 + g2 * g2)
    if kind in ("hess_a", "hess_b", "hess_c", "hess_d"):
        return {"hess_a": k + g1, "hess_c": k - g1}.get(kind, g2)
    return {"kappa": lambda: k * D, "gamma1": lambda: g1 * D, "gamma2": lambda: g2 * D, "mass": lambda: k,
            "mu": lambda: 1. / ((1. - k * D) ** 2 - (g1 * D) ** 2 - (g2 * D) ** 2),
            "ampli1": lambda: 1. / ((1. - k * D - g * D) * (1. - k * D + g * D)), "ampli5": lambda: k,
            "shear1": lambda: g * D, "psi": lambda: h["psi"] * D}[kind]()


def _points(grid, device):
    """Pixel coordinates, one band of rows after another."""
    x = grid.xmin + torch.arange(grid.nx, dtype=torch.float64, device=device) * grid.dx
    rows = max(1, 2 ** 25 // grid.nx)
    for j in range(0, grid.ny, rows):
        y = grid.ymin + torch.arange(j, min(grid.ny, j + rows), dtype=torch.float64, device=device) * grid.dy
        yield x.repeat(len(y)), y.repeat_interleave(grid.nx)


def _exact_maps(profiles, grid, maps, D, device, weighted=False):
    want = tuple({"psi": "psi", "ax": "alpha", "ay": "alpha"}.get(m, "hess") for m in maps)
    parts = {m: [] for m in maps}
    for px, py in _points(grid, device):
        h = _sums(profiles, px, py, want, weighted)
        for m in maps:
            parts[m].append(h[m] if m in ("ax", "ay") else _map(m, h, D))
    return {m: torch.cat(p).reshape(grid.ny, grid.nx) for m, p in parts.items()}


def exact(case, seed):
    if case["op"] == "chi2":
        return None  # linked images of a search over grid cells: a count and a sum, no value to be near to
    lt = _package()
    device = "cuda" if torch.cuda.is_available() else "cpu"
    D = _efficiency(seed)
    if case["op"] == "posterior":
        d, sides, _, p = _posterior_inputs(case, seed)
        out = []
        for r, n in enumerate(sides):
            q = dict(d, **{f: p[f][r] for f in p})
            q["theta"] = np.radians(q["theta"])
            out.append(_exact_maps(_profiles(q), _grid(lt, case, n, n), case["maps"].split(","), D, device))
        return out
    prof = _profiles(_halos(case, seed))
    if case["op"] == "mass":
        return _exact_maps(prof, _grid(lt, case), ["mass"], D, device, weighted=True)["mass"]
    maps = {"deflection": ["ax", "ay"], "potential": ["psi"]}.get(case["op"]) or case["maps"].split(",")
    return _exact_maps(prof, _grid(lt, case), maps, D, device)
