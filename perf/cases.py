"""Timed cases of the spectral Green's-function path, through the package's public Python API.

Each case is a dict of plain values whose "kind" names one use of the framework:

  film       one film stack on a 1D rule: build_cavity_transfer_1d + closed_form_G
  contour    the same on a deformed kρ contour: build_cavity_transfer_1d_contour + closed_form_G
  film_batch many film stacks at once: build_cavity_transfer_batch + closed_form_G_batch
  grid2d     one stack on a (kρ, φ) grid: build_cavity_transfer_2d + closed_form_G
  plan       an uneven batch of stacks replayed as one BatchPlan
  response   the cavity response on a window of kρ (the pole scan's and the windows' call)
  mlp        the node-placement network: forward over scan grids, or one batch's gradients

`exact` restates the physics in 64 bits with torch alone: per node the tangential-field modes of
every layer, one linear system for all mode amplitudes with a dipole's field jump as its source,
and the Sommerfeld or Fourier sum. Units are nm, as in bench.py.
"""
import math

import numpy as np
import torch

from yellowthinfilms_b200 import api
from yellowthinfilms_b200.materials import (BiaxialMaterial, FlatOpticalLayer, GyrotropicMaterial, IsotropicMaterial,
                                            UniaxialMaterial)

C128 = torch.complex128
MLP_SIZES = (154, 256, 256, 256, 256, 2)


def listed():
    return [
        # one quick look at a film: the package's smoke problem, every term, G on the host
        dict(name="film_point", kind="film", panels=32, order=8, kmax=20.0, nr=8, ny=1, nz=4, even=True,
             terms="all", precision="fp64", host=True),
        # the 3-layer dipole problem in the default precision, at odd sizes
        dict(name="film_map_fp64", kind="film", panels=583, order=7, kmax=20.0, nr=251, ny=1, nz=61, even=True,
             terms="scattered", precision="fp64", host=False),
        # the Bessel synthesis at scale: 4096 radii x 65536 nodes x 256 heights
        dict(name="film_wide_int8", kind="film", panels=8192, order=8, kmax=20.0, nr=4096, ny=1, nz=256, even=True,
             terms="scattered", precision="int8x3", host=False),
        # the dipole problem on the deformed contour
        dict(name="film_contour_int8", kind="contour", panels=512, order=8, nr=256, ny=1, nz=64, even=True,
             terms="all", precision="int8x3", host=False),
        # one refinement level of many stacks, as the adaptive quadrature runs it
        dict(name="film_batch_int8", kind="film_batch", stacks=32, panels=1450, order=8, kmax=119.0, nr=256, nz=64,
             terms="scattered", precision="int8x3"),
        # one wavelength of the 8-layer biaxial/gyrotropic solve: 65536 (kρ, φ) nodes, 32 x 32 offsets
        dict(name="gyro_int8", kind="grid2d", stack="aniso", layers=8, src=4, obs=4, every=False, panels=128, order=8,
             kmax=20.0, nphi=64, nx=32, ny=32, nz=8, terms="all", precision="int8x3", host=False),
        # a smaller anisotropic stack in the default precision, field in another layer, every layer cached
        dict(name="aniso_fp64", kind="grid2d", stack="aniso", layers=5, src=2, obs=4, every=True, panels=57, order=7,
             kmax=12.0, nphi=36, nx=21, ny=13, nz=5, terms="all", precision="fp64", host=True),
        # a film on the 2D grid: one solve per kρ rotated to every φ
        dict(name="film_rotated_fp64", kind="grid2d", stack="film", layers=3, src=1, obs=1, every=False, panels=64,
             order=8, kmax=20.0, nphi=96, nx=24, ny=24, nz=4, terms="scattered", precision="fp64", host=False),
        # the uneven batch: 2-24 layers, isotropic / hyperbolic / gyrotropic, a few pixels each
        dict(name="uneven_plan", kind="plan", items=96, nk_lo=512, nk_hi=8192, nx=4, nz=4),
        # a window of the pole scan
        dict(name="response_window", kind="response", layers=3, n=2048),
        # the network's prediction for 32 stacks on their 2048-point scan grids
        dict(name="mlp_forward", kind="mlp", what="forward", rows=65536),
        # one training batch: loss and gradients
        dict(name="mlp_gradients", kind="mlp", what="gradients", rows=8192),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["film", "film", "contour", "film_batch", "grid2d", "grid2d", "plan", "response", "mlp"])
    terms = rng.choice(["all", "scattered"])
    if kind in ("film", "contour"):
        precision = rng.choice(["fp64", "int8x3"])
        c = dict(kind=kind, panels=size(32, 2048 if kind == "film" else 512), order=rng.choice([7, 8, 10]), kmax=20.0,
                 nr=size(4, 512), ny=1, nz=size(2, 96), even=rng.random() < 0.7, terms=terms, precision=precision,
                 host=rng.random() < 0.4)
        if rng.random() < 0.3:
            c.update(nr=size(3, 40), ny=size(2, 20))
        if kind == "contour":
            del c["kmax"]
        return c
    if kind == "film_batch":
        return dict(kind=kind, stacks=size(2, 32), panels=size(200, 1450), order=rng.choice([8, 10]), kmax=119.0,
                    nr=size(32, 256), nz=size(8, 64), terms=terms, precision="int8x3")
    if kind == "grid2d":
        layers = rng.randint(3, 8)
        src = rng.randint(1, layers - 1)
        every = rng.random() < 0.3
        film = rng.random() < 0.3
        if film:
            layers, src, every = 3, 1, False
        obs = rng.randint(1, layers) if every else src
        return dict(kind=kind, stack="film" if film else "aniso", layers=layers, src=src, obs=obs, every=every,
                    panels=size(16, 96), order=rng.choice([7, 8]), kmax=rng.uniform(8.0, 20.0), nphi=size(8, 64),
                    nx=size(2, 32), ny=size(2, 32), nz=size(1, 8), terms="all" if obs != src else terms,
                    precision=rng.choice(["fp64", "int8x3", "split_bf16"]), host=rng.random() < 0.4)
    if kind == "plan":
        return dict(kind=kind, items=size(8, 96), nk_lo=256, nk_hi=size(1024, 8192), nx=rng.randint(2, 5),
                    nz=rng.randint(1, 5))
    if kind == "response":
        return dict(kind=kind, layers=rng.randint(3, 8), n=size(129, 65536))
    if rng.random() < 0.3:
        return dict(kind="mlp", what="gradients", rows=size(512, 8192))
    return dict(kind="mlp", what="forward", rows=size(2048, 65536))


# ------------------------------------------------------------------------------------
# problems (plain numpy, from the seed alone): layers are (kind, [εx, εy, εz, εxy], d)
# ------------------------------------------------------------------------------------
def _film(rng):
    """Air / uniaxial film / substrate (the learned workload's distribution) and λ."""
    lam = rng.uniform(450.0, 750.0)
    eo = complex(-rng.uniform(1.0, 6.0), 10 ** rng.uniform(-2.5, -0.3))
    ee = complex(rng.uniform(2.0, 6.0), 10 ** rng.uniform(-2.7, -0.5))
    sub = complex(rng.uniform(1.5, 4.0))
    return [("iso", [1.0 + 0j] * 3 + [0j], 200.0), ("uni", [eo, eo, ee, 0j], rng.uniform(20.0, 100.0)),
            ("iso", [sub] * 3 + [0j], 100.0)], lam


def _symmetric(rng, n):
    """n isotropic / uniaxial layers between lossless half-spaces."""
    lam = rng.uniform(450.0, 750.0)
    out = [("iso", [1.0 + 0j] * 3 + [0j], 200.0)]
    for _ in range(n - 2):
        if rng.random() < 0.5:
            e = complex(rng.uniform(1.5, 5.0), rng.uniform(0.01, 0.3))
            out.append(("iso", [e] * 3 + [0j], rng.uniform(10.0, 150.0)))
        else:
            eo = complex(-rng.uniform(1.0, 6.0), rng.uniform(0.01, 0.5))
            ee = complex(rng.uniform(2.0, 6.0), rng.uniform(0.01, 0.5))
            out.append(("uni", [eo, eo, ee, 0j], rng.uniform(10.0, 150.0)))
    e = complex(rng.uniform(1.5, 4.0))
    return out + [("iso", [e] * 3 + [0j], 100.0)], lam


def _aniso(rng, n):
    """n biaxial / ε_xy-gyrotropic layers (the batched solve's distribution)."""
    lam = rng.uniform(450.0, 750.0)
    out = []
    for l in range(n):
        d = [complex(a, b) for a, b in zip(rng.uniform(-6.0, 6.0, 3), rng.uniform(0.01, 1.0, 3))]
        g = rng.uniform(0.0, 1.5)
        out.append(("gyro", d + [1j * g], rng.uniform(10.0, 200.0)) if rng.random() < 0.5
                   else ("bi", d + [0j], rng.uniform(10.0, 200.0)))
    return out, lam


def _uneven(rng):
    """One stack of the uneven batch: 2-24 layers, isotropic half-spaces."""
    n = int(rng.integers(2, 25))
    out = []
    for l in range(n):
        d = rng.uniform(5.0, 300.0)
        half = l in (0, n - 1)
        kind = 0 if half else int(rng.integers(0, 3))
        if kind == 0:
            e = complex(rng.uniform(1.0, 2.5 if half else 6.0), rng.uniform(0.001, 0.3))
            out.append(("iso", [e] * 3 + [0j], d))
        elif kind == 1:
            s = 1.0 if rng.random() < 0.5 else -1.0
            eo = complex(-s * rng.uniform(1.0, 6.0), rng.uniform(0.01, 0.5))
            ee = complex(s * rng.uniform(1.0, 6.0), rng.uniform(0.01, 0.5))
            out.append(("uni", [eo, eo, ee, 0j], d))
        else:
            e = [complex(a, b) for a, b in zip(rng.uniform(1.0, 6.0, 3), rng.uniform(0.01, 0.5, 3))]
            out.append(("gyro", e + [1j * rng.uniform(0.0, 1.5)], d))
    return out, rng.uniform(450.0, 750.0)


def _layers(stack):
    """The package's layer objects of a problem's stack."""
    out = []
    for kind, (ex, ey, ez, exy), d in stack:
        if kind == "iso":
            m = IsotropicMaterial(ex)
        elif kind == "uni":
            m = UniaxialMaterial(ex, ez)
        elif kind == "bi":
            m = BiaxialMaterial(ex, ey, ez)
        else:
            m = GyrotropicMaterial([[ex, exy, 0], [-exy, ey, 0], [0, 0, ez]])
        out.append(FlatOpticalLayer(m, d))
    return out


def _rule(panels, order, kmax):
    """Gauss-Legendre rule on uniform panels over [0, kmax]."""
    x, w = np.polynomial.legendre.leggauss(order)
    e = np.linspace(0.0, kmax, panels + 1)
    h = 0.5 * np.diff(e)
    return (0.5 * (e[1:] + e[:-1])[:, None] + h[:, None] * x).ravel(), (h[:, None] * w).ravel()


def _contour(panels, order, k0):
    """kρ(t) = t - 0.05i k0 sin(π t / 20 k0), t in [0, 20 k0]."""
    t, w = _rule(panels, order, 20.0 * k0)
    L, h = 20.0 * k0, 0.05 * k0
    return t - 1j * h * np.sin(np.pi * t / L), w * (1.0 - 1j * h * (np.pi / L) * np.cos(np.pi * t / L))


def _heights(rng, nz, lo, hi, even):
    return np.linspace(lo, hi, nz) if even else np.sort(rng.uniform(lo, hi, nz))


def _problem(case, seed):
    """Stack, frequency, source, rule and observation set of a case, as plain values."""
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    p = {}
    if kind in ("film", "contour"):
        p["stack"], lam = _film(rng)
        k0 = 2 * np.pi / lam
        p.update(k0=k0, src=1, obs=1, zsrc=20.0, z=_heights(rng, case["nz"], 0.5, 199.5, case["even"]))
        if case["ny"] == 1:
            p.update(x=np.geomspace(0.01 * lam, 5.0 * lam, case["nr"]), y=np.zeros(1))
        else:
            p.update(x=np.linspace(-0.8 * lam, 0.9 * lam, case["nr"]), y=np.linspace(-0.5 * lam, 0.6 * lam, case["ny"]))
        p["k"], p["w"] = (_contour(case["panels"], case["order"], k0) if kind == "contour"
                          else _rule(case["panels"], case["order"], case["kmax"] * k0))
    elif kind == "film_batch":
        p["items"] = []
        for _ in range(case["stacks"]):
            stack, lam = _film(rng)
            k0 = 2 * np.pi / lam
            k, w = _rule(int(case["panels"] * rng.uniform(0.75, 1.0)), case["order"], case["kmax"] * k0)
            p["items"].append(dict(stack=stack, k0=k0, src=1, obs=1, zsrc=20.0, z=np.linspace(0.0, 200.0, case["nz"]),
                                   x=np.geomspace(0.01 * lam, 5.0 * lam, case["nr"]), y=np.zeros(1), k=k, w=w))
    elif kind == "grid2d":
        p["stack"], lam = _film(rng) if case["stack"] == "film" else _aniso(rng, case["layers"])
        k0 = 2 * np.pi / lam
        d, do = p["stack"][case["src"] - 1][2], p["stack"][case["obs"] - 1][2]
        p.update(k0=k0, src=case["src"], obs=case["obs"], zsrc=0.1 * d if case["stack"] == "film" else 0.5 * d,
                 z=np.linspace(0.05 * do, 0.95 * do, case["nz"]) if case["nz"] > 1 else np.array([0.3 * do]),
                 x=np.linspace(-0.2 * lam, 0.2 * lam, case["nx"]), y=np.linspace(-0.2 * lam, 0.2 * lam, case["ny"]))
        p["k"], p["w"] = _rule(case["panels"], case["order"], case["kmax"] * k0)
        p["phi"] = 2 * np.pi * np.arange(case["nphi"]) / case["nphi"]
        p["wphi"] = np.full(case["nphi"], 2 * np.pi / case["nphi"])
    elif kind == "plan":
        p["items"] = []
        for _ in range(case["items"]):
            stack, lam = _uneven(rng)
            k0 = 2 * np.pi / lam
            gyro = any(l[0] == "gyro" for l in stack)
            src = int(rng.integers(1, len(stack)))
            nk = int(np.exp(rng.uniform(np.log(case["nk_lo"]), np.log(case["nk_hi"]))))
            k, w = _rule(max(1, (nk // 8 if gyro else nk) // 8), 8, 20.0 * k0)
            d = stack[src - 1][2]
            xy = np.linspace(-0.2 * lam, 0.2 * lam, case["nx"])
            it = dict(stack=stack, k0=k0, src=src, obs=src, zsrc=0.5 * d, z=np.linspace(0.1 * d, 0.9 * d, case["nz"]),
                      x=xy, y=xy, k=k, w=w)
            if gyro:
                it.update(phi=2 * np.pi * np.arange(8) / 8, wphi=np.full(8, 2 * np.pi / 8))
            p["items"].append(it)
    elif kind == "response":
        p["stack"], lam = _symmetric(rng, case["layers"])
        k0 = 2 * np.pi / lam
        p.update(k0=k0, src=1 if case["layers"] == 3 else 2, k=k0 * np.geomspace(0.25, 100.0, case["n"]))
    return p


def _network(case, seed):
    """Weights (He-uniform) and inputs of the network: feature rows of 3-layer stacks (ε / 10,
    thickness, λ), each over a scan grid, as the node placement forms them."""
    rng = np.random.default_rng(seed)
    params = np.concatenate([np.concatenate([
        rng.uniform(-1.0, 1.0, (o, i)).astype(np.float32).ravel() * np.float32(math.sqrt(6.0 / i)),
        rng.normal(0.0, 0.05, o).astype(np.float32)]) for i, o in zip(MLP_SIZES[:-1], MLP_SIZES[1:])])
    n = case["rows"]
    g = 2048 if n >= 2048 else 64
    rows = np.zeros((-(-n // g), MLP_SIZES[0]), np.float32)
    for r in rows:
        stack, lam = _film(rng)
        for l, (_, e, d) in enumerate(stack):
            for j, v in zip((0, 4, 8), e[:3]):
                r[19 * l + j], r[19 * l + 9 + j] = v.real / 10.0, v.imag / 10.0
            r[19 * l + 18] = d / lam
        r[-2] = 600.0 / lam
    X = np.repeat(rows, g, axis=0)[:n]
    X[:, -1] = np.tile(np.geomspace(0.25, 160.0, g) / 160.0, len(rows))[:n]
    T = np.stack([rng.normal(0.0, 1.0, n), rng.uniform(0.0, 1.0, n)], 1).astype(np.float32)
    return params, X, T


# ------------------------------------------------------------------------------------
# what a program keeps, and one pass of it
# ------------------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind == "mlp":
        params, X, T = _network(case, seed)
        net = api.MLP(MLP_SIZES)
        net.params = params
        return dict(case=case, net=net, X=torch.from_numpy(X).cuda() if case["what"] == "forward" else X, T=T)
    p = _problem(case, seed)
    s = dict(case=case, p=p)
    if kind in ("film_batch", "plan"):
        n = 9 * len(p["items"][0]["x"]) * len(p["items"][0]["y"]) * len(p["items"][0]["z"])
        s["out"] = torch.zeros((len(p["items"]), n), dtype=C128, device="cuda")
        tr, gr = [], []
        for it, out in zip(p["items"], s["out"]):
            t = dict(stack=api.Stack(_layers(it["stack"])), omega=it["k0"], source_layer=it["src"], obs_layers=[it["obs"]])
            if "phi" in it:
                t.update(kr_nodes=it["k"], kr_weights=it["w"], phi_nodes=it["phi"], phi_weights=it["wphi"], rotation=False)
            elif kind == "film_batch":  # rules stay in device memory, as the refinement keeps them
                t.update(kx_nodes=torch.from_numpy(it["k"]).cuda(), wt_nodes=torch.from_numpy(it["w"]).cuda())
            else:
                t.update(kx_nodes=it["k"], wt_nodes=it["w"])
            tr.append(t)
            gr.append(dict(obs_layer=it["obs"], zsrc_local=it["zsrc"], z_obs=it["z"], xs=it["x"], ys=it["y"], out=out))
        if kind == "plan":
            s["plan"] = api.BatchPlan(tr, gr)
        else:
            s["transfer"] = tr
            s["green"] = [dict(g, terms=case["terms"], precision=case["precision"]) for g in gr]
        return s
    s["stack"] = api.Stack(_layers(p["stack"]))
    if kind != "response" and not case["host"]:
        s["out"] = torch.zeros(9 * len(p["x"]) * len(p["y"]) * len(p["z"]), dtype=C128, device="cuda")
    return s


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "mlp":
        if case["what"] == "forward":
            return state["net"].forward(state["X"])
        return state["net"].gradients(state["X"], state["T"])
    p = state["p"]
    if kind == "plan":
        state["plan"]()
        return state["out"]
    if kind == "film_batch":
        caches = api.build_cavity_transfer_batch(state["transfer"])
        api.closed_form_G_batch([dict(g, cache=c) for g, c in zip(state["green"], caches)])
        return state["out"]
    if kind == "response":
        return api.cavity_response(state["stack"], p["k0"], p["src"], p["k"])
    if kind == "film":
        cache = api.build_cavity_transfer_1d(state["stack"], p["k0"], p["src"], p["k"], p["w"], obs_layers=[p["obs"]])
    elif kind == "contour":
        cache = api.build_cavity_transfer_1d_contour(state["stack"], p["k0"], p["src"], p["k"], p["w"],
                                                     obs_layers=[p["obs"]])
    else:
        cache = api.build_cavity_transfer_2d(state["stack"], p["k0"], p["src"], p["k"], p["w"], p["phi"], p["wphi"],
                                             obs_layers=None if case["every"] else [p["obs"]])
    return api.closed_form_G(cache, p["obs"], p["zsrc"], p["z"], p["x"], p["y"], terms=case["terms"],
                             precision=case["precision"], out=state.get("out"))


def work(case):
    """Bytes: inputs once, outputs once. Flops: about 3200 per (node, layer) of the solve (2 modes,
    an interface and a star product), 2 per real multiply-add of the synthesis (10 real
    coefficient columns per height on an azimuthally symmetric 1D rule, 9 complex ones in 2D) and
    50 per (node, radius) of the Bessel functions."""
    kind = case["kind"]
    if kind == "mlp":
        macs = case["rows"] * sum(i * o for i, o in zip(MLP_SIZES[:-1], MLP_SIZES[1:]))
        params = sum(i * o + o for i, o in zip(MLP_SIZES[:-1], MLP_SIZES[1:]))
        step = case["what"] == "gradients"
        return {"bytes": 4.0 * (case["rows"] * (154 + 2 + 2 * step) + params * (1 + step)),
                "flops": 2.0 * macs * (3 if step else 1)}
    if kind == "response":
        return {"bytes": 16.0 * case["n"], "flops": 3200.0 * case["layers"] * case["n"]}
    if kind == "plan":
        mean = (case["nk_hi"] - case["nk_lo"]) / math.log(case["nk_hi"] / case["nk_lo"])
        n, pix = mean * case["items"], case["nx"] ** 2
        return {"bytes": 16.0 * n + 144.0 * case["items"] * pix * case["nz"],
                "flops": n * (3200.0 * 13 + 72.0 * pix * case["nz"])}
    if kind == "grid2d":
        n, pix = case["panels"] * case["order"] * case["nphi"], case["nx"] * case["ny"]
        solved = n / case["nphi"] if case["stack"] == "film" else n
        return {"bytes": 16.0 * (case["panels"] * case["order"] + case["nphi"]) + 144.0 * pix * case["nz"],
                "flops": 3200.0 * case["layers"] * solved + 72.0 * n * pix * case["nz"]}
    n, nr = case["panels"] * case["order"], case["nr"] * case.get("ny", 1)
    mul = case["stacks"] * 0.875 if kind == "film_batch" else 1.0
    cols = 20.0 * (2 if kind == "contour" else 1)
    return {"bytes": mul * (16.0 * n + 144.0 * nr * case["nz"]),
            "flops": mul * n * (3200.0 * 3 + nr * (50.0 + cols * case["nz"]))}


# ------------------------------------------------------------------------------------
# the same results in 64 bits
# ------------------------------------------------------------------------------------
def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _c(v):
    return torch.as_tensor(np.asarray(v), device=_dev()).to(C128)


def _modes(layer, w, kx, ky):
    """q and tangential vectors (Ex, Ey, Hx, Hy) of a layer's modes: (qf, qb) [n, 2] and
    (Vf, Vb) [n, 4, 2], forward = decaying (or carrying power) upward in z."""
    kind, (ex, ey, ez, exy), _ = layer
    if kind in ("iso", "uni"):
        kr = torch.sqrt(kx * kx + ky * ky)
        c, s = torch.where(kr == 0, torch.ones_like(kr), kx / kr), torch.where(kr == 0, torch.zeros_like(kr), ky / kr)
        qo, qe = torch.sqrt(w * w * ex - kr * kr), torch.sqrt(ex * (w * w - kr * kr / ez))
        qo, qe = torch.where(qo.imag < 0, -qo, qo), torch.where(qe.imag < 0, -qe, qe)
        # lossless media: a real qe of a negative-index pair carries power along -qe / εx
        o, z = torch.ones_like(qo), torch.zeros_like(qo)
        te = lambda q: torch.stack([-s * o, c * o, -q * c / w, -q * s / w], 1)
        tm = lambda q: torch.stack([q * c / (w * ex), q * s / (w * ex), -s + z, c + z], 1)
        return (torch.stack([qo, qe], 1), torch.stack([-qo, -qe], 1), torch.stack([te(qo), tm(qe)], 2),
                torch.stack([te(-qo), tm(-qe)], 2))
    # no xz/yz coupling: B = [[0, P], [R, 0]], q² the eigenvalues of P R
    e21 = -exy
    P = torch.stack([torch.stack([kx * ky / (w * ez), w - kx * kx / (w * ez)], 1),
                     torch.stack([-w + ky * ky / (w * ez), -kx * ky / (w * ez)], 1)], 1)
    R = torch.stack([torch.stack([-kx * ky / w - w * e21, kx * kx / w - w * ey], 1),
                     torch.stack([-ky * ky / w + w * ex, kx * ky / w + w * exy], 1)], 1)
    M = P @ R
    h = (M[:, 0, 0] - M[:, 1, 1]) / 2
    disc, mid = torch.sqrt(h * h + M[:, 0, 1] * M[:, 1, 0]), (M[:, 0, 0] + M[:, 1, 1]) / 2
    qs, As = [], []
    for sg in (1.0, -1.0):
        d = sg * disc
        a = torch.stack([M[:, 0, 1], d - h], 1)
        b = torch.stack([h + d, M[:, 1, 0]], 1)
        a = torch.where((torch.linalg.vector_norm(a, dim=1) >= torch.linalg.vector_norm(b, dim=1))[:, None], a, b)
        q = torch.sqrt(mid + d)
        qs.append(torch.where(q.imag < 0, -q, q))
        As.append(a / torch.linalg.vector_norm(a, dim=1)[:, None])
    q, A = torch.stack(qs, 1), torch.stack(As, 2)
    H = (R @ A) / q[:, None, :]
    return q, -q, torch.cat([A, H], 1), torch.cat([A, -H], 1)


def _amplitudes(p, kx, ky):
    """Obs-layer modes and the amplitudes of a unit dipole's field at every node: (qf, qb, Ef, Eb
    [n, 3, 2], f, b [n, 2, 3] scattered, df, db [n, 2, 3] direct or None, source position)."""
    w, stack, s, o = p["k0"], p["stack"], p["src"] - 1, p["obs"] - 1
    N, n = len(stack), len(kx)
    modes = [_modes(l, w, kx, ky) for l in stack]
    d = [l[2] for l in stack]
    zp = d[s] - p["zsrc"] if s == 0 else p["zsrc"]
    ez = stack[s][1][2]
    J = torch.zeros((n, 4, 3), dtype=C128, device=kx.device)
    jw = -1j * w
    J[:, 2, 1], J[:, 3, 0] = jw, -jw
    J[:, 0, 2], J[:, 1, 2] = kx * jw / (ez * w), ky * jw / (ez * w)
    qf, qb, Vf, Vb = modes[s]
    seed = torch.linalg.solve(torch.cat([Vf, Vb], 2), J)
    df, db = seed[:, :2], -seed[:, 2:]
    # unknowns b_1, (f_j, b_j) of the inner layers, f_N; f at a layer's lower edge, b at its upper one
    A = torch.zeros((n, 4 * (N - 1), 4 * (N - 1)), dtype=C128, device=kx.device)
    F = torch.zeros((n, 4 * (N - 1), 3), dtype=C128, device=kx.device)
    for j in range(N - 1):
        r = slice(4 * j, 4 * j + 4)
        (q0, p0, V0, W0), (q1, p1, V1, W1) = modes[j], modes[j + 1]
        if j > 0:
            A[:, r, 4 * j - 2:4 * j] = V0 * torch.exp(1j * q0 * d[j])[:, None, :]
        A[:, r, 4 * j:4 * j + 2] = W0
        A[:, r, 4 * j + 2:4 * j + 4] = -V1
        if j + 1 < N - 1:
            A[:, r, 4 * j + 4:4 * j + 6] = -W1 * torch.exp(-1j * p1 * d[j + 1])[:, None, :]
        if j == s:
            F[:, r] -= V0 @ (torch.exp(1j * qf * (d[s] - zp))[:, :, None] * df)
        if j + 1 == s:
            F[:, r] += W1 @ (torch.exp(-1j * qb * zp)[:, :, None] * db)
    X = torch.linalg.solve(A, F)
    zero = torch.zeros((n, 2, 3), dtype=C128, device=kx.device)
    f = zero if o == 0 else X[:, 4 * o - 2:4 * o]
    b = zero if o == N - 1 else X[:, 4 * o:4 * o + 2]
    qf, qb, Vf, Vb = modes[o]
    eo = stack[o][1][2]
    E = lambda V: torch.cat([V[:, :2], (-(kx[:, None] * V[:, 3] - ky[:, None] * V[:, 2]) / (w * eo))[:, None]], 1)
    return qf, qb, E(Vf), E(Vb), f, b, (df, db) if o == s else None, zp, d[o]


def _field(p, amp, z, terms):
    """E[n, component, moment] at height z of the obs layer."""
    qf, qb, Ef, Eb, f, b, direct, zp, d = amp
    f, b = torch.exp(1j * qf * z)[:, :, None] * f, torch.exp(1j * qb * (z - d))[:, :, None] * b
    if terms == "all" and direct is not None:
        if z > zp:
            f = f + torch.exp(1j * qf * (z - zp))[:, :, None] * direct[0]
        elif z < zp:
            b = b + torch.exp(1j * qb * (z - zp))[:, :, None] * direct[1]
    return Ef @ f + Eb @ b


def _bessel(x):
    """J_0, J_1, J_2 by the trapezoid rule of Bessel's integral (it converges geometrically past
    |x| points; for real x one quarter of the circle serves the rest); torch's own above x = 30."""
    if x.is_complex():
        m = int(x.abs().max()) + 80
        out = [torch.zeros_like(x) for _ in range(3)]
        for t in range(m):
            th = 2 * math.pi * t / m
            e = torch.exp(-1j * math.sin(th) * x) / m
            for n in range(3):
                out[n] += e * complex(math.cos(n * th), math.sin(n * th))
        return out
    j0, j1 = torch.special.bessel_j0(x), torch.special.bessel_j1(x)
    j2 = 2 * j1 / x.clamp(min=1.0) - j0
    near = x < 30.0
    u, m = x[near], 96
    s0, s1, s2 = torch.zeros_like(u), torch.zeros_like(u), torch.zeros_like(u)
    for t in range(m // 4 + 1):
        th, wt = 2 * math.pi * t / m, (2.0 if t in (0, m // 4) else 4.0) / m
        a = math.sin(th) * u
        c = torch.cos(a)
        s0 += wt * c
        s1 += wt * math.sin(th) * torch.sin(a)
        s2 += wt * math.cos(2 * th) * c
    j0[near], j1[near], j2[near] = s0, s1, s2
    return j0, j1, j2


def _radial(p, terms):
    """G (moment, component, z, y, x) on a 1D rule."""
    nz = len(p["z"])
    X, Y = np.meshgrid(p["x"], p["y"])
    rho, inv = np.unique(np.hypot(X, Y).ravel(), return_inverse=True)
    r = torch.as_tensor(rho, device=_dev())
    S = [torch.zeros((len(rho), m * nz), dtype=C128, device=_dev()) for m in (2, 2, 1)]
    step = max(256, int(2.5e7 / max(len(rho), 10 * nz)))
    for a in range(0, len(p["k"]), step):
        k, w = p["k"][a:a + step], _c(p["w"][a:a + step])
        kc = _c(k)
        amp = _amplitudes(p, kc, torch.zeros_like(kc))
        g = w * kc / (4 * math.pi)
        cols = [[], [], []]
        for z in p["z"]:
            E = _field(p, amp, float(z), terms)
            cols[0] += [g * (E[:, 0, 0] + E[:, 1, 1]), 2 * g * E[:, 2, 2]]
            cols[1] += [2j * g * E[:, 2, 0], 2j * g * E[:, 0, 2]]
            cols[2] += [g * (E[:, 1, 1] - E[:, 0, 0])]
        J = _bessel(r[:, None] * (kc[None] if np.iscomplexobj(k) else torch.as_tensor(k, device=_dev())[None]))
        for n in range(3):
            C = torch.stack(cols[n], 1)
            S[n] += J[n] @ C if J[n].is_complex() else torch.view_as_complex(
                (J[n] @ torch.view_as_real(C).reshape(len(C), -1)).reshape(len(rho), -1, 2))
    P0, P1, P2 = S[0].reshape(-1, nz, 2), S[1].reshape(-1, nz, 2), S[2].reshape(-1, nz)
    R = torch.zeros((len(rho), nz, 3, 3), dtype=C128, device=_dev())  # component, moment along the radius
    R[..., 0, 0], R[..., 1, 1], R[..., 2, 2] = P0[..., 0] + P2, P0[..., 0] - P2, P0[..., 1]
    R[..., 2, 0], R[..., 0, 2] = P1[..., 0], P1[..., 1]
    h = np.hypot(X, Y).ravel()
    cp, sp = np.where(h == 0, 1.0, X.ravel() / np.where(h == 0, 1.0, h)), np.where(h == 0, 0.0, Y.ravel() / np.where(h == 0, 1.0, h))
    rot = np.zeros((len(h), 3, 3))
    rot[:, 0, 0] = rot[:, 1, 1] = cp
    rot[:, 0, 1], rot[:, 1, 0], rot[:, 2, 2] = -sp, sp, 1.0
    rot = _c(rot)[:, None]
    G = rot @ R[torch.as_tensor(inv.reshape(-1), device=_dev())] @ rot.transpose(2, 3)  # pixel, z, component, moment
    return G.permute(3, 2, 1, 0).reshape(3, 3, nz, len(p["y"]), len(p["x"]))


def _planar(p, terms):
    """G (moment, component, z, y, x) on a (kρ, φ) grid."""
    nz, npix = len(p["z"]), len(p["x"]) * len(p["y"])
    K, PHI = [a.ravel() for a in np.meshgrid(p["k"], p["phi"])]
    W = np.outer(p["wphi"], p["k"] * p["w"]).ravel() / (4 * math.pi ** 2)
    x, y = _c(np.tile(p["x"], len(p["y"]))), _c(np.repeat(p["y"], len(p["x"])))
    G = torch.zeros((npix, 9 * nz), dtype=C128, device=_dev())
    step = max(256, min(16384, int(4e7 / max(npix, (4 * len(p["stack"])) ** 2))))
    for a in range(0, len(K), step):
        kx, ky = _c(K[a:a + step] * np.cos(PHI[a:a + step])), _c(K[a:a + step] * np.sin(PHI[a:a + step]))
        amp, w = _amplitudes(p, kx, ky), _c(W[a:a + step])
        S = torch.stack([_field(p, amp, float(z), terms) for z in p["z"]], 1)  # n, z, component, moment
        S = (w[:, None, None, None] * S).permute(0, 3, 2, 1).reshape(len(kx), -1)
        G += torch.exp(1j * (x[:, None] * kx[None] + y[:, None] * ky[None])) @ S
    return G.reshape(len(p["y"]), len(p["x"]), 3, 3, nz).permute(2, 3, 4, 0, 1)


def _reflections(p):
    """max(|r|, 1 / |1 - r_below r_above e^{2iqd}|) of the source layer's two polarisations."""
    w, stack, s = p["k0"], p["stack"], p["src"] - 1
    k = _c(p["k"])
    best = torch.zeros(len(k), dtype=torch.float64, device=_dev())
    for pol in (0, 1):
        q = [_modes(l, w, k, torch.zeros_like(k))[0][:, pol] for l in stack]
        Y = [qj if pol == 0 else qj / l[1][0] for qj, l in zip(q, stack)]
        side = {}
        for name, chain in (("above", range(len(stack) - 1, s, -1)), ("below", range(0, s))):
            up = 1 if name == "above" else -1
            r = torch.zeros_like(k)
            for j in chain:
                r = r * torch.exp(2j * q[j] * stack[j][2]) if j not in (0, len(stack) - 1) else r
                t = (Y[j - up] - Y[j]) / (Y[j - up] + Y[j])
                r = (t + r) / (1 + t * r)
            side[name] = r
        best = torch.maximum(best, torch.maximum(side["above"].abs(), side["below"].abs()))
        if s > 0:
            best = torch.maximum(best, 1 / (1 - side["above"] * side["below"] * torch.exp(2j * q[s] * stack[s][2])).abs())
    return best


def _network_exact(case, seed):
    params, X, T = _network(case, seed)
    t = lambda a: torch.as_tensor(a, device=_dev()).double()
    layers, o = [], 0
    for i, n in zip(MLP_SIZES[:-1], MLP_SIZES[1:]):
        W = torch.as_tensor(params[o:o + n * i].reshape(n, i), device=_dev()).bfloat16().double()
        layers.append((W, t(params[o + n * i:o + n * i + n])))
        o += n * i + n
    H, Z = [t(X)], []
    for l, (W, b) in enumerate(layers):
        Z.append(H[-1] @ W.T + b)
        H.append(torch.nn.functional.gelu(Z[-1]) if l + 1 < len(layers) else Z[-1])
    if case["what"] == "forward":
        return H[-1]
    out, tt, n = H[-1], t(T), len(X)
    e = out[:, 0] - tt[:, 0]
    loss = float((e * e + torch.nn.functional.softplus(out[:, 1]) - tt[:, 1] * out[:, 1]).mean())
    dZ, grads = torch.stack([2 * e / n, (torch.sigmoid(out[:, 1]) - tt[:, 1]) / n], 1), []
    for l in range(len(layers) - 1, -1, -1):
        if l + 1 < len(layers):
            z = Z[l]
            dZ = dZ * (0.5 * (1 + torch.erf(z / math.sqrt(2))) + z * torch.exp(-0.5 * z * z) / math.sqrt(2 * math.pi))
        grads = [torch.cat([(dZ.T @ H[l]).reshape(-1), dZ.sum(0)])] + grads
        dZ = dZ @ layers[l][0]
    return loss, torch.cat(grads)


def exact(case, seed):
    kind = case["kind"]
    if kind == "mlp":
        return _network_exact(case, seed)
    p = _problem(case, seed)
    if kind == "response":
        return _reflections(p)
    if kind == "film_batch":
        return torch.stack([_radial(it, case["terms"]).reshape(-1) for it in p["items"]])
    if kind == "plan":
        return torch.stack([(_planar if "phi" in it else _radial)(it, "all").reshape(-1) for it in p["items"]])
    G = (_planar if kind == "grid2d" else _radial)(p, case["terms"])
    return G.permute(4, 3, 2, 1, 0) if case["host"] else G.reshape(-1)
