"""The work a user has this library do, through its public entry points: single particle FMM calls
from a few thousand to millions of points, fixed geometries solved again for new charges, batches of
independent problems, Hessians, Helmholtz calls and layer potentials on triangulated surfaces.

Coordinates, charges and densities have the distributions of the benchmark's workloads: points in
the unit cube, on the unit sphere or in a Plummer ball, strengths with parts uniform in [-1, 1]."""
import math

import numpy as np
import torch

import fmmlib3d_b200 as F
from fmmlib3d_b200 import meshes

PAIRS_EXACT = 1.0e11    # pairs of a direct sum that plain torch does in a few seconds
SIDE = 2048             # rows and columns of one block of a direct sum


def listed():
    return [
        # the smallest: the reference's own drivers call it with 2,000 points and host arrays
        dict(name="laplace-host-2k", kind="laplace", shape="cube", n=2000, m=2000, iprec=1, charge=True, dipole=True,
             mixed=False, host=True, plan=False, hess=False),
        # repeated solves on one geometry (an iterative solver, a served geometry): a kept plan, new charges
        dict(name="laplace-plan-sphere-10k", kind="laplace", shape="sphere", n=10000, m=0, iprec=1, charge=True,
             dipole=False, mixed=False, host=False, plan=True, hess=False),
        # one ordinary call on a surface, where the tree is adaptive
        dict(name="laplace-sphere-100k", kind="laplace", shape="sphere", n=100000, m=0, iprec=1, charge=True,
             dipole=False, mixed=False, host=False, plan=False, hess=False),
        # the largest: the headline workload's points in the default (FP64) form
        dict(name="laplace-cube-2m", kind="laplace", shape="cube", n=2000000, m=2000000, iprec=1, charge=True,
             dipole=True, mixed=False, host=False, plan=False, hess=False),
        # six more digits: high-order expansions
        dict(name="laplace-cube-1m-iprec2", kind="laplace", shape="cube", n=1000000, m=1000000, iprec=2, charge=True,
             dipole=True, mixed=False, host=False, plan=False, hess=False),
        # the mixed form (FP32 near field), at a size where every output can be checked by direct summation
        dict(name="laplace-mixed-cube-200k", kind="laplace", shape="cube", n=200003, m=200000, iprec=1, charge=True,
             dipole=True, mixed=True, host=False, plan=False, hess=False),
        # many independent problems of uneven size in one call (the batched workload), mixed form
        dict(name="laplace-batched-24", kind="batched", instances=24, smallest=1000, largest=200000, iprec=1,
             mixed=True),
        # Hessians on a strongly adaptive tree
        dict(name="laplace-hessian-plummer-40k", kind="laplace", shape="plummer", n=40000, m=25000, iprec=1,
             charge=True, dipole=False, mixed=False, host=False, plan=False, hess=True),
        # the Helmholtz workload: a surface of several wavelengths
        dict(name="helmholtz-sphere-1m", kind="helmholtz", shape="sphere", n=1000000, m=0, iprec=2, zr=8 * math.pi,
             zi=0.0, charge=True, dipole=False),
        # a small lossy Helmholtz call with targets and both kinds of source
        dict(name="helmholtz-cube-10k", kind="helmholtz", shape="cube", n=10007, m=5000, iprec=1, zr=6.0, zi=0.5,
             charge=True, dipole=True),
        # layer potentials on the benchmark's mesh
        dict(name="laplace-triangles-328k", kind="triangles", level=7, iprec=1, zr=0.0, squash=1.0),
        dict(name="helmholtz-triangles-20k", kind="triangles", level=5, iprec=1, zr=4 * math.pi, squash=1.0),
    ]


def _between(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    kind = rng.choice(["laplace", "laplace", "laplace", "plan", "batched", "helmholtz", "triangles"])
    if kind == "batched":
        return dict(kind="batched", instances=rng.randint(5, 24), smallest=_between(rng, 500, 3000),
                    largest=_between(rng, 20000, 200000), iprec=rng.choice([0, 1]), mixed=rng.random() < 0.7)
    if kind == "triangles":
        lap = rng.random() < 0.5
        return dict(kind="triangles", level=rng.randint(3, 7 if lap else 6), iprec=rng.choice([0, 1]),
                    zr=0.0 if lap else rng.uniform(1.0, 4 * math.pi), squash=rng.uniform(0.4, 1.0))
    if kind == "helmholtz":
        iprec = rng.choice([0, 1, 2])
        shape = rng.choice(["cube", "sphere"])
        n = _between(rng, 2000, 1000000 if shape == "sphere" and iprec < 2 else 300000)
        m = rng.choice([0, n // rng.randint(2, 9)])
        charge, dipole = rng.choice([(True, False), (True, True), (False, True)])
        return dict(kind="helmholtz", shape=shape, n=n, m=m, iprec=iprec, zr=rng.uniform(1.0, 8 * math.pi),
                    zi=rng.choice([0.0, rng.uniform(0.0, 2.0)]), charge=charge, dipole=dipole)
    plan = kind == "plan"
    shape = rng.choice(["cube", "sphere", "plummer"])
    mixed = rng.random() < 0.3
    iprec = rng.choice([-1, 0, 1] if mixed else [-1, 0, 1, 2, 3])
    # mixed results are held to direct sums, so those sizes stay where the sums are quick
    most = 200000 if mixed else {2: 500000, 3: 100000}.get(iprec, 2000000 if shape == "cube" else 400000)
    n = _between(rng, 2000, most)
    m = rng.choice([0, n, n // rng.randint(2, 9)])
    charge, dipole = rng.choice([(True, False), (True, False), (True, True), (False, True)])
    return dict(kind="laplace", shape=shape, n=n, m=m, iprec=iprec, charge=charge, dipole=dipole, mixed=mixed,
                host=not plan and n <= 200000 and rng.random() < 0.25, plan=plan, hess=False)


# ------------------------------------------------------------------ inputs

def _unit(n, g):
    v = torch.randn((n, 3), generator=g, dtype=torch.float64, device="cuda")
    return v / v.norm(dim=1, keepdim=True)


def _points(shape, n, g):
    if shape == "cube":
        return torch.rand((n, 3), generator=g, dtype=torch.float64, device="cuda")
    v = _unit(n, g)
    if shape == "sphere":
        return v
    if shape == "ellipsoid":
        return v * torch.tensor([0.9, 0.4, 0.6], dtype=torch.float64, device="cuda")
    # Plummer ball of core radius 0.1 inside the unit ball (the mass fraction inside is its cdf at 1)
    u = torch.rand(n, generator=g, dtype=torch.float64, device="cuda").clamp(1e-9, None) * (1 + 0.01) ** -1.5
    return v * (0.1 / torch.sqrt(u ** (-2 / 3) - 1))[:, None]


def _strength(n, g):
    return torch.rand((n, 2), generator=g, dtype=torch.float64, device="cuda") * 2 - 1


def _empty(n, width):
    return torch.empty((n, width), dtype=torch.float64, device="cuda")


def _sizes(case):
    """Instance sizes of a batch, spread evenly over their logarithm."""
    k, a, b = case["instances"], case["smallest"], case["largest"]
    return [int(a * (b / a) ** ((i + 0.5) / k)) for i in range(k)]


def _inputs(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    if case["kind"] == "triangles":
        # the mesh, turned and squashed by the seed
        tri = meshes.icosphere(case["level"], axes=(1.0, 1.0, case["squash"]))
        rng = np.random.default_rng(seed)
        turn, _ = np.linalg.qr(rng.normal(size=(3, 3)))
        if np.linalg.det(turn) < 0:
            turn[:, 0] = -turn[:, 0]
        tri = tri @ turn.T
        nrm, cen = meshes.normals_centroids(tri)
        n = len(tri)
        s = dict(tri=tri.reshape(n, 9), nrm=nrm, src=cen)
        s = {k: torch.from_numpy(np.ascontiguousarray(v)).cuda() for k, v in s.items()}
        return dict(s, q=_strength(n, g), d=_strength(n, g), v=None, trg=None)
    if case["kind"] == "batched":
        sizes = _sizes(case)
        src = torch.cat([_points(("cube", "plummer", "ellipsoid")[i % 3], k, g) for i, k in enumerate(sizes)])
        off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int32)
        return dict(src=src, q=_strength(len(src), g), d=None, v=None, trg=None, off=off)
    n, m = case["n"], case["m"]
    s = dict(src=_points(case["shape"], n, g), q=_strength(n, g) if case["charge"] else None, d=None, v=None)
    if case["dipole"]:
        s["d"], s["v"] = _strength(n, g), _unit(n, g)
    s["trg"] = _points(case["shape"], m, g) * 0.98 if m else None
    return s


def prepare(case, seed):
    s = _inputs(case, seed)
    s["case"] = case
    n = s["src"].shape[0]
    m = 0 if s["trg"] is None else s["trg"].shape[0]
    if case["kind"] == "laplace" and case["host"]:
        c = lambda t: None if t is None else torch.view_as_complex(t).cpu().numpy()  # noqa: E731
        h = lambda t: None if t is None else t.cpu().numpy()  # noqa: E731
        return dict(case=case, src=h(s["src"]), q=c(s["q"]), d=c(s["d"]), v=h(s["v"]), trg=h(s["trg"]))
    s["out"] = dict(pot=_empty(n, 2), fld=_empty(n, 6))
    if m:
        s["out"].update(pottarg=_empty(m, 2), fldtarg=_empty(m, 6))
    if case["kind"] == "laplace" and case["hess"]:
        s["out"]["hess"] = _empty(n, 12)
        if m:
            s["out"]["hesstarg"] = _empty(m, 12)
    if case["kind"] == "laplace" and case["plan"]:
        F.set_precision_thread(1 if case["mixed"] else 0)
        s["plan"] = F.LaplacePlan(case["iprec"], s["src"], int(case["charge"]), int(case["dipole"]), 1, 1, s["trg"],
                                  int(m > 0), int(m > 0), stream=torch.cuda.current_stream().cuda_stream)
    return s


# ------------------------------------------------------------------ one pass

def run(s):
    case = s["case"]
    stream = torch.cuda.current_stream().cuda_stream
    F.set_precision_thread(1 if case.get("mixed") else 0)
    if case["kind"] == "laplace" and case["host"]:
        t = int(s["trg"] is not None)
        got = F.lfmm3dparttarg(case["iprec"], s["src"], int(case["charge"]), s["q"], int(case["dipole"]), s["d"],
                               s["v"], 1, 1, s["trg"], t, t)
        ier, out = got[0], dict(zip(("pot", "fld", "pottarg", "fldtarg"), got[1:] if t else got[1:3]))
    else:
        out = s["out"]
        if case["kind"] == "batched":
            ier = F.lfmm3dparttarg_batched_device(case["iprec"], s["off"], s["src"], s["q"], None, None, out["pot"],
                                                  out["fld"], stream=stream)
        elif case["kind"] == "triangles" and case["zr"]:
            ier = F.hfmm3dtriatarg_device(case["iprec"], case["zr"], s["tri"], s["nrm"], s["src"], s["q"], s["d"],
                                          out["pot"], out["fld"], stream=stream)
        elif case["kind"] == "triangles":
            ier = F.lfmm3dtriatarg_device(case["iprec"], s["tri"], s["nrm"], s["src"], s["q"], s["d"], out["pot"],
                                          out["fld"], stream=stream)
        elif case["kind"] == "helmholtz":
            ier = F.hfmm3dparttarg_device(case["iprec"], complex(case["zr"], case["zi"]), s["src"], s["q"], s["d"],
                                          s["v"], out["pot"], out["fld"], s["trg"], out.get("pottarg"),
                                          out.get("fldtarg"), stream=stream)
        elif case["plan"]:
            ier = s["plan"].execute(s["q"], s["d"], s["v"], out["pot"], out["fld"], out.get("pottarg"),
                                    out.get("fldtarg"), use_graph=True, stream=stream)
        elif case["hess"]:
            ier = F.lfmm3dparttarg_hess_device(case["iprec"], s["src"], s["q"], s["d"], s["v"], out["pot"],
                                               out["fld"], out["hess"], s["trg"], out.get("pottarg"),
                                               out.get("fldtarg"), out.get("hesstarg"), stream=stream)
        else:
            ier = F.lfmm3dparttarg_device(case["iprec"], s["src"], s["q"], s["d"], s["v"], out["pot"], out["fld"],
                                          s["trg"], out.get("pottarg"), out.get("fldtarg"), stream=stream)
    if ier:
        raise RuntimeError("ier=%d: %s" % (ier, F.last_error()))
    return out


# ------------------------------------------------------------------ the work of a pass

def work(case):
    """Inputs read and outputs written once; the near field's pairs and the expansions of the points.
    A pair counts 31 flops for a charge and as many for a dipole (twice that with an exponential)."""
    if case["kind"] == "batched":
        n, m, kinds = sum(_sizes(case)), 0, 1
    elif case["kind"] == "triangles":
        n, m, kinds = 20 * 4 ** case["level"], 0, 4
    else:
        n, m, kinds = case["n"], case["m"], int(case["charge"]) + int(case["dipole"])
    leaf = {-2: 40, -1: 50, 0: 80, 1: 160, 2: 400, 3: 800}[case["iprec"]] / 2.5
    digits = {-2: 0.3, -1: 1.3, 0: 2.3, 1: 3.3, 2: 6.3, 3: 9.3}[case["iprec"]]
    terms = (digits / 0.239 + 1) ** 2
    wave = 2 if case.get("zr") else 1
    near = min(27 * leaf, n) * (n + m) * 31 * kinds * wave
    far = (n * kinds + 2 * (n + m)) * terms * 8 * wave
    width = 3 + (15 if case["kind"] == "triangles" else 5 * kinds)
    out = 8 + (12 if case.get("hess") else 0)
    return {"bytes": 8.0 * (n * width + 3 * m + (n + m) * out), "flops": float(near + far)}


# ------------------------------------------------------------------ the same in 64 bits, by direct summation

def _laplace_sum(trg, src, q, d, v, own, hess):
    """Potentials, fields (minus the gradient) and, for charges, Hessians at trg; own: trg is src, each
    point without itself."""
    m, n = trg.shape[0], src.shape[0]
    pot, fld, hs = trg.new_zeros((m, 2)), trg.new_zeros((m, 3, 2)), trg.new_zeros((m, 6, 2)) if hess else None
    dv = None if d is None else (v[:, :, None] * d[:, None, :]).reshape(n, 6)
    for i in range(0, m, SIDE):
        t = trg[i:i + SIDE]
        for j in range(0, n, SIDE):
            c = slice(j, j + SIDE)
            r = [t[:, a, None] - src[None, c, a] for a in range(3)]
            r2 = (r[0] * r[0]).addcmul_(r[1], r[1]).addcmul_(r[2], r[2])
            if own and -r2.shape[0] < i - j < r2.shape[1]:
                r2.diagonal(i - j).fill_(math.inf)
            u = r2.rsqrt_()
            u2 = u * u
            u3 = u2 * u
            if q is not None:
                pot[i:i + SIDE].addmm_(u, q[c])
                for a in range(3):
                    fld[i:i + SIDE, a] += (r[a] * u3) @ q[c]
                if hess:
                    u5 = u3 * u2 * 3
                    for k, (a, b) in enumerate(((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))):
                        w = r[a] * r[b] * u5
                        hs[i:i + SIDE, k] += ((w - u3) if a == b else w) @ q[c]
            if d is not None:
                w = (r[0] * v[None, c, 0]).addcmul_(r[1], v[None, c, 1]).addcmul_(r[2], v[None, c, 2]).mul_(u3)
                pot[i:i + SIDE].addmm_(w, d[c])
                fld[i:i + SIDE] -= (u3 @ dv[c]).reshape(-1, 3, 2)
                w.mul_(u2).mul_(3)
                for a in range(3):
                    fld[i:i + SIDE, a] += r[a].mul_(w) @ d[c]
    return (pot, fld.reshape(m, 6)) + ((hs.reshape(m, 12),) if hess else ())


def _helmholtz_sum(trg, src, zk, q, d, v, own):
    m, n = trg.shape[0], src.shape[0]
    c = lambda t: None if t is None else torch.view_as_complex(t)  # noqa: E731
    q, d = c(q), c(d)
    pot = torch.zeros(m, dtype=torch.complex128, device="cuda")
    fld = torch.zeros((m, 3), dtype=torch.complex128, device="cuda")
    for i in range(0, m, SIDE // 2):
        e = slice(i, i + SIDE // 2)
        for j in range(0, n, SIDE // 2):
            f = slice(j, j + SIDE // 2)
            x = trg[e, None, :] - src[None, f, :]
            r2 = (x * x).sum(-1)
            if own and i == j:
                r2.diagonal().fill_(1.0)
            r = r2.sqrt()
            g = torch.exp(1j * zk * r) / r
            if own and i == j:
                g.diagonal().zero_()
            a = (1 / r2 - 1j * zk / r) * g
            if q is not None:
                pot[e] += g @ q[f]
                fld[e] += torch.einsum("ij,ija,j->ia", a, x.to(a.dtype), q[f])
            if d is not None:
                s = (x * v[None, f, :]).sum(-1)
                pot[e] += (s * a) @ d[f]
                b = (zk * zk * g - 3 * a) / r2 * s
                fld[e] -= a @ (d[f, None] * v[f]) + torch.einsum("ij,ija,j->ia", b, x.to(a.dtype), d[f])
    return torch.view_as_real(pot), torch.view_as_real(fld).reshape(m, 6)


def exact(case, seed):
    if case["kind"] == "triangles":
        return None     # integrals over panels, singular ones among them: no plain sum gives them
    if case["kind"] == "batched":
        sizes = _sizes(case)
        if sum(k * k for k in sizes) > PAIRS_EXACT:
            return None
    elif case["n"] * (case["n"] + case["m"]) * (1 if case["kind"] == "laplace" else 8) > PAIRS_EXACT:
        return None
    s = _inputs(case, seed)
    if case["kind"] == "batched":
        got = [_laplace_sum(x, x, q, None, None, True, False)
               for x, q in zip(s["src"].split(sizes), s["q"].split(sizes))]
        return dict(pot=torch.cat([g[0] for g in got]), fld=torch.cat([g[1] for g in got]))
    out = {}
    for own, at, word in ((True, s["src"], ""), (False, s["trg"], "targ")):
        if at is None:
            continue
        if case["kind"] == "helmholtz":
            got = _helmholtz_sum(at, s["src"], complex(case["zr"], case["zi"]), s["q"], s["d"], s["v"], own)
        else:
            got = _laplace_sum(at, s["src"], s["q"], s["d"], s["v"], own, case["hess"])
        out.update(zip(("pot" + word, "fld" + word, "hess" + word), got))
    if case["kind"] == "laplace" and case["host"]:
        out = {k: torch.view_as_complex(v.reshape(v.shape[0], -1, 2)).squeeze(-1).cpu().numpy() for k, v in out.items()}
    return out
