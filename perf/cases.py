"""Performance cases of the view-factor assembly: what a user's program has it compute.

A case is a mesh (plates, cube enclosure, cylinder or 2-D cavity, from the package's own seeded
builders), a method (quadrature, Duffy, Monte Carlo) and the way the program calls it:

* "resident"  the mesh is on the device and stays there; every pass is one ``DeviceMesh.solve``
              that leaves F on the device and returns areas, group factors and row sums;
* "call"      the whole ``compute_view_factors`` call, host mesh to host result;
* "server"    a burst of requests submitted to a ``Server``; each result is copied on the device
              and released when it finishes.

``listed()`` are the fixed cases, ``draw()`` gives further ones of the same ranges, ``exact()`` the
same quantities in 64 bits from plain torch.
"""
from __future__ import annotations

import ctypes
import importlib.util
import math
import sys
from pathlib import Path

import numpy as np
import torch

ROOT = Path(__file__).resolve().parent.parent
PKG_DIR = ROOT / "radiativeviewfactor.jl_b200"
BOX_GROUP = 7          # cube enclosures carry their box as this group
CIRCLES = [5, 6, 7, 8]  # groups of the cavity's circles


def _package():
    if "rvf_b200" not in sys.modules:
        spec = importlib.util.spec_from_file_location("rvf_b200", PKG_DIR / "__init__.py",
                                                      submodule_search_locations=[str(PKG_DIR)])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["rvf_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["rvf_b200"]


def _case(name, how, geo, size, family, box, method, nquad, precision, geometric=False, self_vf=False):
    c = {"how": how, "geo": geo, "size": size, "family": family, "box": box, "method": method, "nquad": nquad,
         "precision": precision, "geometric": geometric, "self_vf": self_vf}
    return {"name": name, **c} if name else c


def listed():
    return [
        # A small part inside an outer loop (design or time stepping): latency and launches.
        _case("cube192-fp64", "resident", "cube", 4, "tri3", 2, "quadrature", 3, "fp64"),
        # Two coaxial plates, 800 Quad4, nquad 4: the analytic check and the smallest benchmark configuration.
        _case("plates800-fp64", "resident", "plates", 20, "quad4", 0, "quadrature", 4, "fp64"),
        # A one-off script: mesh in, ViewFactorResult out, everything between inside the pass.
        _case("call-cube1728-mixed", "call", "cube", 12, "tri3", 4, "quadrature", 3, "mixed"),
        # An ordinary occluded enclosure at the default precision.
        _case("cube6912-fp64", "resident", "cube", 24, "tri3", 12, "quadrature", 3, "fp64"),
        # The headline enclosure, 43,200 elements with a box, in both precisions: the largest solves.
        _case("cube43200-mixed", "resident", "cube", 60, "tri3", 12, "quadrature", 3, "mixed"),
        _case("cube43200-fp64", "resident", "cube", 60, "tri3", 12, "quadrature", 3, "fp64"),
        # Quadratic quads with 16 points, true obstruction vertices, a count that is no multiple of a tile.
        _case("quad8214-mixed-geo", "resident", "cube", 37, "quad", 8, "quadrature", 4, "mixed", geometric=True),
        # Closed cylinder of Quad8 with shared edges: Duffy integrals for the touching pairs.
        _case("cylinder3072-duffy", "resident", "cylinder", 64, "quad", 0, "duffy", 5, "fp64"),
        # 2-D cavity with four circles in the way, stratified Monte Carlo of 64 samples.
        _case("cavity4000-mc64", "resident", "cavity", 800, "line3", 4, "mc", 64, "fp64"),
        # The same cavity by quadrature.
        _case("cavity4000-quad", "resident", "cavity", 800, "line3", 4, "quadrature", 4, "fp64"),
        # Surface Monte Carlo with a box in the way, as a fifth of a service's requests are.
        _case("cube2166-mc64", "resident", "cube", 19, "quad4", 8, "mc", 64, "fp64"),
        # A service: sixteen meshes of several geometries, families and rules at once.
        _case("server-burst16", "server", "mix", 16, "mix", 8, "mix", 0, "mixed"),
    ]


def draw(rng):
    kind = rng.choice(["cube", "cube", "cube", "plates", "cylinder", "duffy", "cavity", "cavity-mc", "surface-mc",
                       "call", "server"])
    fam = rng.choice(["tri3", "tri", "quad4", "quad"])
    prec = rng.choice(["fp64", "mixed"])
    if kind == "server":
        return _case(None, "server", "mix", rng.randrange(6, 20), "mix", rng.randrange(2, 10), "mix", 0, "mixed")
    if kind == "surface-mc":
        samples = rng.choice([16, 30, 64])
        n = _log_uniform(rng, 1e5, 2e8)
        per = 12 if fam in ("tri3", "tri") else 6
        m = max(2, round(math.sqrt(math.sqrt(2 * n / samples) / per)))
        return _case(None, "resident", "cube", m, fam, rng.randrange(2, 10), "mc", samples, "fp64",
                     geometric=rng.random() < 0.3)
    if kind == "cavity-mc":
        samples = rng.choice([16, 30, 64, 100])
        n = _log_uniform(rng, 1e5, 5e8)
        return _case(None, "resident", "cavity", max(4, round(math.sqrt(2 * n / samples) / 5)), "line3", 4, "mc",
                     samples, "fp64")
    nquad = rng.choice([2, 3, 4, 5])
    if kind == "cavity":
        n = _log_uniform(rng, 1e5, 3e8)
        return _case(None, "resident", "cavity", max(4, round(math.sqrt(2 * n) / nquad / 5)), "line3",
                     rng.choice([0, 4]), "quadrature", nquad, "fp64")
    if kind in ("cylinder", "duffy"):
        n = _log_uniform(rng, 1e6, 4e9)
        nc = max(8, round(math.sqrt(math.sqrt(2 * n) / nquad ** 2 / 0.75) / 4) * 4)
        return _case(None, "resident", "cylinder", nc, "quad", 0, "duffy" if kind == "duffy" else "quadrature", nquad,
                     prec, self_vf=kind == "cylinder" and rng.random() < 0.3)
    n = _log_uniform(rng, 1e6, 3e8 if kind == "call" else 1.5e10)
    per = (2 if fam in ("tri3", "tri") else 1) * (2 if kind == "plates" else 6)
    m = max(2, min(60, round(math.sqrt(math.sqrt(2 * n) / _points_per_element(fam, nquad) / per))))
    box = 0 if kind == "plates" or rng.random() < 0.3 else rng.randrange(2, 13)
    return _case(None, "call" if kind == "call" else "resident", "plates" if kind == "plates" else "cube", m, fam, box,
                 "quadrature", nquad, prec, geometric=box > 0 and rng.random() < 0.3)


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _points_per_element(family, nquad):
    if family in ("tri3", "tri"):
        return {1: 1, 2: 3, 3: 7}.get(nquad, 13)
    return nquad if family == "line3" else nquad * nquad


# ----------------------------------------------------------------------------
# inputs
# ----------------------------------------------------------------------------
def _mesh(case, seed):
    """The case's mesh for a seed: node jitter, plate distance or circle places are drawn from it."""
    M = _package().meshes
    seed = int(seed) % (1 << 31)
    geo, size, fam, box = case["geo"], case["size"], case["family"], case["box"]
    if geo == "plates":
        return M.parallel_plates(size, fam, gap=float(np.random.default_rng(seed).uniform(0.5, 1.5))), []
    if geo == "cylinder":
        return M.cylinder(nc=size, na=max(2, size // 2), cap_rings=max(2, size // 8), jitter=0.01, seed=seed), []
    if geo == "cavity":
        return M.cavity_2d(n_wall=size, n_circle=max(4, size // 4), n_circles=4, seed=seed), CIRCLES if box else []
    md = M.cube_enclosure(size, family=fam, jitter=0.3, seed=seed, box=box > 0, box_edge=0.3, box_m=max(box, 1))
    return md, [BOX_GROUP] if box else []


def _options(case, seed):
    mc = case["method"] == "mc"
    return _package().make_options(3 if mc else case["nquad"], monte_carlo=mc,
                                   n_samples=case["nquad"] if mc else 10000, use_duffy=case["method"] == "duffy",
                                   seed=int(seed), precision=case["precision"], geometric_soup=case["geometric"],
                                   self_vf=case["self_vf"])


def _burst(case, seed):
    """The requests of a server case: a fixed mix of geometries, families, rules and sizes (300 to
    2,600 elements; a third occluded, every fifth Monte Carlo), the meshes jittered by the seed."""
    out = []
    for k in range(case["size"]):
        fam = ["tri3", "quad4", "quad"][k % 3]
        n = 300 * (2600 / 300) ** (((7 * k) % case["size"]) / max(1, case["size"] - 1))
        mc = k % 5 == 3
        if k % 4 == 1:
            c = _case(None, "resident", "cylinder", max(8, round(math.sqrt(n / 0.75) / 4) * 4), "quad", 0,
                      "quadrature", 2 + k % 3, "mixed")
        elif k % 4 == 2:
            per = 4 if fam == "tri3" else 2
            c = _case(None, "resident", "plates", max(2, round(math.sqrt(n / per))), fam, 0, "quadrature", 2 + k % 3,
                      "mixed")
        else:
            per = 12 if fam == "tri3" else 6
            c = _case(None, "resident", "cube", max(2, round(math.sqrt(n / per))), fam,
                      case["box"] if k % 3 == 0 else 0, "quadrature", 2 + k % 3, "mixed")
        if mc:
            c.update(method="mc", nquad=64, precision="fp64")
        out.append((c, int(seed) + 1000 * k))
    return out


class _DeviceF:
    """F of a mesh on the device for torch, without a copy: element [j, i] is F[i, j].  It holds the
    mesh, whose memory it is."""

    def __init__(self, pointer, n, owner):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (n, n), "typestr": "<f8", "version": 3,
                                         "data": (ctypes.cast(pointer, ctypes.c_void_p).value, False)}


def _device_f(pointer, n, owner):
    return torch.as_tensor(_DeviceF(pointer, n, owner), device="cuda")


_SERVER = []  # one server on the session, as a service keeps it


def prepare(case, seed):
    rvf = _package()
    torch.cuda.current_device()
    session = rvf.B200Backend().session
    if case["how"] == "server":
        if not _SERVER:
            from rvf_b200 import _abi
            _SERVER.append(_abi.Server(session))
        reqs = []
        for c, s in _burst(case, seed):
            md, obs = _mesh(c, s)
            reqs.append((rvf.mesh_desc_arrays(md, obs), _options(c, s), md.n_elems))
        return {"case": case, "server": _SERVER[0], "requests": reqs}
    md, obs = _mesh(case, seed)
    if case["how"] == "call":
        return {"case": case, "mesh": md, "obstructions": obs, "seed": int(seed)}
    n, g = md.n_elems, len(md.group_tags)
    return {"case": case, "mesh": rvf.DeviceMesh(session, rvf.mesh_desc_arrays(md, obs)),
            "options": _options(case, seed), "A": np.empty(n), "F_group": np.empty((g, g), order="F"),
            "A_group": np.empty(g), "row_sums": np.empty(n)}


def run(state):
    """One pass.  "F" is the transpose of F_elem (the device and host layout is column-major)."""
    case = state["case"]
    if case["how"] == "call":
        r = _package().compute_view_factors(state["mesh"], nquad=case["nquad"], seed=state["seed"], verbose=False,
                                            obstruction_groups=state["obstructions"], precision=case["precision"],
                                            geometric_soup=case["geometric"], self_vf=case["self_vf"])
        return {"F": r.F_elem.T, "A": r.A_elem, "F_group": r.F_group, "A_group": r.A_group}
    if case["how"] == "server":
        server, out = state["server"], {}
        ids = {server.submit(desc, opts): (k, n) for k, (desc, opts, n) in enumerate(state["requests"])}
        while ids:
            rid = server.wait_any()
            k, n = ids.pop(rid)
            out[k] = _device_f(server.result_device(rid), n, None).clone()
            torch.cuda.current_stream().synchronize()  # the request's memory is given back next
            server.release(rid)
        return [out[k] for k in sorted(out)]
    dm = state["mesh"]
    dm.solve(state["options"], None, state["A"], state["F_group"], state["A_group"], state["row_sums"])
    return {"F": _device_f(dm.result_device(), dm.n_elems, dm), "A": state["A"], "F_group": state["F_group"],
            "A_group": state["A_group"], "row_sums": state["row_sums"]}


# ----------------------------------------------------------------------------
# work
# ----------------------------------------------------------------------------
def _elements(case):
    size, tri = case["size"], case["family"] in ("tri3", "tri")
    if case["geo"] == "plates":
        return 2 * size * size * (2 if tri else 1)
    if case["geo"] == "cylinder":
        return size * max(2, size // 2) + 2 * size * max(2, size // 8)
    if case["geo"] == "cavity":
        return 4 * size + 4 * max(4, size // 4)
    return 6 * size * size * (2 if tri else 1)


def work(case):
    """Bytes: F written once (plus what describes the mesh).  Flops: 23 per 3-D point pair, 26 per 2-D one (kernel
    and sum), 118 / 260 per line / surface Monte Carlo sample pair (two element evaluations, kernel, sum); point
    pairs of elements in one plane are left out (half of the plates', a sixth of the cube's).  The shadow rays a
    solve cannot do without depend on the geometry and are left out too."""
    if case["how"] == "server":
        parts = [work(c) for c, _ in _burst(case, 0)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    n = _elements(case)
    pairs = n * (n - 1) / 2
    if case["method"] == "mc":
        flops = pairs * case["nquad"] * (118 if case["geo"] == "cavity" else 260)
    else:
        facing = {"plates": 0.5, "cube": 5 / 6}.get(case["geo"], 1.0)
        flops = pairs * facing * _points_per_element(case["family"], case["nquad"]) ** 2 * (
            26 if case["geo"] == "cavity" else 23)
    return {"bytes": 8.0 * n * n + 200.0 * n, "flops": flops}


# ----------------------------------------------------------------------------
# the same quantities in 64 bits, from the definitions
# ----------------------------------------------------------------------------
_DEV = "cuda" if torch.cuda.is_available() else "cpu"
_ROOM = 4_000_000 if _DEV == "cuda" else 200_000  # values of one temporary
_CORNERS = {0: 4, 1: 3, 2: 4, 3: 3, 4: 2, 5: 2}


def _t(a, dtype=torch.float64):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=dtype, device=_DEV)


def _shape(fam, x, e):
    """Shape functions and their derivatives at (x, e), stacked along the last axis."""
    if fam == 0:
        sx, se = (-1, 1, 1, -1), (-1, -1, 1, 1)
        N, dx, de = [], [], []
        for a, b in zip(sx, se):
            N.append(0.25 * (1 + a * x) * (1 + b * e) * (a * x + b * e - 1))
            dx.append(0.25 * a * (1 + b * e) * (2 * a * x + b * e))
            de.append(0.25 * b * (1 + a * x) * (a * x + 2 * b * e))
        for k, b in ((0, -1), (1, 1), (2, 1), (3, -1)):
            if k in (0, 2):
                N.append(0.5 * (1 - x * x) * (1 + b * e))
                dx.append(-x * (1 + b * e))
                de.append(0.5 * b * (1 - x * x))
            else:
                N.append(0.5 * (1 + b * x) * (1 - e * e))
                dx.append(0.5 * b * (1 - e * e))
                de.append(-e * (1 + b * x))
    elif fam == 1:
        l1 = 1 - x - e
        one = torch.ones_like(x)
        N = [l1 * (2 * l1 - 1), x * (2 * x - 1), e * (2 * e - 1), 4 * l1 * x, 4 * x * e, 4 * l1 * e]
        dx = [1 - 4 * l1, 4 * x - 1, 0 * one, 4 * (l1 - x), 4 * e, -4 * e]
        de = [1 - 4 * l1, 0 * one, 4 * e - 1, -4 * x, 4 * x, 4 * (l1 - e)]
    elif fam == 2:
        N, dx, de = [], [], []
        for a, b in ((-1, -1), (1, -1), (1, 1), (-1, 1)):
            N.append(0.25 * (1 + a * x) * (1 + b * e))
            dx.append(0.25 * a * (1 + b * e))
            de.append(0.25 * b * (1 + a * x))
    elif fam == 3:
        one = torch.ones_like(x)
        N, dx, de = [1 - x - e, x, e], [-one, one, 0 * one], [-one, 0 * one, one]
    else:
        N, dx = [-0.5 * x * (1 - x), 0.5 * x * (1 + x), 1 - x * x], [x - 0.5, x + 0.5, -2 * x]
        de = dx
    return torch.stack(N, -1), torch.stack(dx, -1), torch.stack(de, -1)


def _evaluate(fam, nodes, x, e):
    """Points, unit normals and area elements; nodes (..., k, 3), x and e of the leading shape."""
    N, dx, de = (v.unsqueeze(-1) for v in _shape(fam, x, e))
    p, a = (N * nodes).sum(-2), (dx * nodes).sum(-2)
    if fam == 4:
        d = a.norm(dim=-1)
        u = a / d.unsqueeze(-1)
        return p, torch.stack([-u[..., 1], u[..., 0], torch.zeros_like(d)], -1), d
    c = torch.linalg.cross(a, (de * nodes).sum(-2))
    d = c.norm(dim=-1)
    return p, c / d.unsqueeze(-1), d


def _rule(fam, nquad):
    if fam in (1, 3):
        if nquad == 2:
            return [1 / 6, 2 / 3, 1 / 6], [1 / 6, 1 / 6, 2 / 3], [1 / 6] * 3
        orbit = (lambda a, w: [(a, a, w), (1 - 2 * a, a, w), (a, 1 - 2 * a, w)])
        if nquad == 3:  # Dunavant, degree 5
            pts = (orbit(0.101286507323456, 0.125939180544827) + orbit(0.470142064105115, 0.132394440720100)
                   + [(1 / 3, 1 / 3, 0.225)])
        else:  # Dunavant, degree 7
            a, b = 0.048690315425316, 0.312865496004875
            c, w = 1 - a - b, 0.077113760890257
            pts = (orbit(0.260345966079038, 0.175615257433204) + orbit(0.065130102902216, 0.053347235608839)
                   + [(u, v, w) for u, v in ((a, b), (b, a), (a, c), (c, a), (b, c), (c, b))]
                   + [(1 / 3, 1 / 3, -0.149570044467670)])
        x, e, w = zip(*pts)
        return x, e, [v / 2 for v in w]
    p, w = np.polynomial.legendre.leggauss(nquad)
    if fam == 4:
        return p, 0 * p, w
    return np.tile(p, nquad), np.repeat(p, nquad), np.outer(w, w).ravel()


def _nodes(md):
    fam = int(md.elem_family[0])
    k = {0: 8, 1: 6, 2: 4, 3: 3, 4: 3}[fam]
    return fam, _t(md.coords.T)[_t(md.elem_nodes[:, :k] - 1, torch.int64)]


class _Obstruction:
    """The obstruction's primitives in leaves of at most 8 (median splits of the longest axis), as the
    reference's tree has them: a primitive is tested by the rays that pass its leaf's box."""

    def __init__(self, md, groups, geometric):
        soup = np.concatenate([md.group_tri_soup[g] for g in groups])
        tag = np.concatenate([np.full(len(md.group_tri_soup[g]), g) for g in groups])
        lo, hi, mid = soup.min(1), soup.max(1), soup.mean(1)
        leaves, todo = [], [np.arange(len(soup))]
        while todo:
            idx = todo.pop()
            if len(idx) <= 8:
                leaves.append(idx)
                continue
            axis = int(np.argmax(hi[idx].max(0) - lo[idx].min(0)))
            idx = idx[np.argsort(mid[idx, axis], kind="stable")]
            half = (len(idx) + 1) // 2
            todo += [idx[:half], idx[half:]]
        pad = np.array([list(v) + [v[0]] * (8 - len(v)) for v in leaves])
        self.lo = _t(np.array([lo[v].min(0) for v in leaves]))
        self.hi = _t(np.array([hi[v].max(0) for v in leaves]))
        # the reference reads a stored triangle transposed unless true vertices are asked for
        self.prim = _t((soup if geometric or soup.shape[1] == 2 else soup.transpose(0, 2, 1))[pad])
        self.tag = _t(tag[pad], torch.int64)
        self.size = len(leaves)

    def _passing(self, test, n):
        """(ray, leaf) indices of the rays that pass leaf boxes, in parts; the root's box first."""
        alive = torch.nonzero(test(slice(None), self.lo.amin(0), self.hi.amax(0))[:, 0]).squeeze(1)
        step = max(1, _ROOM // self.size)
        for at in range(0, len(alive), step):
            some = alive[at:at + step]
            r, leaf = torch.nonzero(test(some, self.lo, self.hi), as_tuple=True)
            for b in range(0, len(r), _ROOM // 8):
                yield some[r[b:b + _ROOM // 8]], leaf[b:b + _ROOM // 8]

    def blocked(self, p, q, gp, gq):
        """Whether the segments p -> q (n, 3) are blocked by a primitive of another group than gp, gq."""
        hit = torch.zeros(len(p), dtype=torch.bool, device=p.device)
        if not len(p):
            return hit
        if self.prim.shape[2] == 2:
            s, e = torch.minimum(p, q)[:, None, :2], torch.maximum(p, q)[:, None, :2]
            test = (lambda r, lo, hi: ((lo[..., :2] <= e[r]) & (hi[..., :2] >= s[r])).all(-1))
            for r, leaf in self._passing(test, len(p)):
                g, a, b = self.tag[leaf], p[r][:, None], q[r][:, None]
                v0, v1 = self.prim[leaf].unbind(2)
                d, f = b - a, v1 - v0
                den = d[..., 0] * f[..., 1] - d[..., 1] * f[..., 0]
                w = v0 - a
                s1 = (w[..., 0] * f[..., 1] - w[..., 1] * f[..., 0]) / den
                t1 = (w[..., 0] * d[..., 1] - w[..., 1] * d[..., 0]) / den
                ok = (den.abs() >= 1e-8) & (s1 > 1e-8) & (s1 < 1 - 1e-8) & (t1 > 1e-8) & (t1 < 1 - 1e-8)
                ok &= (g != gp[r][:, None]) & (g != gq[r][:, None])
                hit[r[ok.any(1)]] = True
            return hit
        d = q - p
        far = d.norm(dim=1)
        d = d / far[:, None]
        inv = 1 / d

        def test(r, lo, hi):
            t1, t2 = (lo - p[r][:, None]) * inv[r][:, None], (hi - p[r][:, None]) * inv[r][:, None]
            near = torch.minimum(t1, t2).amax(-1).clamp(min=0)
            return near <= torch.minimum(torch.maximum(t1, t2).amin(-1), far[r][:, None])

        for r, leaf in self._passing(test, len(p)):
            g, o, u = self.tag[leaf], p[r][:, None], d[r][:, None].expand(-1, 8, -1)
            v0, v1, v2 = self.prim[leaf].unbind(2)
            e1, e2, s = v1 - v0, v2 - v0, o - v0
            h = torch.linalg.cross(u, e2)
            a = (e1 * h).sum(-1)
            x = (s * h).sum(-1) / a
            k = torch.linalg.cross(s, e1)
            y, t = (u * k).sum(-1) / a, (e2 * k).sum(-1) / a
            ok = (a.abs() >= 1e-10) & (x >= 0) & (x <= 1) & (y >= 0) & (x + y <= 1)
            ok &= (t > float(np.float32(1e-6))) & (t < far[r][:, None])
            ok &= (g != gp[r][:, None]) & (g != gq[r][:, None])
            hit[r[ok.any(1)]] = True
        return hit


def _kernel(p, n, q, m, dim):
    """cos cos / (pi r^2), in the plane cos cos / (2 r), zero where a cosine is not positive."""
    r = q - p
    r2 = (r * r).sum(-1)
    ci, cj = (n * r).sum(-1), -(m * r).sum(-1)
    K = ci * cj / (math.pi * r2 * r2 if dim == 2 else 2 * r2 * r2.sqrt())
    return torch.where((ci > 0) & (cj > 0) & (r2 >= 1e-30), K, torch.zeros_like(K))


def _raw_quadrature(md, obs, nquad, self_vf):
    fam, nodes = _nodes(md)
    rx, re, rw = (_t(v) for v in _rule(fam, nquad))
    P, n = len(rx), len(nodes)
    x, nrm, dA = _evaluate(fam, nodes[:, None], rx.expand(n, P), re.expand(n, P))
    w = dA * rw
    raw = torch.zeros(n, n, dtype=torch.float64, device=_DEV)
    tag = _t(md.elem_group, torch.int64)
    wide = max(1, min(n, _ROOM // (P * P)))
    for j0 in range(0, n, wide):
        j1 = min(n, j0 + wide)
        tall = max(1, _ROOM // (P * P * (j1 - j0)))
        for i0 in range(0, j1, tall):
            i1 = min(j1, i0 + tall)
            p, q = x[i0:i1, None, :, None], x[None, j0:j1, None, :]
            K = _kernel(p, nrm[i0:i1, None, :, None], q, nrm[None, j0:j1, None, :], md.mesh_dim)
            keep = torch.arange(i0, i1, device=_DEV)[:, None] < torch.arange(j0, j1, device=_DEV) + int(self_vf)
            K *= keep[:, :, None, None]
            if obs is not None:
                a, b, u, v = torch.nonzero(K, as_tuple=True)
                # rays leave the element with the lower index
                a2, b2 = a + i0, b + j0
                K[a, b, u, v] *= ~obs.blocked(x[a2, u], x[b2, v], tag[a2], tag[b2])
            raw[i0:i1, j0:j1] = torch.einsum("abuv,au,bv->ab", K, w[i0:i1], w[j0:j1])
    return raw.triu(0 if self_vf else 1), w.sum(1)


_GOLDEN, _M1, _M2 = (v - (1 << 64) for v in (0x9E3779B97F4A7C15, 0xBF58476D1CE4E5B9, 0x94D049BB133111EB))


def _shr(z, k):
    return (z >> k) & ((1 << (64 - k)) - 1)


def _stream(seed, tid):
    """splitmix64 of the pair's number, then xorshift64 draws in [0, 1]."""
    seed = int(seed) & ((1 << 64) - 1)
    z = tid * _GOLDEN + (seed - (1 << 64) if seed >> 63 else seed)
    z = (z ^ _shr(z, 30)) * _M1
    z = (z ^ _shr(z, 27)) * _M2
    z = z ^ _shr(z, 31)
    while True:
        z = z ^ (z << 13)
        z = z ^ _shr(z, 7)
        z = z ^ (z << 17)
        yield _shr(z, 11).double() / float((1 << 53) - 1)


def _mc_samples(md, i, j, samples, seed):
    """For each stratified sample of the pairs (i, j): points, normals and area elements of both elements."""
    fam, nodes = _nodes(md)
    n, s = len(nodes), math.isqrt(samples)
    draws = _stream(seed, i * n + j + 1)
    for k in range(samples):
        u = [next(draws) for _ in range(4)]
        if k < s * s:
            si, sj = divmod(k, s)
            u = [(si + u[0]) / s, (sj + u[1]) / s, ((sj if fam == 4 else si) + u[2]) / s, (sj + u[3]) / s]
        out = []
        for e, a, b in ((i, u[0], u[1]), (j, u[2], u[3])):
            if fam in (1, 3):
                flip = a + b > 1
                a, b = torch.where(flip, 1 - a, a), torch.where(flip, 1 - b, b)
            else:
                a, b = 2 * a - 1, 2 * b - 1
            out += _evaluate(fam, nodes[e], a, b)
        yield out


def _raw_mc(md, obs, samples, seed, exclude):
    n = md.n_elems
    measure = {0: 4.0, 2: 4.0, 1: 0.5, 3: 0.5, 4: 2.0}[int(md.elem_family[0])]
    tag = _t(md.elem_group, torch.int64) if exclude else torch.zeros(n, dtype=torch.int64, device=_DEV)
    raw = torch.zeros(n, n, dtype=torch.float64, device=_DEV)
    first = torch.arange(n - 1, device=_DEV)
    area = torch.zeros(n, dtype=torch.float64, device=_DEV)
    for p, a, da, q, b, db in _mc_samples(md, first, first + 1, samples, seed):
        area[:-1] += da
        area[-1] += db[-1]
    pairs = torch.triu_indices(n, n, 1, device=_DEV)
    for at in range(0, pairs.shape[1], _ROOM):
        i, j = pairs[:, at:at + _ROOM]
        total = torch.zeros(len(i), dtype=torch.float64, device=_DEV)
        for p, a, da, q, b, db in _mc_samples(md, i, j, samples, seed):
            K = _kernel(p, a, q, b, md.mesh_dim)
            if obs is not None:
                r = torch.nonzero(K).squeeze(1)
                K[r] *= ~obs.blocked(p[r], q[r], tag[i[r]], tag[j[r]])
            total += K * da * db
        raw[i, j] = total * measure ** 2 / samples
    return raw, area * measure / samples


def _duffy_points(region, vertex, r, a, b, c):
    """The four coordinates of a Duffy region on the touching corner (0, 0) or edge v = 0 of both unit squares."""
    if vertex:
        if region < 4:  # r on the first element
            du, dv = (r, r * a) if region < 2 else (r * a, r)
            ds, dt = (r * b, r * b * c) if region % 2 == 0 else (r * b * c, r * b)
        else:
            ds, dt = (r, r * a) if region < 6 else (r * a, r)
            du, dv = (r * b, r * b * c) if region % 2 == 0 else (r * b * c, r * b)
        return du, dv, ds, dt
    if region == 0:
        A = r * (1 - a * (1 - c))
        return A, r * a * b * c, A - r * a * (1 - b) * c + r * a * b * c, r * a * (1 - b) * c
    if region == 1:
        A = r * (1 - a * b * c)
        return A, r * a * c * (1 - b), A + r * a * b * c - r * a * c, r * a * b * c
    if region == 2:
        A = r * (1 - a * b)
        return A, r * a * b * c, A - r * a * b * (1 - c), r * a * b * (1 - c)
    h = r * (1 - a) * b * c
    if region == 3:
        return r * (b * c + a * (1 - b * c)), h, r * b * c, h
    return r * a * c, h, r * a * c * (1 - b) + r * a * b * c, h


def _add_duffy(md, raw, nquad):
    """Quad8 pairs that share a corner or an edge, integrated in Duffy coordinates."""
    fam, nodes = _nodes(md)
    corner = md.elem_nodes[:, :4]
    owners = {}
    for e, c in enumerate(corner):
        for v in c:
            owners.setdefault(int(v), []).append(e)
    touch = sorted({(i, j) for es in owners.values() for i in es for j in es if i < j})
    gp, gw = np.polynomial.legendre.leggauss(nquad)
    r, a, b, c = (v.reshape(-1) for v in torch.meshgrid(*[_t((gp + 1) / 2)] * 4, indexing="ij"))
    w = torch.einsum("a,b,c,d->abcd", *[_t(gw / 2)] * 4).reshape(-1) * r ** 3
    edge = {(1, 2): 1, (2, 3): 2, (3, 4): 3, (1, 4): 4}
    at = [(0.0, 0.0), (1.0, 0.0), (1.0, 1.0), (0.0, 1.0)]
    turn = {1: lambda u, v: (u, v), 2: lambda u, v: (1 - v, u), 3: lambda u, v: (1 - u, 1 - v),
            4: lambda u, v: (v, 1 - u)}
    kinds = {}
    for i, j in touch:
        m = [(x + 1, y + 1) for x in range(4) for y in range(4) if corner[i][x] == corner[j][y]]
        if len(m) == 1:
            key = (True, m[0][0], m[0][1])
        else:
            key = (False, *(edge.get(tuple(sorted((m[0][k], m[1][k]))), 1) for k in (0, 1)))
        kinds.setdefault(key, []).append((i, j))
    for (vertex, ki, kj), some in kinds.items():
        for s0 in range(0, len(some), max(1, _ROOM // (24 * len(r)))):
            part = _t(np.array(some[s0:s0 + max(1, _ROOM // (24 * len(r)))]), torch.int64)
            total = 0.0
            for region in range(8 if vertex else 5):
                u, v, s, t = _duffy_points(region, vertex, r, a, b, c)
                if vertex:
                    (u0, v0), (s0_, t0) = at[ki - 1], at[kj - 1]
                    u, v = (1 - u if u0 else u), (1 - v if v0 else v)
                    s, t = (1 - s if s0_ else s), (1 - t if t0 else t)
                else:
                    (u, v), (s, t) = turn[ki](u, v), turn[kj](s, t)
                ok = ((u >= 0) & (u <= 1) & (v >= 0) & (v <= 1) & (s >= 0) & (s <= 1) & (t >= 0) & (t <= 1)).double()
                u, v, s, t = ((2 * z - 1).expand(len(part), -1) for z in (u, v, s, t))
                one = _evaluate(fam, nodes[part[:, 0], None], u, v)
                two = _evaluate(fam, nodes[part[:, 1], None], s, t)
                K = _kernel(one[0], one[1], two[0], two[1], 2)
                total = total + (K * one[2] * two[2] * 16 * ok * w).sum(1)
            raw[part[:, 0], part[:, 1]] = total


def exact(case, seed):
    """What run() returns, in 64 bits; None for the largest solves, which would take minutes this way."""
    if case["how"] == "server":
        return [(exact(c, s) or {}).get("F") for c, s in _burst(case, seed)]
    n = _elements(case)
    per = case["nquad"] if case["method"] == "mc" else _points_per_element(case["family"], case["nquad"]) ** 2
    cost = n * (n - 1) / 2 * per * (5 if case["method"] == "mc" else 1) * (2 if case["box"] else 1)
    if cost > 5e9:
        return None
    md, groups = _mesh(case, seed)
    obs = _Obstruction(md, groups, case["geometric"]) if groups else None
    if case["method"] == "mc":
        raw, area = _raw_mc(md, obs, case["nquad"], seed, md.mesh_dim == 1)
    else:
        raw, area = _raw_quadrature(md, obs, case["nquad"], case["self_vf"])
        if case["method"] == "duffy":
            _add_duffy(md, raw, case["nquad"])
    F = (raw + raw.triu(1).T) / area[:, None]
    tags = sorted(md.group_tags)
    member = _t(md.elem_group[:, None] == np.array(tags)[None, :], torch.float64)
    A_group = member.T @ area
    out = {"F": F.T.contiguous(), "A": area, "F_group": (member.T @ (area[:, None] * (F @ member))) / A_group[:, None],
           "A_group": A_group, "row_sums": F.sum(1)}
    if case["how"] == "call":
        del out["row_sums"]
    return out
