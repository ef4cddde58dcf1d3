"""Performance cases: what programs ask of this library, through its public entry points.

Sizes are RWG counts N of the meshes that the configurations, tests and the
benchmark use (96 to 10,680 unknowns, 3 GHz, edges near a twentieth of a
wavelength).  A seed moves the frequency by up to one percent and draws the
incidences, impedances and vectors, so the impedance matrix, the right-hand
sides and the solution of another seed are others.  ``exact`` is the same
discretisation written again in torch at 64 bits: dense matrix, LU solves.
"""
import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "diffmom.jl_b200"))
import diffmom_b200 as dm  # noqa: E402
from diffmom_b200.mesh import make_geodesic_sphere  # noqa: E402
from diffmom_b200.workloads import impedance_surface_batch  # noqa: E402

C0 = dm.C0_DEFAULT
ETA0 = dm.ETA0_DEFAULT
FREQ = 3e9
LAM = C0 / FREQ
PREC_BYTES = {"fp64": 16, "mixed": 8}


# --------------------------------------------------------------------------
# the cases
# --------------------------------------------------------------------------
def listed():
    return [
        # the smallest solve (6 x 6 plate, 96 unknowns): a call's launches and host steps
        {"name": "direct_plate_96", "what": "scattering", "body": "plate", "a": 6, "b": 6, "precision": "fp64",
         "precond": "auto"},
        # solve_scattering's own choice below 2,000 unknowns: dense direct, FP64
        {"name": "direct_plate_1825", "what": "scattering", "body": "plate", "a": 25, "b": 25, "precision": "fp64",
         "precond": "auto"},
        # its choice up to 10,000: dense GMRES with the near-field factor, FP64, and the bistatic RCS cut
        # that the Mie checks take of this sphere
        {"name": "gmres_sphere_7680", "what": "scattering", "body": "sphere", "a": 16, "b": 0, "precision": "fp64",
         "precond": "auto", "cut": 181},
        # the same method in mixed precision, an oblong plate
        {"name": "gmres_plate_4693_mixed", "what": "scattering", "body": "plate", "a": 37, "b": 43,
         "precision": "mixed", "precond": "auto"},
        # a closed perturbed body with the learned preconditioner: about a hundred GMRES iterations
        {"name": "learned_ellipsoid_9720", "what": "scattering", "body": "ellipsoid", "a": 18, "b": 99,
         "precision": "mixed", "precond": "learned"},
        # its choice above 10,000: H-matrix build, near-field factor of its dense blocks, GMRES
        {"name": "aca_plate_10680", "what": "scattering", "body": "plate", "a": 60, "b": 60, "precision": "fp64",
         "precond": "auto"},
        # the benchmark's job: monostatic RCS of 1,024 incidences, mixed precision
        {"name": "sweep_plate_10680x1024", "what": "sweep", "body": "plate", "a": 60, "b": 60,
         "precision": "mixed", "waves": 1024, "currents": False},
        # an FP64 angle sweep of a mid-size plate, the currents wanted too
        {"name": "sweep_plate_4720x181_fp64", "what": "sweep", "body": "plate", "a": 40, "b": 40,
         "precision": "fp64", "waves": 181, "currents": True},
        # uneven impedance-loaded surfaces of 500 to 6,000 unknowns, one incidence each
        {"name": "surfaces_24", "what": "surfaces", "count": 24, "largest": 6000,
         "meshes": 20260004, "precision": "mixed"},
        # one step of an impedance design: forward, adjoint, gradient (quadrants of a plate)
        {"name": "design_plate_2640", "what": "design", "body": "plate", "a": 30, "b": 30, "precision": "fp64"},
        # the operator in a program's own iteration, entries recomputed per product
        {"name": "product_free_disk_4640", "what": "product", "body": "disk", "a": 20, "b": 80, "operator": "free"},
        # the impedance matrix itself, handed to the program
        {"name": "matrix_plate_1825", "what": "matrix", "body": "plate", "a": 25, "b": 25, "precision": "fp64"},
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _body(rng, lo, hi, disks=True):
    """A body with about lo..hi unknowns (log-uniform), odd sizes among them.
    Disks have slivers at the centre, which a 32-bit matrix does not resolve
    without impedance loading: they come in FP64."""
    n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    body = rng.choice(["plate", "plate", "disk", "sphere"] if disks else ["plate", "plate", "sphere"])
    if body == "plate":
        a = max(3, int(round(math.sqrt(n / 3) * rng.uniform(0.7, 1.0))))
        return {"body": body, "a": a, "b": max(3, min(int((hi + a) / (3 * a - 1)), int(round((n + a) / (3 * a - 1)))))}
    if body == "disk":
        nr = max(3, int((8 + math.sqrt(64 + 48 * n)) / 24))
        return {"body": body, "a": nr, "b": 4 * nr - rng.randrange(2)}
    return {"body": body, "a": max(3, int(math.sqrt(n / 30))), "b": 0}


def draw(rng):
    what = rng.choice(["direct", "gmres", "gmres", "learned", "aca", "sweep", "sweep", "surfaces", "design",
                       "product", "matrix"])
    precision = rng.choice(["fp64", "fp64", "mixed"])
    disks = precision == "fp64"
    if what == "direct":
        return {"what": "scattering", **_body(rng, 96, 2000, disks), "precision": precision, "precond": "auto"}
    if what == "gmres":
        return {"what": "scattering", **_body(rng, 2001, 9900, disks), "precision": precision, "precond": "auto",
                "cut": rng.choice([0, 91, 181])}
    if what == "learned":
        return {"what": "scattering", "body": "ellipsoid", "a": rng.randrange(9, 19), "b": rng.randrange(1, 200),
                "precision": "mixed", "precond": rng.choice(["learned", "local"])}
    if what == "aca":
        a = rng.randrange(50, 61)
        return {"what": "scattering", "body": "plate", "a": a, "b": rng.randrange(a - 20, (10700 + a) // (3 * a - 1)),
                "precision": "fp64", "precond": "auto", "method": "aca_gmres"}
    if what == "sweep":
        precision = rng.choice(["fp64", "mixed"])
        return {"what": "sweep", **_body(rng, 400, 4800 if precision == "fp64" else 10600, precision == "fp64"),
                "precision": precision, "waves": _spread(rng, 8, 256 if precision == "fp64" else 1000),
                "currents": rng.random() < 0.5}
    if what == "surfaces":
        return {"what": "surfaces", "count": _spread(rng, 4, 24), "largest": rng.randrange(1000, 6000),
                "meshes": rng.randrange(1 << 20), "precision": "mixed"}
    if what == "design":
        return {"what": "design", **_body(rng, 300, 4800), "precision": "fp64"}
    if what == "product":
        operator = rng.choice(["free", "dense", "mixed"])
        return {"what": "product", **_body(rng, 300, 9900), "operator": operator}
    return {"what": "matrix", **_body(rng, 96, 2000), "precision": precision}


# --------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------
def _mesh(case):
    a, b = case["a"], case["b"]
    h = LAM / 20
    if case["body"] == "plate":
        return dm.make_rect_plate(a * h, b * h, a, b)
    if case["body"] == "disk":
        return dm.make_circular_plate(a * h, a, b)
    if case["body"] == "sphere":
        return make_geodesic_sphere(0.5 * LAM, a)
    return dm.make_perturbed_ellipsoid(LAM, b, frequency=a)


def _waves(rng, k, count):
    """Plane waves from above: theta below 80 degrees, theta- or phi-polarised."""
    out = []
    for _ in range(count):
        th, ph = math.radians(rng.uniform(0, 80)), math.radians(rng.uniform(0, 360))
        back = np.array([math.sin(th) * math.cos(ph), math.sin(th) * math.sin(ph), math.cos(th)])
        pol = np.array([math.cos(th) * math.cos(ph), math.cos(th) * math.sin(ph), -math.sin(th)]) \
            if rng.integers(2) else np.array([-math.sin(ph), math.cos(ph), 0.0])
        out.append(dm.make_plane_wave(-k * back, 1.0, pol))
    return out


def _inputs(case, seed):
    """What both the library and exact() start from."""
    rng = np.random.default_rng(seed)
    freq = FREQ * rng.uniform(0.99, 1.01)
    k = 2 * math.pi * freq / C0
    s = {"case": case, "freq": freq, "k": k}
    if case["what"] == "surfaces":
        s["surfaces"] = impedance_surface_batch(case["count"], seed=case["meshes"], freq_hz=FREQ,
                                                n_range=(500, case["largest"]))
        for f in s["surfaces"]:
            f.excitation = _waves(rng, k, 1)[0]
            f.zs = rng.uniform(0, 200, f.mesh.ntriangles) + 1j * rng.uniform(-300, 300, f.mesh.ntriangles)
        return s
    mesh = _mesh(case)
    rwg = dm.build_rwg(mesh)
    s.update(mesh=mesh, rwg=rwg)
    if case["what"] in ("scattering", "sweep"):
        s["waves"] = _waves(rng, k, case.get("waves", 1))
    elif case["what"] == "design":
        s["waves"] = _waves(rng, k, 1)
        s["zs"] = rng.uniform(0, 200, mesh.ntriangles) + 0j
        cen = dm.triangle_centers(mesh)
        s["patch"] = 1 + (cen[:, 0] > 0) + 2 * (cen[:, 1] > 0)
        s["receive"] = rng.standard_normal(rwg.nedges) + 1j * rng.standard_normal(rwg.nedges)
    elif case["what"] == "product":
        s["x"] = rng.standard_normal(rwg.nedges) + 1j * rng.standard_normal(rwg.nedges)
    if case.get("cut"):
        s["grid"] = dm.phi_cut_grid(rng.uniform(0, math.pi), np.linspace(0, 180, case["cut"]))
    return s


def prepare(case, seed):
    s = _inputs(case, seed)
    if case["what"] == "surfaces":
        s["batch"] = dm.SurfaceBatch(8)
        return s
    if case["what"] == "product" and case["operator"] == "free":
        s["op"] = dm.matrixfree_efie_operator(s["mesh"], s["rwg"], s["k"])
        return s
    s["dev"] = dm.EFIEDevice(s["mesh"], s["rwg"])
    if case["what"] == "product":
        s["dev"].assemble(s["k"], precision="fp64" if case["operator"] == "dense" else "mixed")
    if case["what"] == "design":
        s["Mp"] = dm.precompute_patch_mass(s["mesh"], s["rwg"], dm.PatchPartition(s["patch"], 4), device=s["dev"])
    return s


# --------------------------------------------------------------------------
# one pass
# --------------------------------------------------------------------------
def run(s):
    case = s["case"]
    what = case["what"]
    if what == "scattering":
        r = dm.solve_scattering(s["mesh"], s["freq"], s["waves"][0], method=case.get("method", "auto"),
                                precision=case["precision"], preconditioner=case["precond"], device=s["dev"],
                                rwg=s["rwg"])
        if not case.get("cut"):
            return {"I": r.I_coeffs}
        return {"I": r.I_coeffs, "E": dm.compute_farfield(s["dev"], s["grid"], r.I_coeffs, k=s["k"])}
    if what == "sweep":
        r = dm.monostatic_rcs_sweep(s["mesh"], s["freq"], s["waves"], precision=case["precision"],
                                    return_currents=case["currents"], device=s["dev"], rwg=s["rwg"])
        return {"sigma": r.sigma, "I": r.currents} if case["currents"] else {"sigma": r.sigma}
    if what == "surfaces":
        r = dm.solve_surfaces(s["surfaces"], s["freq"], precision=case["precision"], return_currents=True,
                              batch=s["batch"])
        return {"sigma": r.sigma, "I": np.concatenate(r.currents)}
    if what == "design":
        dev = s["dev"]
        v = dm.assemble_excitation(s["mesh"], s["rwg"], s["waves"][0], device=dev)
        dev.assemble(s["k"], precision=case["precision"])
        dev.apply_impedance(s["zs"])
        P = dm.build_nearfield_preconditioner(dev, C0 / s["freq"])
        I, _ = dm.solve_gmres(dev, v, preconditioner=P)
        # J = |g^T I|^2, dJ/dI* = conj(g) (g^T I)
        q = np.conj(s["receive"]) * (s["receive"] @ I)
        lam = dm.solve_adjoint_rhs(dev, q, preconditioner=P)
        return {"I": I, "lambda": lam, "grad": dm.gradient_impedance(s["Mp"], I, lam)}
    if what == "product":
        return {"y": s["op"] @ s["x"] if case["operator"] == "free" else s["dev"].matvec(s["x"])}
    return {"Z": dm.assemble_Z_efie(s["mesh"], s["rwg"], s["k"], precision=case["precision"], device=s["dev"])}


# --------------------------------------------------------------------------
# what a pass cannot do without, and how exact it is
# --------------------------------------------------------------------------
def _counts(case):
    """(triangles, unknowns) of a case's mesh."""
    a, b = case["a"], case["b"]
    if case["body"] == "plate":
        return 2 * a * b, 3 * a * b - a - b
    if case["body"] == "disk":
        return b * (2 * a - 1), (3 * b * (2 * a - 1) - b) // 2
    return 20 * a * a, 30 * a * a


def work(case):
    """600 flops per triangle pair of the assembly, 8 per complex multiply-add;
    the factor, one product and one solve with it per right-hand side.  Bytes:
    the mesh and its basis in, the results out."""
    what = case["what"]
    if what == "surfaces":
        n = 0.5 * (500 + case["largest"])
        nt, mean3 = 2 * n / 3, n * (500 ** 2 + case["largest"] ** 2) / 2
        flops = case["count"] * (300 * nt * nt + 8 / 6 * mean3 + 16 * n * n)
        return {"bytes": case["count"] * (140 * n + 16 * n), "flops": flops}
    nt, n = _counts(case)
    mesh = 60 * nt + 100 * n
    if what == "matrix":
        return {"bytes": mesh + 16 * n * n, "flops": 300 * nt * nt}
    if what == "product":
        if case["operator"] == "free":
            return {"bytes": mesh + 32 * n, "flops": 300 * nt * nt}
        return {"bytes": PREC_BYTES["fp64" if case["operator"] == "dense" else "mixed"] * n * n + 32 * n,
                "flops": 8 * n * n}
    if what == "scattering" and (case.get("method") == "aca_gmres" or n > 10000):
        stored = 64 * n * math.log2(n / 64)
        return {"bytes": mesh + 16 * n + 16 * stored, "flops": 600 * stored}
    waves = case.get("waves", 2 if what == "design" else 1)
    factor = 0 if case.get("precond") in ("learned", "local") else 8 / 6 * n ** 3
    out = 8 * waves + (16 * n * waves if what != "sweep" or case["currents"] else 0)
    return {"bytes": mesh + out, "flops": 300 * nt * nt + factor + 16 * n * n * waves}


def tolerance(case):
    """About four times the largest distance from exact() measured over the
    ranges: rounding where the result is direct (2e-14 for products and
    matrices, 4e-13 for solves on a disk), the 32-bit far field of the mixed
    paths (3e-7 a matrix entry, 3e-6 to 8e-6 a current), and the GMRES tolerance
    of 1e-6 (1e-8 in a design step) where a preconditioner is not the inverse."""
    what, n = case["what"], 0 if case["what"] == "surfaces" else _counts(case)[1]
    if what in ("product", "matrix"):
        if "mixed" in (case.get("operator"), case.get("precision")):
            return {"rel": 1.2e-6}
        return {"rel": 1e-13, "max": 2e-11}
    if what == "design":
        return {"rel": 8e-8}
    if what == "surfaces":
        return {"rel": 2e-5, "max": 5e-4}
    if what == "sweep":
        return {"rel": 1.2e-5, "max": 2e-4} if case["precision"] == "mixed" else {"rel": 2e-12, "max": 2e-11}
    if case["precision"] == "mixed":
        return {"rel": 4e-5}
    return {"rel": 2e-12} if n <= 2000 and "method" not in case else {"rel": 6e-6}


# --------------------------------------------------------------------------
# the same discretisation in torch, 64 bits
# --------------------------------------------------------------------------
_RULE3 = (np.array([[1 / 6, 1 / 6], [2 / 3, 1 / 6], [1 / 6, 2 / 3]]), np.full(3, 1 / 6))
_B1, _A1, _B2, _A2 = 0.470142064105115, 0.059715871789770, 0.101286507323456, 0.797426985353087
_RULE7 = (np.array([[1 / 3, 1 / 3], [_B1, _B1], [_A1, _B1], [_B1, _A1], [_B2, _B2], [_A2, _B2], [_B2, _A2]]),
          np.array([0.1125] + 3 * [0.0661970763942530] + 3 * [0.0629695902724135]))


class _Body:
    """Quadrature points and basis values of a mesh, on the GPU."""

    def __init__(self, mesh, rwg):
        def t(a):
            return torch.as_tensor(np.ascontiguousarray(a), device="cuda")
        self.n, self.nt = rwg.nedges, mesh.ntriangles
        V = t(mesh.xyz)
        self.V = V[t(mesh.tri) - 1]                                          # nt, 3 vertices, 3
        e1, e2 = self.V[:, 1] - self.V[:, 0], self.V[:, 2] - self.V[:, 0]
        self.area = 0.5 * torch.linalg.norm(torch.linalg.cross(e1, e2), dim=1)
        self.tri = torch.stack([t(rwg.tplus), t(rwg.tminus)], 1) - 1          # n, 2 sides
        opp = V[torch.stack([t(rwg.vplus_opp), t(rwg.vminus_opp)], 1) - 1]   # n, 2, 3
        sign = torch.tensor([1.0, -1.0], dtype=torch.float64, device="cuda")
        self.s = sign * (t(rwg.len)[:, None] / (2 * self.area[self.tri]))     # n, 2
        self.div = 2 * self.s
        self.qp, self.f, self.w = [], [], []
        for x, w in (_RULE3, _RULE7):
            x = t(x)
            q = self.V[:, :1] + x[None, :, :1] * e1[:, None] + x[None, :, 1:] * e2[:, None]
            self.qp.append(q)                                                 # nt, points, 3
            self.f.append(self.s[..., None, None] * (q[self.tri] - opp[:, :, None]))  # n, 2, points, 3
            self.w.append(t(w))
        # triangles that share an edge, and each triangle's basis functions
        edges = np.sort(mesh.tri[:, [0, 1, 1, 2, 2, 0]].reshape(-1, 2), axis=1)
        order = np.lexsort((edges[:, 1], edges[:, 0]))
        same = np.flatnonzero(np.all(edges[order][1:] == edges[order][:-1], axis=1))
        p, q = t(order[same] // 3), t(order[same + 1] // 3)
        self.pairs = torch.cat([torch.stack([p, q], 1), torch.stack([q, p], 1)])
        self.near = torch.eye(self.nt, dtype=torch.bool, device="cuda")
        self.near[self.pairs[:, 0], self.pairs[:, 1]] = True
        slots = np.full((self.nt, 3), -1)
        count = np.zeros(self.nt, dtype=int)
        for side, tr in enumerate((rwg.tplus - 1, rwg.tminus - 1)):
            for m, tm in enumerate(tr):
                slots[tm, count[tm]] = 2 * m + side
                count[tm] += 1
        self.slots = t(slots)

    def _slot_pairs(self, pairs):
        """(pair index, slot i, slot j) of the pairs' basis functions that exist."""
        i = self.slots[pairs[:, 0]][:, :, None].expand(-1, 3, 3)
        j = self.slots[pairs[:, 1]][:, None, :].expand(-1, 3, 3)
        at = torch.nonzero((i >= 0) & (j >= 0))
        return at[:, 0], i[tuple(at.T)], j[tuple(at.T)]

    def matrix(self, k, zs=None):
        n = self.n
        Z = torch.empty((n, n), dtype=torch.complex128, device="cuda")
        q, f, w = self.qp[0], self.f[0], self.w[0]
        step = max(1, 60_000_000 // n)
        for r0 in range(0, n, step):
            rows = slice(r0, min(n, r0 + step))
            acc = torch.zeros((rows.stop - r0, n), dtype=torch.complex128, device="cuda")
            for s in range(2):
                tm = self.tri[rows, s]
                for u in range(2):
                    tn = self.tri[:, u]
                    far = (~self.near[tm][:, tn]).to(torch.float64)
                    dd = torch.outer(self.div[rows, s], self.div[:, u]) / (k * k)
                    for a in range(3):
                        for b in range(3):
                            pm, pn = q[tm, a], q[tn, b]
                            d = [pm[:, c, None] - pn[None, :, c] for c in range(3)]
                            R = torch.sqrt(d[0] * d[0] + d[1] * d[1] + d[2] * d[2])
                            del d
                            R = torch.where(far > 0, R, torch.ones_like(R))
                            g = far * (f[rows, s, a] @ f[:, u, b].T - dd) / R
                            g *= torch.outer(w[a] * 2 * self.area[tm], w[b] * 2 * self.area[tn]) / (4 * math.pi)
                            acc += torch.complex(g * torch.cos(k * R), -g * torch.sin(k * R))
            Z[rows] = acc
        self._add_near(Z, k)
        Z *= -1j * k * ETA0
        if zs is not None:
            own = torch.arange(self.nt, device="cuda")[:, None].expand(-1, 2)
            at, m, p, val = self._mass(own)
            Z.index_put_((m, p), -torch.as_tensor(zs, device="cuda")[at] * val, accumulate=True)
        return Z

    def _mass(self, own):
        at, i, j = self._slot_pairs(own)
        m, p = i // 2, j // 2
        f = self.f[0]
        val = torch.einsum("xqc,xqc,q->x", f[m, i % 2], f[p, j % 2], self.w[0]) * 2 * self.area[at]
        return at, m, p, val

    def _add_near(self, Z, k):
        own = torch.arange(self.nt, device="cuda")[:, None].expand(-1, 2)
        for pairs, itself in ((own, True), (self.pairs, False)):
            at, i, j = self._slot_pairs(pairs)
            m, p = i // 2, j // 2
            keep = m <= p                  # the entry of (m, p) with m <= p stands for both
            at, i, j, m, p = at[keep], i[keep], j[keep], m[keep], p[keep]
            tm, tn = pairs[at, 0], pairs[at, 1]
            dd = self.div[m, i % 2] * self.div[p, j % 2] / (k * k)
            rule = 1 if itself else 0
            fm, fp, w = self.f[rule][m, i % 2], self.f[rule][p, j % 2], self.w[rule]
            R = torch.linalg.norm(self.qp[rule][tm][:, :, None] - self.qp[rule][tn][:, None], dim=-1)
            zero = R == 0
            R1 = torch.where(zero, torch.ones_like(R), R)
            sm = torch.complex(-2 * torch.sin(0.5 * k * R) ** 2 / R1, -torch.sin(k * R) / R1)
            sm = torch.where(zero, torch.full_like(sm, -1j * k), sm) / (4 * math.pi)
            ww = 4 * self.area[tm] * self.area[tn]
            val = torch.einsum("xab,xab,a,b->x", (torch.einsum("xac,xbc->xab", fm, fp) - dd[:, None, None]).to(sm.dtype),
                               sm, w.to(sm.dtype), w.to(sm.dtype)) * ww
            # the static part: the inner integral of 1/R in closed form
            fm, fp, w = self.f[1][m, i % 2], self.f[1][p, j % 2], self.w[1]
            R = torch.linalg.norm(self.qp[1][tm][:, :, None] - self.qp[1][tn][:, None], dim=-1)
            inv = torch.where(R == 0, torch.zeros_like(R), 1 / torch.where(R == 0, torch.ones_like(R), R)) / (4 * math.pi)
            S = self._one_over_r(self.qp[1][tm], self.V[tn]) / (4 * math.pi)
            outer = w * 2 * self.area[tm][:, None]
            if itself:
                lead = torch.einsum("xac,xac->xa", fm, fp) * S
                df = fp[:, None] - fp[:, :, None]
                rest = torch.einsum("xac,xabc,xab,b->xa", fm, df, inv, w) * 2 * self.area[tn][:, None]
            else:
                lead = torch.einsum("xac,xbc,xab,b->xa", fm, fp, inv, w) * 2 * self.area[tn][:, None]
                rest = 0
            val = val + torch.sum((lead + rest - dd[:, None] * S) * outer, dim=1)
            Z.index_put_((m, p), val, accumulate=True)
            off = m != p
            Z.index_put_((p[off], m[off]), val[off], accumulate=True)

    @staticmethod
    def _one_over_r(P, V):
        """Integral of 1/R over the triangles V seen from the points P (pairs, points, 3)."""
        nrm = torch.linalg.cross(V[:, 1] - V[:, 0], V[:, 2] - V[:, 0])
        nrm = nrm / torch.linalg.norm(nrm, dim=1, keepdim=True)
        h = torch.einsum("xpc,xc->xp", P - V[:, :1], nrm)
        foot = P - h[..., None] * nrm[:, None]
        ah, total = h.abs(), 0
        for e in range(3):
            A, B = V[:, e], V[:, (e + 1) % 3]
            l = (B - A) / torch.linalg.norm(B - A, dim=1, keepdim=True)
            out = torch.linalg.cross(l, nrm)
            d = torch.einsum("xpc,xc->xp", A[:, None] - foot, out)
            sm = torch.einsum("xpc,xc->xp", A[:, None] - foot, l)
            sp = torch.einsum("xpc,xc->xp", B[:, None] - foot, l)
            Rm, Rp = torch.linalg.norm(P - A[:, None], dim=-1), torch.linalg.norm(P - B[:, None], dim=-1)
            ratio = (sp + Rp) / (sm + Rm)
            log = torch.where(d != 0, torch.log(torch.where(d != 0, ratio, torch.ones_like(ratio))), torch.zeros_like(d))
            total = total + d * log
            R0 = d * d + h * h
            ang = torch.atan(d * sp / (R0 + ah * Rp)) - torch.atan(d * sm / (R0 + ah * Rm))
            total = total - ah * torch.where((ah != 0) & (d != 0), ang, torch.zeros_like(ang))
        return total

    def _phases(self, k, dirs, sign):
        """sum over sides and points of w 2A f exp(sign i k dir . r): n, dirs, 3."""
        out = torch.zeros((self.n, dirs.shape[0], 3), dtype=torch.complex128, device="cuda")
        for s in range(2):
            for a in range(3):
                t = self.tri[:, s]
                arg = sign * k * (self.qp[0][t, a] @ dirs.T)
                wt = (self.w[0][a] * 2 * self.area[t])[:, None]
                out += (wt * torch.complex(torch.cos(arg), torch.sin(arg)))[..., None] * self.f[0][:, s, a][:, None]
        return out

    def rhs(self, waves):
        out = []
        for w in waves:
            kv = torch.as_tensor(w.k_vec, device="cuda")
            k = torch.linalg.norm(kv)
            out.append(-w.E0 * (self._phases(k, (kv / k)[None], -1)[:, 0] @
                                torch.as_tensor(w.pol, device="cuda").to(torch.complex128)))
        return torch.stack(out, 1)

    def field(self, k, dirs, I):
        """Far field E (3, dirs, columns) of currents I (n, columns)."""
        out = []
        for r in range(0, dirs.shape[0], 256):
            d = dirs[r:r + 256]
            c = torch.einsum("ndc,nr->cdr", self._phases(k, d, 1), I)
            dt = d.T.to(c.dtype)[..., None]
            out.append(1j * k * ETA0 / (4 * math.pi) * (dt * torch.sum(dt * c, 0, keepdim=True) - c))
        return torch.cat(out, 1)

    def sigma(self, waves, I):
        out = []
        for r, w in enumerate(waves):
            k = float(np.linalg.norm(w.k_vec))
            E = self.field(k, torch.as_tensor(-w.k_vec / k, device="cuda")[None], I[:, r:r + 1])
            out.append(4 * math.pi * torch.sum(E.abs() ** 2) / w.E0 ** 2)
        return torch.stack(out)


def exact(case, seed):
    s = _inputs(case, seed)
    what, k = case["what"], s["k"]
    if what == "surfaces":
        sigma, I = [], []
        for f in s["surfaces"]:
            B = _Body(f.mesh, f.rwg)
            x = torch.linalg.solve(B.matrix(k, f.zs), B.rhs([f.excitation]))
            sigma.append(B.sigma([f.excitation], x)[0])
            I.append(x[:, 0])
        return {"sigma": torch.stack(sigma).cpu().numpy(), "I": torch.cat(I).cpu().numpy()}
    B = _Body(s["mesh"], s["rwg"])
    Z = B.matrix(k, s.get("zs"))
    if what == "matrix":
        return {"Z": Z.cpu().numpy()}
    if what == "product":
        return {"y": (Z @ torch.as_tensor(s["x"], device="cuda")).cpu().numpy()}
    V = B.rhs(s["waves"])
    I = torch.linalg.solve(Z, V)
    if what == "scattering":
        out = {"I": I[:, 0].cpu().numpy()}
        if case.get("cut"):
            out["E"] = B.field(k, torch.as_tensor(s["grid"].rhat, device="cuda"), I)[:, :, 0].cpu().numpy()
        return out
    if what == "sweep":
        out = {"sigma": B.sigma(s["waves"], I).cpu().numpy()}
        return {**out, "I": I.cpu().numpy()} if case["currents"] else out
    I = I[:, 0]
    g = torch.as_tensor(s["receive"], device="cuda")
    lam = torch.linalg.solve(Z.conj().T, torch.conj(g) * (g @ I))
    at, m, p, val = B._mass(torch.arange(B.nt, device="cuda")[:, None].expand(-1, 2))
    patch = torch.as_tensor(s["patch"] - 1, device="cuda")[at]
    grad = torch.zeros(4, dtype=torch.float64, device="cuda")
    grad.index_add_(0, patch, 2 * (torch.conj(lam[m]) * val * I[p]).real)
    return {"I": I.cpu().numpy(), "lambda": lam.cpu().numpy(), "grad": grad.cpu().numpy()}
