"""What the performance of this framework is measured on.

Every case is one pass of work that a program using the framework has it do,
through the public classes (or, for the LU protocol, the C ABI of
include/bem200.h).  Kinds:

* ``solve``  -- one wavelength of a spectrum: a resident ``BEMRet`` is cleared,
  assembles and factors at the wavelength and solves for the plane wave; the
  pass ends with the surface charges, currents and the extinction on the host;
* ``sweep``  -- ``solve_sweep`` over a small batch of uneven meshes, several
  wavelengths, on worker streams (solvers constructed in the call);
* ``gmres``  -- ``BEMRetIter``: H-matrix operator, no preconditioner, restarted
  GMRES (the path of meshes whose dense factors are not wanted);
* ``vgrad``  -- extinction and its gradient over every vertex coordinate
  (reverse mode: one solve, one transposed solve, the contraction);
* ``field``  -- potentials and electric / magnetic fields of a solution at the
  faces, on both sides of the surface;
* ``lu``     -- the LU protocol: factor a complex128 matrix with partial pivoting
  and solve for a few right-hand sides (``bem200_getrf`` / ``bem200_getrs``).

Sizes are those of the tests, the benchmark and the sweep batch: 116 to about
10,000 faces, curved and flat, triangles and quadrilaterals, one or two
polarisations.  The seed sets the particle dimensions, the wavelength, the
direction of propagation and the polarisations.
"""
import math

import numpy as np
import torch

from mnpbem_b200 import ComParticle, EpsConst, EpsDrude, PlaneWaveRet, trisphere
from mnpbem_b200 import _native as nat
from mnpbem_b200.bem import BEMRet
from mnpbem_b200.bem_iter import BEMRetIter
from mnpbem_b200.geometry import tricube, triellipsoid, trirod
from mnpbem_b200.planewave import CompStruct
from mnpbem_b200.shape import extinction_vertex_vjp
from mnpbem_b200.sweep import solve_sweep

GOLD = (9.84, 9.0, 0.067)
SILVER = (3.7, 9.17, 0.021)
# vertex counts of the stored energy-minimised sphere point sets
SPHERES = (60, 144, 169, 225, 256, 289, 324, 361, 400, 441, 484, 529, 576, 625, 676, 729, 784, 841, 900, 961, 1024,
           1225, 1444)


def listed():
    return [
        # the smallest production mesh: latency and launches count
        dict(name="solve_fp64_sphere284", kind="solve", shape="sphere", a=144, b=0, c=0, metal="gold", npol=1,
             precision="fp64"),
        dict(name="solve_mixed_sphere284", kind="solve", shape="sphere", a=144, b=0, c=0, metal="gold", npol=1,
             precision="mixed"),
        # an ordinary curved rod of odd face count, both polarisations
        dict(name="solve_mixed_rod1325", kind="solve", shape="rod", a=26, b=14, c=28, metal="gold", npol=2,
             precision="mixed"),
        # the 2400-face rod of the gradient configuration, in the default precision
        dict(name="solve_fp64_rod2400", kind="solve", shape="rod", a=41, b=16, c=31, metal="gold", npol=2,
             precision="fp64"),
        # the benchmark's sphere dimer, mixed and in the default precision
        dict(name="solve_mixed_dimer5768", kind="solve", shape="dimer", a=1444, b=0, c=0, metal="gold", npol=1,
             precision="mixed"),
        dict(name="solve_fp64_dimer5768", kind="solve", shape="dimer", a=1444, b=0, c=0, metal="gold", npol=1,
             precision="fp64"),
        # a large rounded cube (quadrilaterals)
        dict(name="solve_mixed_cube10080", kind="solve", shape="cube", a=42, b=0, c=0, metal="gold", npol=1,
             precision="mixed"),
        # a batch of uneven meshes on four worker streams
        dict(name="sweep_uneven", kind="sweep", a=382, b=784, c=8, metal="gold", npol=2, workers=4),
        # the matrix-free iterative path
        dict(name="gmres_hmatrix_ellipsoid3600", kind="gmres", shape="ellipsoid", a=1802, b=0, c=0, metal="gold",
             npol=1, cleaf=64),
        # the gradient configuration
        dict(name="vgrad_rod2400", kind="vgrad", shape="rod", a=41, b=16, c=31, metal="gold", npol=1),
        # near fields of a solution
        dict(name="field_sphere2884", kind="field", shape="sphere", a=1444, b=0, c=0, metal="gold", npol=1),
        # the LU protocol on a complex128 matrix of ragged size
        dict(name="lu_c128_1537", kind="lu", n=1537, nrhs=4),
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _draw_shape(rng, lo, hi):
    """A particle of about log-uniformly many faces in [lo, hi]."""
    nf = _log_uniform(rng, lo, hi)
    shape = rng.choice(["sphere", "dimer", "ellipsoid", "rod", "cube"])
    if shape == "sphere" and nf > 2 * SPHERES[-1]:
        shape = "ellipsoid"
    if shape == "dimer" and not 4 * SPHERES[0] < nf < 4 * SPHERES[-1]:
        shape = "rod"
    if shape in ("sphere", "dimer"):
        per = 2 if shape == "sphere" else 4
        a, b, c = min(SPHERES, key=lambda v: abs(per * v - nf)), 0, 0
    elif shape == "ellipsoid":
        a, b, c = max(60, int(nf / 2) + 2), 0, 0
    elif shape == "rod":
        a = max(9, int(math.sqrt(nf / 1.5) * rng.uniform(0.8, 1.1)))
        rest = max(12, int(nf / (a - 1)))
        b = max(4, int(rest * rng.uniform(0.2, 0.3)))
        c = max(3, rest - 2 * (b - 1) + 1)
    else:
        a, b, c = max(5, int(math.sqrt(nf / 6)) + 1), 0, 0
    return dict(shape=shape, a=a, b=b, c=c)


def draw(rng):
    kind = rng.choice(["solve"] * 6 + ["sweep", "gmres", "vgrad", "field", "lu"])
    metal = rng.choice(["gold", "gold", "silver"])
    npol = rng.choice([1, 2])
    if kind == "solve":
        precision = rng.choice(["mixed", "mixed", "fp64"])
        return dict(kind=kind, **_draw_shape(rng, 116, 9600 if precision == "mixed" else 5200), metal=metal, npol=npol,
                    precision=precision)
    if kind == "sweep":
        return dict(kind=kind, a=int(_log_uniform(rng, 100, 400)), b=int(_log_uniform(rng, 200, 800)),
                    c=rng.randint(3, 8), metal=metal, npol=npol, workers=rng.choice([1, 2, 4]))
    if kind == "gmres":
        return dict(kind=kind, **_draw_shape(rng, 400, 3600), metal="gold", npol=1, cleaf=rng.choice([64, 128, 200]))
    if kind == "vgrad":
        return dict(kind=kind, **_draw_shape(rng, 116, 2400), metal="gold", npol=npol)
    if kind == "field":
        return dict(kind=kind, **_draw_shape(rng, 116, 2884), metal="gold", npol=npol)
    return dict(kind=kind, n=int(_log_uniform(rng, 65, 2048)), nrhs=rng.randint(1, 16))


def _faces(case):
    a, b, c = case["a"], case["b"], case["c"]
    return {"sphere": 2 * a - 4, "dimer": 4 * a - 8, "ellipsoid": 2 * a - 4, "rod": (a - 1) * (2 * (b - 1) + c - 1),
            "cube": 6 * (a - 1) ** 2}[case["shape"]]


def _particle(case, rng):
    """The compound particle of a case, dimensions (nm) from the seed."""
    a, b, c = case["a"], case["b"], case["c"]
    metal = EpsDrude(*(GOLD if case["metal"] == "gold" else SILVER))
    interp, eps_b = "curv", 1.0
    if case["shape"] == "sphere":
        parts = [trisphere(a, rng.uniform(18.0, 22.0))]
    elif case["shape"] == "dimer":
        d, gap = rng.uniform(38.0, 42.0), rng.uniform(1.9, 2.1)
        parts = [trisphere(a, d), trisphere(a, d)]
        parts[0].shift([-(d + gap) / 2, 0, 0])
        parts[1].shift([(d + gap) / 2, 0, 0])
        eps_b = 1.77
    elif case["shape"] == "ellipsoid":
        parts, interp = [triellipsoid(a, rng.uniform(18.0, 30.0, size=3))], "flat"
    elif case["shape"] == "rod":
        parts, eps_b = [trirod(rng.uniform(18.0, 22.0), rng.uniform(70.0, 90.0), [a, b, c], interp="curv")], 1.77
    else:
        parts = [tricube(a, rng.uniform(80.0, 100.0), e=0.25)]
    n = len(parts)
    return ComParticle([EpsConst(eps_b), metal], parts, [[2, 1]] * n, *range(1, n + 1), interp=interp)


def _wave(npol, rng):
    """A plane wave of random direction; polarisations orthogonal to it."""
    q, r = np.linalg.qr(rng.standard_normal((3, 3)))
    q = q * np.sign(np.diag(r))
    return [q[:, 1 + i].tolist() for i in range(npol)], [q[:, 0].tolist()] * npol


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "lu":
        g = torch.Generator(device="cuda").manual_seed(int(seed))
        n, nrhs = case["n"], case["nrhs"]
        f64 = dict(generator=g, device="cuda", dtype=torch.float64)
        # well-conditioned, not diagonally dominant: partial pivoting exchanges rows
        A = torch.view_as_complex(torch.randn((n, n, 2), **f64))
        A = A + 2 * math.sqrt(n) * torch.eye(n, device="cuda", dtype=A.dtype)[torch.randperm(n, generator=g,
                                                                                            device="cuda")]
        B = torch.view_as_complex(torch.randn((n, nrhs, 2), **f64))
        L = nat.lib()
        wsb = int(L.bem200_getrf_workspace_size(nat.C128, 0, n))
        scr = int(L.bem200_getrs_workspace_size(nat.C128, n, nrhs))
        i32 = dict(dtype=torch.int32, device="cuda")
        return dict(case=case, A=A.contiguous(), B=B.contiguous(), LU=torch.empty_like(A), X=torch.empty_like(B),
                    rowmap=torch.empty(n, **i32), ipiv=torch.empty(n, **i32),
                    info=torch.zeros(1, **i32), status=torch.zeros(1, **i32),
                    ws=torch.empty(wsb, dtype=torch.uint8, device="cuda"), wsb=wsb,
                    scr=torch.empty(scr, dtype=torch.uint8, device="cuda"))
    pol, dirs = _wave(case["npol"], rng)
    if kind == "sweep":
        sub = [dict(shape="ellipsoid", a=case["a"], b=0, c=0, metal=case["metal"]),
               dict(shape="sphere", a=min(SPHERES, key=lambda v: abs(v - case["b"])), b=0, c=0, metal=case["metal"])]
        return dict(case=case, parts=[_particle(s, rng) for s in sub], pol=pol, dirs=dirs,
                    enei=np.linspace(rng.uniform(500, 520), rng.uniform(680, 720), case["c"]))
    p = _particle(case, rng)
    exc = PlaneWaveRet(pol, dirs)
    enei = float(rng.uniform(550.0, 750.0))
    state = dict(case=case, p=p, exc=exc, enei=enei)
    if kind == "gmres":
        state["bem"] = BEMRetIter(p, precond=None, hmatrix=True, cleaf=case["cleaf"])
    elif kind == "field":
        # a solution in hand (from an earlier solve of the program)
        n, npol = p.n, case["npol"]

        def values(*shape):
            return rng.standard_normal(shape) + 1j * rng.standard_normal(shape)
        tail = (npol,) if npol > 1 else ()
        state["bem"] = BEMRet(p)
        state["sig"] = CompStruct(p, enei, sig1=values(n, *tail), sig2=values(n, *tail), h1=values(n, 3, *tail),
                                  h2=values(n, 3, *tail))
    else:
        state["bem"] = BEMRet(p, precision=case.get("precision", "mixed"))
    return state


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "lu":
        n = case["n"]
        s["LU"].copy_(s["A"])
        s["X"].copy_(s["B"])
        st = nat.stream_ptr()
        nat.call("bem200_getrf", nat.C128, 0, n, nat.ptr(s["LU"]), n, nat.ptr(s["rowmap"]),
                 nat.ptr(s["ipiv"]), nat.ptr(s["info"]), nat.ptr(s["ws"]), s["wsb"], st)
        nat.call("bem200_getrs", nat.C128, 0, n, case["nrhs"], nat.ptr(s["LU"]), n, nat.ptr(s["rowmap"]),
                 nat.ptr(s["X"]), case["nrhs"], nat.ptr(s["ws"]), s["wsb"], nat.ptr(s["scr"]), nat.ptr(s["status"]),
                 st)
        return dict(x=s["X"], ipiv=s["ipiv"], info=s["info"], status=s["status"])
    if kind == "sweep":
        r = solve_sweep(s["parts"], s["enei"], s["pol"], s["dirs"], workers=case["workers"])
        return dict(ext=r["ext"], sca=r["sca"])
    bem, exc, p, enei = s["bem"], s["exc"], s["p"], s["enei"]
    if kind == "vgrad":
        bem.clear()
        ext, grad = extinction_vertex_vjp(bem, exc, enei)
        return dict(ext=ext, grad=grad)
    if kind == "field":
        out = {}
        for side in (1, 2):
            pot, fld = bem.potential(s["sig"], side), bem.field(s["sig"], side)
            for k in ("phi", "a"):
                out["%s%d" % (k, side)] = pot["%s%d" % (k, side)]
                out["%s%dp" % (k, side)] = pot["%s%dp" % (k, side)]
            out["e%d" % side], out["h%d" % side] = fld.e, fld.h
        return out
    bem.clear()
    sig, _ = bem.solve(exc.potential(p, enei))
    return dict(sig1=sig.sig1, sig2=sig.sig2, h1=sig.h1, h2=sig.h2, ext=np.asarray(exc.extinction(sig)))


def work(case):
    """Multiply-adds count two; a complex multiply-add eight.  The retarded BEM
    needs G1, G2, Delta and Sigma factored or inverted and two right divisions
    by matrices: 32 n^3 real operations with LU factors and triangular solves."""
    kind = case["kind"]
    if kind == "lu":
        n = case["n"]
        return {"bytes": 16 * (2 * n * n + 2 * n * case["nrhs"]), "flops": 8 / 3 * n ** 3 + 8 * n * n * case["nrhs"]}
    if kind == "sweep":
        ns = (2 * case["a"] - 4, 2 * min(SPHERES, key=lambda v: abs(v - case["b"])) - 4)
        return {"bytes": case["c"] * sum(64.0 * n * n for n in ns), "flops": case["c"] * sum(32.0 * n ** 3 for n in ns)}
    n = _faces(case)
    io = 16.0 * 16 * n * case["npol"]
    if kind == "field":      # two sides, two region terms: G, F and Gp of every pair, about 100 operations each
        return {"bytes": io * 3, "flops": 4 * 100.0 * n * n}
    if kind == "gmres":      # the entries of four compressed matrices (about a third of dense) and ten products
        return {"bytes": 4 * 16.0 * n * n / 3 * 10, "flops": 10 * 8 * 8.0 * n * n / 3 * 4}
    flops = 32.0 * n ** 3
    if kind == "vgrad":
        flops += 400.0 * n * n
    return {"bytes": 64.0 * n * n + io, "flops": flops}


def exact(case, seed):
    """The solution of the LU case in 64 bits; the pivots have no such value
    (they depend on the rounding of the elimination), and a whole BEM solve
    has none without this package's refinement integrals."""
    if case["kind"] != "lu":
        return None
    s = prepare(case, seed)
    return dict(x=torch.linalg.solve(s["A"], s["B"]), ipiv=None, info=None, status=None)
