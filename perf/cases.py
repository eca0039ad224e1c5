"""Measured cases of the solver: what a user of the library has it do, through its public calls.

A case is one of three kinds:

  solve    a context (piks3d_b200.Solver) whose image is set up, as a driver holds it between
           checks of main.F90's loop. A pass is `checks` rounds of chkConvergeStep iterations
           and one convergence check, then the macroscopic fields of the box.
  batch    several contexts iterated together (piks3d_b200.Batch), the same pass for all of them.
  refined  one whole call of solve.solve_one: image on the host in, set-up, FP32 iterations with
           extrapolation, FP64 refinement to a 1e-4 permeability tolerance, fields out.

Precision "fp64" is the reference's arithmetic, "fp32" the refined solver's bulk phase (FP32
distribution function, FP64 moments and wall densities).
"""
import heapq
import math

import numpy as np
import torch

import piks3d_b200 as pk
from piks3d_b200 import images
from piks3d_b200.solve import solve_one

STEP = 10  # chkConvergeStep of every case (initParams' default)


def listed():
    """The listed cases."""
    return [
        # the plain solve that also runs on a CPU with the reference: 32^3 box, one centred sphere
        # of radius 12, 64 velocities, Kn about 1, second-order wall extrapolation (the default).
        # Launch latency and the length of the upwind chain decide.
        dict(name="sphere32_nv64_fp64", kind="solve", image="sphere", nx=32, ny=32, nz=32, porosity=0.78, nc=2,
             kn=1.0, order=2, layer=0, precision="fp64", checks=10),
        # a small pack as a parameter study runs it, 512 velocities, in both phases of a refined solve
        dict(name="pack48_nv512_fp64", kind="solve", image="pack", nx=48, ny=48, nz=48, porosity=0.45, nc=4,
             kn=2.0, order=1, layer=0, precision="fp64", checks=10),
        dict(name="pack48_nv512_fp32", kind="solve", image="pack", nx=48, ny=48, nz=48, porosity=0.45, nc=4,
             kn=2.0, order=1, layer=0, precision="fp32", checks=10),
        # 64 velocities (8 per octant) on an ordinary image: the narrowest rows
        dict(name="pack96_nv64_fp32", kind="solve", image="pack", nx=96, ny=96, nz=96, porosity=0.5, nc=2,
             kn=5.0, order=1, layer=0, precision="fp32", checks=10),
        # the shipped tutorial's geometry: quarter sphere in a 100^3 box, porosity 0.75
        dict(name="tutorial100_nv512_fp64", kind="solve", image="quarter", nx=100, ny=100, nz=100, porosity=0.75,
             nc=4, kn=0.1, order=1, layer=0, precision="fp64", checks=3),
        # the benchmark's image: 128^3 sphere pack, porosity 0.40, 512 velocities, Kn 0.5
        dict(name="pack128_nv512_fp64", kind="solve", image="pack", nx=128, ny=128, nz=128, porosity=0.40, nc=4,
             kn=0.5, order=1, layer=0, precision="fp64", checks=4),
        dict(name="pack128_nv512_fp32", kind="solve", image="pack", nx=128, ny=128, nz=128, porosity=0.40, nc=4,
             kn=0.5, order=1, layer=0, precision="fp32", checks=6),
        # the large single solve: 256^3 Gaussian random field, porosity 0.20, Kn 0.1
        dict(name="field256_nv512_fp32", kind="solve", image="field", nx=256, ny=256, nz=256, porosity=0.20, nc=4,
             kn=0.1, order=1, layer=0, precision="fp32", checks=4),
        # a box with unequal odd edges, fluid layers at inlet and outlet, 1728 velocities
        dict(name="ragged_nv1728_fp64", kind="solve", image="pack", nx=75, ny=53, nz=37, porosity=0.55, nc=6,
             kn=1.0, order=1, layer=2, precision="fp64", checks=3),
        # eight images of a batch (edges 32-96, 64 or 512 velocities), its FP32 phase
        dict(name="batch8_fp32", kind="batch", members=8, emin=32, emax=96, porosity=0.45, kn=1.0, order=1,
             precision="fp32", checks=3),
        # five of them in their FP64 phase
        dict(name="batch5_fp64", kind="batch", members=5, emin=32, emax=64, porosity=0.45, kn=1.0, order=1,
             precision="fp64", checks=4),
        # one request as a user of the refined solver sends it: image in, fields out
        dict(name="refined48_nv512", kind="refined", image="pack", nx=48, ny=48, nz=48, porosity=0.45, nc=4,
             kn=1.0, order=1, layer=0, precision="refined", checks=0),
    ]


def draw(rng):
    """One more case of the same ranges."""
    def logi(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    kind = rng.choice(("solve", "solve", "solve", "solve", "batch", "refined"))
    kn = round(math.exp(rng.uniform(math.log(0.05), math.log(10.0))), 4)
    porosity = round(rng.uniform(0.3, 0.6), 3)
    if kind == "batch":
        precision = rng.choice(("fp32", "fp64"))
        lo = logi(20, 40)
        return dict(kind="batch", members=rng.randint(2, 6), emin=lo, emax=lo + rng.randint(8, 40), porosity=porosity,
                    kn=kn, order=1, precision=precision, checks=rng.randint(1, 4))
    if kind == "refined":
        n = logi(24, 64)
        return dict(kind="refined", image="pack", nx=n, ny=n, nz=n, porosity=porosity, nc=rng.choice((2, 4)),
                    kn=max(kn, 0.5), order=1, layer=0, precision="refined", checks=0)
    nc = rng.choice((2, 4, 4, 4, 6, 8))
    top = {2: 160, 4: 128, 6: 72, 8: 48}[nc]
    image = rng.choice(("pack", "pack", "field", "quarter"))
    nx, ny, nz = (logi(24, top) for _ in range(3))
    if image == "quarter":
        ny = nz = nx
    return dict(kind="solve", image=image, nx=nx, ny=ny, nz=nz, porosity=porosity if image != "quarter" else 0.75,
                nc=nc, kn=kn, order=1, layer=rng.choice((0, 0, 1, 2)), precision=rng.choice(("fp64", "fp32")),
                checks=rng.randint(1, 4))


# ---- inputs -----------------------------------------------------------------------------

def _field(nx, ny, nz, porosity, corr, seed):
    """A Gaussian-correlated random field thresholded at `porosity` (1 = solid)."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    noise = torch.from_numpy(np.random.default_rng(seed).standard_normal((nz, ny, nx), dtype=np.float32)).to(dev)
    k2 = sum(torch.meshgrid(*(torch.fft.fftfreq(n, device=dev) ** 2 for n in (nz, ny, nx)), indexing="ij"))
    f = torch.fft.ifftn(torch.fft.fftn(noise) * torch.exp(-2.0 * (math.pi * corr) ** 2 * k2)).real
    thr = torch.sort(f.reshape(-1)).values[int(porosity * f.numel())]
    return (f >= thr).to(torch.uint8).cpu().numpy()


def _image(case, seed):
    """The case's image (uint8, z-y-x, 1 = solid) and Knudsen number for a seed."""
    nx, ny, nz, kn = case["nx"], case["ny"], case["nz"], case["kn"]
    if case["image"] == "sphere":   # one geometry; the seed moves the Knudsen number
        return images.centred_sphere(nx, 12.0 * nx / 32.0), kn * (0.8 + 0.4 * np.random.default_rng(seed).random())
    if case["image"] == "quarter":
        return images.quarter_sphere(nx, case["porosity"]), kn * (0.8 + 0.4 * np.random.default_rng(seed).random())
    if case["image"] == "field":
        return _field(nx, ny, nz, case["porosity"], 6.0, seed), kn
    n = max(nx, ny, nz)
    r = (4.0, 8.0) if n >= 48 else (2.0, 5.0)
    return np.ascontiguousarray(images.sphere_pack(n, case["porosity"], r[0], r[1], seed=seed)[:nz, :ny, :nx]), kn


def _members(case, seed):
    """The members of a batch case, each described as a solve case, and their seeds."""
    rng = np.random.default_rng(seed)
    out = []
    for m in range(case["members"]):
        # edges spread over the range, 64 or 512 velocities in turn (the seed moves the rest)
        n = case["emin"] + (case["emax"] - case["emin"]) * m // max(1, case["members"] - 1)
        out.append((dict(kind="solve", image="pack", nx=n, ny=n, nz=n, porosity=case["porosity"], nc=(4, 2)[m % 2],
                         kn=case["kn"] * float(np.exp(rng.uniform(-1.0, 1.0))), order=case["order"], layer=0,
                         precision=case["precision"], checks=case["checks"]), int(rng.integers(1 << 30))))
    return out


def _params(case, kn):
    return pk.default_params(Nx=case["nx"], Ny=case["ny"], Nz=case["nz"], Nc_fundamental=case["nc"], Kn=kn,
                             pressDrop=1.0, eps=1e-8, chkConvergeStep=STEP, maxStep=4000, wallExtOrder=case["order"],
                             fluidlayer=case["layer"])


def _solver(case, seed):
    img, kn = _image(case, seed)
    s = pk.Solver(_params(case, kn), device=0)
    s.set_precision(pk.PREC_FP32 if case["precision"] == "fp32" else pk.PREC_FP64)
    s.setup_physical_grid(img)
    return s


def prepare(case, seed):
    """What the user's program holds before the call."""
    if case["kind"] == "refined":
        img, kn = _image(case, seed)
        return {"case": case, "image": img, "params": _params(case, kn)}
    if case["kind"] == "batch":
        batch = pk.Batch(device=0)
        for c, sd in _members(case, seed):
            batch.add(_solver(c, sd))
        return {"case": case, "batch": batch, "members": list(batch.members)}
    return {"case": case, "solver": _solver(case, seed)}


def _fields(solver):
    return dict(zip(("rho", "ux", "uy", "uz"), solver.get_macro()))


def run(state):
    """One pass."""
    case = state["case"]
    if case["kind"] == "refined":
        r = solve_one(state["image"], state["params"], precision="refined", tol=1e-4, keep_fields=True)
        return {"steps": r["steps"], "mass": r["mass"], "permeability": r["permeability"],
                "fields": dict(zip(("rho", "ux", "uy", "uz"), r["macro"]))}
    if case["kind"] == "batch":
        checks = []
        for _ in range(case["checks"]):
            state["batch"].iterate(STEP)
            checks.append(np.stack(state["batch"].chk_converge()))
        return {"checks": np.stack(checks), "fields": [_fields(s) for s in state["members"]]}
    s = state["solver"]
    checks = []
    for _ in range(case["checks"]):
        s.iterate(STEP)
        checks.append(s.chk_converge())
    return {"checks": np.array(checks), "fields": _fields(s)}


# ---- the least work ---------------------------------------------------------------------

def _solve_work(case, iterations, value_bytes):
    """Every iteration reads and writes each voxel-velocity of the pore space once and its
    moments once; the fields of the box are written once. An update is some 36 operations:
    the equilibrium (9), the upwind terms (12), the division (1), and its share of the four
    moment sums (14)."""
    voxels = (case["nx"] + 2 * case["layer"]) * case["ny"] * case["nz"]
    fluid = case["porosity"] * case["nx"] * case["ny"] * case["nz"] + 2 * case["layer"] * case["ny"] * case["nz"]
    updates = fluid * 8 * case["nc"] ** 3 * iterations
    return 2 * value_bytes * updates + 64 * fluid * iterations + 32 * voxels, 36 * updates


def work(case):
    """Bytes and operations one pass cannot do without."""
    esz = 8 if case["precision"] == "fp64" else 4
    if case["kind"] == "refined":   # about 200 FP32 and 100 FP64 iterations to the tolerance
        a, b = _solve_work(case, 200, 4), _solve_work(case, 100, 8)
        return {"bytes": a[0] + b[0], "flops": a[1] + b[1]}
    parts = [c for c, _ in _members(case, 0)] if case["kind"] == "batch" else [case]
    each = [_solve_work(c, STEP * c["checks"], esz) for c in parts]
    return {"bytes": sum(e[0] for e in each), "flops": sum(e[1] for e in each)}


# ---- the same values in 64 bits, from the discrete equations -----------------------------
# The scheme of PIKS3D (solver.F90, output.F90) in plain numpy and torch: drill and thin passes
# of the image, wall labels, upwind sweeps by hyperplane, diffuse walls, periodic pressure jump,
# symmetry planes, moments, mass flux.

# half-range Gauss-Hermite abscissae and weights (gaussHermite.F90)
_GH = {
    2: ((3.001939310608394140e-01, 1.252421045333717009e+00), (3.613798911363155786e-01, 1.386201088636844214e-01)),
    4: ((1.337764469960676383e-01, 6.243246901871899457e-01, 1.342537825644992244e+00, 2.262664477010361885e+00),
        (1.835325639596920577e-01, 2.375842404229175642e-01, 7.528686870428026590e-02, 3.596326913110175095e-03)),
    6: ((7.860065941318034044e-02, 3.867394102709340586e-01, 8.664294716825114984e-01, 1.465698049664053704e+00,
         2.172707796939548519e+00, 3.036820169323391827e+00),
        (1.110605364355289615e-01, 1.969891635526184459e-01, 1.451431417821328340e-01, 4.288582043761317297e-02,
         3.865781115609298168e-03, 5.555667649755732833e-05)),
    8: ((5.297864393185112986e-02, 2.673983721677653524e-01, 6.163028841823998683e-01, 1.064246312116224003e+00,
         1.588855862270055264e+00, 2.183921153095858436e+00, 2.863133883708075089e+00, 3.686007162724397102e+00),
        (7.566300718342849896e-02, 1.513894166189734825e-01, 1.556900326896759612e-01, 8.883068100100477427e-02,
         2.528365401139678892e-02, 3.028533438703043430e-03, 1.140022060541547879e-04, 6.728507633561610041e-07)),
}
_SIGN = ((1, 1, 1), (-1, 1, 1), (-1, -1, 1), (1, -1, 1), (1, 1, -1), (-1, 1, -1), (-1, -1, -1), (1, -1, -1))
_SIDES = "EWNSFB"   # fluid at +x, -x, +y, -y, +z, -z of a wall voxel; bit k of its mask
# re-emission of a wall (solver.F90:772-1823): destination store (F: the wall's slots, W: its
# 3-fold corner slots) and octant, face, mirrored source octant. The first face extrapolates
# into F, the second of three into W, the last of two or three into a temporary.
_WALLS = {
    "E": "F102 F403 F506 F807", "W": "F201 F304 F605 F708", "N": "F104 F203 F508 F607",
    "S": "F302 F401 F706 F805", "F": "F105 F206 F307 F408", "B": "F501 F602 F703 F804",
    "EN": "F102 F403 F506 F807 F213 F617 F314 F718", "WN": "F201 F304 F605 F708 F114 F518 F413 F817",
    "ES": "F102 F403 F506 F807 F312 F716 F211 F615", "WS": "F201 F304 F605 F708 F411 F815 F112 F516",
    "NF": "F104 F203 F508 F607 F317 F418 F716 F815", "NB": "F104 F203 F508 F607 F713 F814 F411 F312",
    "SF": "F302 F401 F706 F805 F115 F216 F617 F518", "SB": "F302 F401 F706 F805 F511 F612 F213 F114",
    "EF": "F102 F403 F506 F807 F216 F317 F615 F718", "EB": "F102 F403 F506 F807 F612 F713 F211 F314",
    "WF": "F201 F304 F605 F708 F115 F418 F516 F817", "WB": "F201 F304 F605 F708 F511 F814 F112 F413",
    "ENF": "F102 F403 F506 F807 F213 F617 F327 W114 W518 W226 W428 F725",
    "WNF": "F201 F304 F605 F708 F114 F518 F428 W213 W617 W125 W327 F826",
    "WSF": "F201 F304 F605 F708 F411 F815 F125 W312 W716 W226 W428 F527",
    "ESF": "F102 F403 F506 F807 F312 F716 F226 W411 W815 W125 W327 F628",
    "ENB": "F102 F403 F506 F807 F213 F617 F723 W114 W518 W622 W824 F321",
    "WNB": "F201 F304 F605 F708 F114 F518 F824 W213 W617 W521 W723 F422",
    "WSB": "F201 F304 F605 F708 F411 F815 F521 W312 W716 W622 W824 F123",
    "ESB": "F102 F403 F506 F807 F312 F716 F622 W411 W815 W521 W723 F224",
}
# the slot a reader behind a wall finds (solver.F90:184-204 and the seven like it), per octant:
# walls read by their y-upwind neighbour, then by their z-upwind neighbour; 0: the corner slots
_SWITCH = (
    ("EN3 ENF0 ENB0", "NF8 EF6 WNF0 ESF0 ENF7"), ("WN4 WNF0 WNB0", "NF7 WF5 ENF0 WSF0 WNF8"),
    ("WS1 WSF0 WSB0", "SF6 WF8 WNF0 ESF0 WSF5"), ("ES2 ESF0 ESB0", "SF5 EF7 ENF0 WSF0 ESF6"),
    ("EN7 ENF0 ENB0", "NB4 EB2 ESB0 WNB0 ENB3"), ("WN8 WNF0 WNB0", "NB3 WB1 ENB0 WSB0 WNB4"),
    ("WS8 WSF0 WSB0", "SB2 WB4 WNB0 ESB0 WSB1"), ("ES6 ESF0 ESB0", "SB1 EB3 ENB0 WSB0 ESB2"),
)


def _mask(name):
    return sum(1 << _SIDES.index(c) for c in name)


def _drill_and_thin(g):
    """One drill pass and one thin pass, in raster order, on a box with two ghost layers
    (0 fluid, 1 solid, 4 ghost). Both only open voxels, so a voxel that does not qualify at
    the start of a pass can only come to qualify through an opened neighbour."""
    gz, gy, gx = g.shape
    off = (1, gx, gx * gy)
    v = g.reshape(-1)
    lo, hi = (2, 2, 2), (gz - 2, gy - 2, gx - 2)
    inner = np.zeros(g.shape, bool)
    inner[lo[0]:hi[0], lo[1]:hi[1], lo[2]:hi[2]] = True
    inner = inner.reshape(-1)

    def narrow(a):   # fluid voxels one voxel wide along some axis
        solid = v != 0
        return np.logical_or.reduce([solid[a + o] & solid[a - o] for o in off])

    drillable = inner.copy().reshape(g.shape)
    drillable[:, :, 2] = drillable[:, :, gx - 3] = False
    drillable = drillable.reshape(-1)
    at = np.nonzero(drillable & (v == 0))[0]
    heap = at[narrow(at)].tolist()
    heapq.heapify(heap)
    while heap:
        p = heapq.heappop(heap)
        if not any(v[p + o] != 0 and v[p - o] != 0 for o in off):
            continue
        y, z = p // gx % gy, p // (gx * gy)
        y0, z0 = (-1 if y == gy - 3 else 0), (-1 if z == gz - 3 else 0)
        for dz in (z0, z0 + 1):
            for dy in (y0, y0 + 1):
                for dx in (0, 1):
                    q = p + dx + dy * gx + dz * gx * gy
                    if v[q] != 0:
                        v[q] = 0
                        if q > p and drillable[q]:
                            heapq.heappush(heap, q)
    ghost = ~inner
    v[ghost] = 0
    at = np.nonzero(inner & (v == 1))[0]
    two = np.logical_or.reduce([(v[at + o] == 0) & (v[at - o] == 0) for o in off])
    heap = at[two].tolist()
    heapq.heapify(heap)
    while heap:
        p = heapq.heappop(heap)
        if v[p] == 0:
            continue
        v[p] = 0
        for o in off:
            for q in (p - o, p + o):
                if q > p and inner[q] and v[q] == 1 and any(v[q + r] == 0 and v[q - r] == 0 for r in off):
                    heapq.heappush(heap, q)
    v[ghost] = 4


class _Exact:
    """The iteration on rows (voxel, octant) of velocities, FP64 throughout."""

    def __init__(self, case, img, kn):
        self.dev = dev = "cuda" if torch.cuda.is_available() else "cpu"
        fl = case["layer"]
        nz, ny, nx = img.shape
        nx += 2 * fl
        self.shape = (nz, ny, nx)
        g = np.full((nz + 4, ny + 4, nx + 4), 4, np.uint8)
        g[2:-2, 2:-2, 2:-2] = 0
        g[2:-2, 2:-2, 2 + fl:nx + 2 - fl] = img
        for _ in range(2):
            _drill_and_thin(g)
        gz, gy, gx = g.shape
        off = (1, gx, gx * gy)
        v = torch.from_numpy(g).to(dev).reshape(-1)
        ar = torch.arange(v.numel(), device=dev)
        cx = (ar % gx - 2, ar // gx % gy - 2, ar // (gx * gy) - 2)     # 0-based voxel coordinates
        n3 = (nx, ny, nz)
        fluid = v == 0
        solid = v == 1
        mask = torch.zeros_like(v, dtype=torch.int64)
        for k in range(6):
            d = off[k // 2] * (1 if k % 2 == 0 else -1)
            mask |= (torch.roll(fluid, -d) & solid).to(torch.int64) << k
        both = ((mask & 3) == 3) | ((mask & 12) == 12) | ((mask & 48) == 48)
        mask[both] = 0                                                 # such a solid has no label
        read = fluid.clone()
        for o in off:
            for d in (-2 * o, -o, o, 2 * o):
                read |= torch.roll(fluid, d) & solid
        nodes = torch.cat([torch.nonzero(fluid).reshape(-1), torch.nonzero(read & solid).reshape(-1)])
        self.nf = nf = int(fluid.sum())
        self.nodes, nn = nodes, nodes.numel()
        nodemap = torch.full_like(ar, -1)
        nodemap[nodes] = torch.arange(nn, device=dev)
        corner3 = (mask & 3 > 0) & (mask & 12 > 0) & (mask & 48 > 0)
        corner = torch.full_like(ar, -1)
        corner[corner3] = torch.arange(int(corner3.sum()), device=dev)
        self.ncorner = int(corner3.sum())
        self.fw0, self.zero = nn * 8, (nn + self.ncorner) * 8          # first corner row, the zero row
        xi, wi = (np.array(a) for a in _GH[case["nc"]])
        xi = xi * math.sqrt(2.0)
        n = case["nc"]
        t = lambda a: torch.tensor(np.ascontiguousarray(a.reshape(-1)), dtype=torch.float64, device=dev)  # noqa: E731
        z3, y3, x3 = np.meshgrid(xi, xi, xi, indexing="ij")
        self.c = (t(x3), t(y3), t(z3))
        self.w = t(wi[:, None, None] * wi[None, :, None] * wi[None, None, :])
        self.flux0 = 4.0 * float((self.c[2] * self.w).sum())
        self.nc8 = n ** 3
        self.ds = 1.0 / (nx - 1 - 2 * fl)
        self.mu, self.kn = math.sqrt(math.pi / 2.0) / kn, kn
        self.e = (1.0, 0.0) if case["order"] == 1 else (2.0, -1.0)

        # what a reader finds in a wall's slots, by octant and kind of read
        nb = nodes[nf:]
        nb_mask, nb_corner = mask[nb], corner[nb]
        tab = torch.full((8, 2, 64), -1, device=dev, dtype=torch.int64)
        for o in range(8):
            for axis in (0, 1):
                for r in _SWITCH[o][axis].split():
                    tab[o, axis, _mask(r[:-1])] = int(r[-1]) - 1 if r[-1] != "0" else 8

        def swept(p, o):
            ok = fluid[p]
            for a in range(3):
                ok = ok & ((cx[a][p] >= 1) if _SIGN[o][a] > 0 else (cx[a][p] <= n3[a] - 2))
            return ok

        own, rows, flags, key, commit = [], [[] for _ in range(6)], [[] for _ in range(3)], [], []
        self.sign = []
        base = torch.arange(nf, nn, device=dev) * 8
        for o in range(8):
            s = _SIGN[o]
            ys, zs = tab[o, 0][nb_mask], tab[o, 1][nb_mask]
            ysw = (ys >= 0) & swept(nb + s[1] * off[1], o)
            zsw = (zs >= 0) & swept(nb + s[2] * off[2], o)
            mine = torch.full_like(ys, o)
            after = torch.where(ysw, ys, mine)
            slot = [mine, mine, torch.where(ys >= 0, ys, mine), after, torch.where(zs >= 0, zs, after),
                    torch.where(zsw, zs, after)]
            seen = [torch.where(q < 8, base + q, self.fw0 + nb_corner * 8 + o) for q in slot]
            post = seen[5]
            moved = slot[5] != o
            commit.append(torch.stack([base[moved] + o, post[moved]]))
            f = nodes[:nf]
            f = f[swept(f, o)]
            up = [cx[a][f] if s[a] > 0 else n3[a] - 1 - cx[a][f] for a in range(3)]
            own.append(nodemap[f] * 8 + o)
            key.append(up[0] + up[1] + up[2])
            for a in range(3):
                p1, p2 = f - s[a] * off[a], f - 2 * s[a] * off[a]
                first = (up[a] == 1) | ((mask[p1] >> (2 * a + (0 if s[a] > 0 else 1))) & 1 > 0)
                flags[a].append(first)
                for q, p in ((2 * a, p1), (2 * a + 1, p2)):
                    nd = nodemap[p]
                    r = torch.where(nd >= nf, seen[q][(nd - nf).clamp(min=0)] if nb.numel() else nd, nd * 8 + o)
                    bad = (nd < 0) | (first if q % 2 else torch.zeros_like(first))
                    rows[q].append(torch.where(bad, torch.full_like(r, self.zero), r))
            self.sign.append(torch.tensor(s, dtype=torch.float64, device=dev))
        key = torch.cat(key)
        order = torch.argsort(key)
        self.starts = torch.searchsorted(key[order], torch.arange(int(key.max()) + 2, device=dev)).tolist()
        self.own = torch.cat(own)[order]
        self.rows = [torch.cat(r)[order] for r in rows]
        self.first = [torch.cat(f)[order].to(torch.float64)[:, None] for f in flags]
        self.sign = torch.stack(self.sign)
        self.commit = torch.cat(commit, 1)

        # walls by label; the far point of a face is needed only with second-order extrapolation
        self.walls, self.ok = [], True
        wall = nb[(nb_mask > 0)]
        for name, prog in _WALLS.items():
            p = wall[mask[wall] == _mask(name)]
            if not p.numel():
                continue
            faces = []
            for c in name:
                k = _SIDES.index(c)
                d = off[k // 2] * (1 if k % 2 == 0 else -1)
                inc = [o for o in range(8) if _SIGN[o][k // 2] == (-1 if k % 2 == 0 else 1)]
                far = nodemap[p + 2 * d]
                if self.e[1] and (bool((v[p + 2 * d] != 0).any())):
                    self.ok = False        # far points in walls or ghosts: order of the walls matters
                faces.append((k // 2, inc, nodemap[p + d], far))
            self.walls.append((nodemap[p], corner[p], faces, prog.split()))

        def plane(a, at):
            p = nodes[cx[a][nodes] == at]
            return p

        p1, pn = plane(0, 0), plane(0, nx - 1)
        west = nodemap[p1 + (nx - 1)]      # the node of the same row at the other end of the box
        east = nodemap[pn - (nx - 1)]
        self.inlet = (nodemap[p1], west, nodemap[pn], east)
        self.sym = [nodemap[plane(a, at)] for a, at in ((1, 0), (1, ny - 1), (2, 0), (2, nz - 1))]
        self.cells = [c[nodes[:nf]] for c in cx]
        f = torch.zeros
        self.F = f((self.zero + 1, self.nc8), dtype=torch.float64, device=dev)
        self.mom = f((nf, 4), dtype=torch.float64, device=dev)
        self.gw = f((p1.numel(), 4, self.nc8), dtype=torch.float64, device=dev)
        self.ge = f((pn.numel(), 4, self.nc8), dtype=torch.float64, device=dev)
        self.mass = 1.0

    def iterate(self):
        F, ds, mu = self.F, self.ds, self.mu
        for a, b in zip(self.starts[:-1], self.starts[1:]):
            if a == b:
                continue
            own = self.own[a:b]
            m = self.mom[own >> 3]
            s = self.sign[own & 7]
            cu = sum(s[:, k:k + 1] * m[:, k + 1:k + 2] * self.c[k] for k in range(3))
            num = mu * (self.w * (m[:, :1] + cu) - 0.5 * F[own])
            den = torch.full_like(num, 0.5 * mu)
            for k in range(3):
                f = self.first[k][a:b]
                num += self.c[k] * ((2.0 - f) / ds * F[self.rows[2 * k][a:b]]
                                    - (1.0 - f) * 0.5 / ds * F[self.rows[2 * k + 1][a:b]])
                den += self.c[k] * ((1.5 - 0.5 * f) / ds)
            F[own] = num / den
        F[self.commit[0]] = F[self.commit[1]]
        pos, neg = [0, 3, 4, 7], [1, 2, 5, 6]
        n1, west, nn, east = self.inlet
        F3 = F[:self.fw0].view(-1, 8, self.nc8)
        W3 = F[self.fw0:self.zero].view(-1, 8, self.nc8)
        gw, ge = self.gw, self.ge
        self.gw = torch.where((west >= 0)[:, None, None], F3[west.clamp(min=0)][:, pos], torch.zeros_like(gw))
        self.ge = torch.where((east >= 0)[:, None, None], F3[east.clamp(min=0)][:, neg], torch.zeros_like(ge))
        for node, corner, faces, prog in self.walls:
            val, rho = [], []
            for axis, inc, near, far in faces:
                e = F3[near][:, inc] * self.e[0]
                if self.e[1]:
                    e = e + F3[far][:, inc] * self.e[1]
                val.append({o: e[:, q] for q, o in enumerate(inc)})
                rho.append((e.sum(1) * self.c[axis]).sum(1, keepdim=True) / self.flux0)
            for o, x in val[0].items():
                F3[node, o] = x
            if len(faces) == 3:
                for o, x in val[1].items():
                    W3[corner, o] = x
            for wr in prog:                # accommodation 1: the mirrored part has weight 0
                x = self.w * rho[int(wr[2])]
                if wr[0] == "F":
                    F3[node, int(wr[1]) - 1] = x
                else:
                    W3[corner, int(wr[1]) - 1] = x
        for q, o in enumerate(pos):
            F3[n1, o] = gw[:, q] + self.w
        for q, o in enumerate(neg):
            F3[nn, o] = ge[:, q] - self.w
        for p, pairs in zip(self.sym, (((1, 2), (0, 3), (5, 6), (4, 7)), ((2, 1), (3, 0), (6, 5), (7, 4)),
                                       ((0, 4), (1, 5), (2, 6), (3, 7)), ((4, 0), (5, 1), (6, 2), (7, 3)))):
            for dst, src in pairs:
                F3[p, dst] = F3[p, src]
        for a in range(0, self.nf, 1 << 18):
            f = F3[a:min(self.nf, a + (1 << 18))]
            self.mom[a:a + f.shape[0], 0] = f.sum((1, 2))
            for k in range(3):
                self.mom[a:a + f.shape[0], k + 1] = ((f * self.sign[:, k][None, :, None]).sum(1) * self.c[k]).sum(1)

    def check(self):
        nz, ny, nx = self.shape
        x, y, z = self.cells
        at = x == 1
        half = lambda c, n: torch.where((c == 0) | (c == n - 1), 0.5, 1.0).double()  # noqa: E731
        m = float((self.mom[at, 1] * half(y[at], ny) * half(z[at], nz)).sum()) * self.ds ** 2 * math.sqrt(0.5)
        err = abs(1.0 - m / self.mass) / STEP
        self.mass = m
        return m, m * self.kn * math.sqrt(4.0 / math.pi), err

    def fields(self):
        out = {}
        x, y, z = self.cells
        for k, name in enumerate(("rho", "ux", "uy", "uz")):
            a = torch.zeros(self.shape, dtype=torch.float64, device=self.dev)
            a[z, y, x] = self.mom[:, k]
            out[name] = a.cpu().numpy()
        return out


def _exact_solve(case, seed):
    img, kn = _image(case, seed)
    s = _Exact(case, img, kn)
    if not s.ok:
        return None
    checks = []
    for _ in range(case["checks"]):
        for _ in range(STEP):
            s.iterate()
        checks.append(s.check())
    return {"checks": np.array(checks), "fields": s.fields()}


def exact(case, seed):
    """run()'s outputs in 64 bits. None for a refined solve: it ends within its tolerance of
    the limit, at a number of iterations that its stopping rule picks; and for boxes so large
    that this plain version takes too long."""
    if case["kind"] == "refined":
        return None
    parts = _members(case, seed) if case["kind"] == "batch" else [(case, seed)]
    cost = 0.0   # seconds on the GPU: each hyperplane's launches, and the updates' traffic
    for c, _ in parts:
        nx = c["nx"] + 2 * c["layer"]
        updates = c["porosity"] * nx * c["ny"] * c["nz"] * 8 * c["nc"] ** 3
        cost += c["checks"] * STEP * ((nx + c["ny"] + c["nz"]) * 3.5e-4 + updates * 1.2e-10)
    if cost > 20.0 or sum(c["nx"] * c["ny"] * c["nz"] for c, _ in parts) > 5e6:
        return None
    got = [_exact_solve(c, sd) for c, sd in parts]
    if any(g is None for g in got):
        return None
    if case["kind"] == "batch":
        return {"checks": np.stack([g["checks"] for g in got], 2), "fields": [g["fields"] for g in got]}
    return got[0]
