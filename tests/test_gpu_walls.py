"""GPU tests of the wall kernels that keep a wall's rows on chip (csrc/kernels.cu, kernels_fp32.cu) and
of the FP32 moments: octants of 8, 64, 216 and 512 velocities, walls that read their second
extrapolation point (orders 2 and 3) and walls that do not (order 1), odd node counts.

FP64 against the oracle, tolerance 0 (same operations in the same order). FP32 f against the
oracle's within 1e-5 of max|f| after three iterations (each value passes through some ten FP32
roundings of 6e-8 per iteration and up to some tens of cells). FP32 moments against the FP64 sums
of the same f: n terms summed in another order differ by at most n * 2^-53 * sum |c f| per side."""
import numpy as np
import pytest

import piks3d_b200 as pk
from conftest import base_params
from oracle import Oracle
from piks3d_b200 import images

pytestmark = pytest.mark.gpu

# velocity signs of the octants for the moments Rho, Ux, Uy, Uz
SIGNS = ((1,) * 8, (1, -1, -1, 1, 1, -1, -1, 1), (1, 1, -1, -1, 1, 1, -1, -1), (1, 1, 1, 1, -1, -1, -1, -1))

CASES = [(nf, order) for nf in (2, 4, 6, 8) for order in (1, 2, 3)]


def _case(nf, order):
    img = images.sphere_pack(13, 0.5, 1.2, 3.0, seed=20 + nf)[:11, :12, :].copy()
    p = base_params(13, Nx=13, Ny=12, Nz=11, Nc_fundamental=nf, Kn=0.7, wallExtOrder=order, fluidlayer=1, accom=0.9)
    o = Oracle(p, img.tobytes(), nthreads=8)
    o.iterate(3)
    return img, p, o


@pytest.mark.parametrize("nf,order", CASES)
def test_fp64_walls_equal_the_oracle(nf, order):
    img, p, o = _case(nf, order)
    with pk.Solver(p, device=0) as s:
        s.setup_physical_grid(img)
        s.iterate(3)
        nodes, nc8 = s.geometry_array("node_g"), s.info()["Nc8"]
        f, fw = s.get_f()
        assert np.array_equal(o.f().reshape(8, nc8, -1)[:, :, nodes], f.reshape(8, nc8, -1)[:, :, nodes])
        assert np.array_equal(o.fw(), fw)
        for a, b in zip(o.macro(), s.get_macro()):
            assert np.array_equal(a[2:-2, 2:-2, 2:-2], b)


@pytest.mark.parametrize("nf,order", CASES)
def test_fp32_walls_and_moments(nf, order):
    img, p, o = _case(nf, order)
    with pk.Solver(p, device=0) as s:
        s.set_precision(pk.PREC_FP32)
        s.setup_physical_grid(img)
        s.iterate(3)
        inf = s.info()
        nodes, nc8 = s.geometry_array("node_g"), inf["Nc8"]
        f = s.get_f()[0].reshape(8, nc8, -1)[:, :, nodes]
        fo = o.f().reshape(8, nc8, -1)[:, :, nodes]
        assert np.abs(f - fo).max() <= 1e-5 * np.abs(fo).max()
        fluid = f[:, :, :inf["Nfluid"]]
        g = nodes[:inf["Nfluid"]].astype(np.int64)
        gx, gy = inf["Nx"] + 4, inf["Ny"] + 4
        at = (g % gx - 2) + (g // gx % gy - 2) * inf["Nx"] + (g // (gx * gy) - 2) * inf["Nx"] * inf["Ny"]
        for name, signs, got in zip(("", "cx", "cy", "cz"), SIGNS, s.get_macro()):
            c = s.geometry_array(name) if name else np.ones(nc8)
            terms = np.array(signs)[:, None, None] * c[None, :, None] * fluid
            bound = 2 * 8 * nc8 * 2.0 ** -53 * np.abs(terms).sum(axis=(0, 1))
            assert np.all(np.abs(got.ravel()[at] - terms.sum(axis=(0, 1))) <= bound)


def test_wall_launches_are_counted_as_launched():
    """Walls that read their first extrapolation point only are one launch, others one per level."""
    img = images.sphere_pack(16, 0.45, 1.2, 3.0, seed=5)
    n = {}
    for order in (1, 2):
        with pk.Solver(base_params(16, wallExtOrder=order), device=0) as s:
            s.setup_physical_grid(img)
            n[order], levels = s.launches_per_iteration(), s.info()["nWallLevels"]
    assert levels > 1 and n[2] - n[1] == levels - 1
