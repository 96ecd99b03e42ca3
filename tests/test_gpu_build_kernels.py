"""The kernels around the solve: the sphere mask (FP32 decisions away from the
surface, FP64 near it) and the right-hand side (power-of-two spacings by exponent)
bit for bit against the oracle, the residual on isotropic grids."""
import numpy as np
import pytest

import bbpp
from bbpp import problems

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,bc,scale", [((40, 24, 33), "ppp", 1.0), ((31, 45, 20), "nnn", 1.0),
                                           ((64, 32, 16), "pnp", 1e-20), ((20, 20, 20), "ppn", 1e22)])
def test_sphere_mask_near_the_surface(bbpp_lib, orc, dims, bc, scale):
    """Centres on cell centres and faces with radii of whole and half cells put cells
    exactly on the surface; radii below a cell, across seams and walls, beyond the
    box; lengths whose squares leave FP32's range."""
    nx, ny, nz = dims
    g = bbpp.Grid.make(nx, ny, nz, scale / nx, 0.9 * scale / ny, 1.1 * scale / nz, problems.bc_tuple(bc))
    rng = np.random.default_rng(nx)
    c = rng.random((40, 3)) * [nx, ny, nz]
    c[:10] = np.floor(c[:10]) + 0.5
    c[10:20] = np.floor(c[10:20])
    c[20] = [0.0, 0.0, 0.0]
    c[21] = [nx, ny / 2, nz]
    r = np.concatenate([np.arange(1, 11), np.arange(1, 11) + 0.5, rng.random(20) * 6 + 0.01])
    r[30], r[31] = 0.3, 0.001
    d = np.array([g.dx, g.dy, g.dz])
    cents, radii = c * d, r * g.dx
    s = bbpp.Solver(g)
    out = bbpp.DeviceArray(g.shape, np.uint8)
    for k in (40, 7, 40):  # the buffer of the spheres grows and is kept
        s.sphere_mask(cents[:k], radii[:k], out)
        assert np.array_equal(out.download(), orc.sphere_mask(orc.from_tuple(g.as_tuple()), cents[:k], radii[:k]))


@pytest.mark.parametrize("dims,spacing", [((64, 16, 32), (1 / 64, 1 / 16, 1 / 32)), ((33, 7, 5), (0.25, 0.1, 4.0)),
                                          ((17, 9, 3), (0.3, 0.7, 1.1)), ((8, 8, 8), (2.0 ** -300, 2.0 ** 200, 1.0))])
def test_rhs_div_bit_exact(bbpp_lib, orc, dims, spacing):
    nx, ny, nz = dims
    g = bbpp.Grid.make(nx, ny, nz, *spacing, problems.bc_tuple("ppp"))
    rng = np.random.default_rng(nx)
    u, v, w = (rng.normal(size=s) for s in ((nz, ny, nx + 1), (nz, ny + 1, nx), (nz + 1, ny, nx)))
    for a in (u, v, w):  # zero differences, subnormal and huge ones
        f = a.reshape(-1)
        f[::7] = 0.0
        f[1::7] = 0.0
        f[2::31] = 4e-310
        f[3::37] = 1e306
    s = bbpp.Solver(g)
    du, dv, dw = (bbpp.DeviceArray.from_host(a) for a in (u, v, w))
    out = bbpp.DeviceArray(g.shape, np.float64)
    s.rhs_div(1.7, 1e-3, du, dv, dw, out)
    with np.errstate(all="ignore"):
        want = orc.rhs_div(orc.from_tuple(g.as_tuple()), 1.7, 1e-3, u, v, w)
    assert np.array_equal(out.download(), want, equal_nan=True)


@pytest.mark.parametrize("dims,bc", [((32, 8, 9), "ppp"), ((33, 9, 40), "nnn"), ((5, 17, 3), "npn")])
@pytest.mark.parametrize("xsum", [True, False])
def test_residual_isotropic(bbpp_lib, orc, dims, bc, xsum):
    nx, ny, nz = dims
    g = bbpp.Grid.make(nx, ny, nz, 0.125, 0.125, 0.125, problems.bc_tuple(bc))
    rng = np.random.default_rng(ny)
    mask = (rng.random(g.shape) < 0.1).astype(np.uint8)
    b, x = rng.normal(size=g.shape), rng.normal(size=g.shape)
    s = bbpp.Solver(g)
    s.set_xsum(xsum)
    r = bbpp.DeviceArray(g.shape, np.float64)
    rr, bb = s.residual(bbpp.DeviceArray.from_host(b), bbpp.DeviceArray.from_host(x), r,
                        bbpp.DeviceArray.from_host(mask))
    ref = b - orc.spmv(orc.from_tuple(g.as_tuple()), x, mask)
    # a cell's rounding: under ten operations on terms of the stencil's size
    assert np.abs(r.download() - ref).max() <= 10 * 2.0 ** -53 * 12 / 0.125 ** 2 * np.abs(x).max()
    assert abs(rr - (ref * ref).sum()) <= 1e-12 * rr and abs(bb - (b * b).sum()) <= 1e-12 * bb
