"""Launches of a time step: suli_step chains its kernels (dependent launches), the single calls start
plainly after whatever the caller put on the stream.  Both must give the same bits, and the copies
of the pressure that the convection and projection kernels carry must cover the whole halo box."""
import numpy as np
import pytest

from helpers import pkg, small_params

pytestmark = pytest.mark.gpu

# tile edges (32 x 8 threads, 4 and 8 planes a thread), remainders, the smallest grid
SIZES = [(12, 10, 9), (31, 7, 8), (32, 8, 4), (33, 9, 5), (64, 16, 12), (4, 4, 4)]
FIELDS = ["u", "v", "w", "prd", "prd0", "prd1", "ls", "rho", "ub", "vb", "wb", "Fu", "Fv", "Fw"]


def _start(p):
    s = pkg.Solver(p)
    s.iniciais(0.0)
    rng = np.random.default_rng(7)
    nz = p.nz
    k = np.arange(s.shape("ls")[2], dtype=np.float64)
    ls = np.broadcast_to((k - 0.5 * nz) * p.dz, s.shape("ls"))
    s.upload("ls", np.asfortranarray(ls + 0.2 * p.dz * rng.standard_normal(s.shape("ls"))))
    for f in ("u", "v", "w", "prd1"):
        s.upload(f, 1e-2 * rng.standard_normal(s.shape(f)))
    s.level_set_ini()
    s.contorno(1)
    return s


# the mixed path's grids halve down to its coarsest level
MIXED = [(16, 8, 8), (32, 16, 8), (48, 24, 16), (64, 20, 12), (40, 12, 16)]


@pytest.mark.parametrize("nx,ny,nz,precision", [s + (0,) for s in SIZES] + [s + (1,) for s in MIXED])
def test_step_equals_its_calls(nx, ny, nz, precision):
    p = small_params(nx, ny, nz)
    p.precision = precision
    p.cg_stop = 1
    p.cg_tol = 1e-8
    a, b = _start(p), _start(p)
    for it in (1, 2):
        a.step(it)
        b.level_set()
        for tt in range(1, b.ntt + 1):
            b.set_dt(b.a_dt[tt - 1])
            for call in (b.visco, b.convdiff, lambda: b.tempo(tt, it), lambda: b.contorno(2), b.graddin, b.posdin,
                         lambda: b.contorno(1)):
                b.upload("u", b.download("u"))   # copies between the calls
                call()
    for f in FIELDS:
        np.testing.assert_array_equal(a.download(f), b.download(f), err_msg=f)


@pytest.mark.parametrize("nx,ny,nz", SIZES)
def test_pressure_copies_cover_the_halo(nx, ny, nz):
    p = small_params(nx, ny, nz)
    s = _start(p)
    prd1 = np.asfortranarray(np.random.default_rng(3).standard_normal(s.shape("prd1")))
    s.upload("prd1", prd1)
    s.visco()
    s.convdiff()
    np.testing.assert_array_equal(s.download("prd0"), prd1)
    s.posdin()
    np.testing.assert_array_equal(s.download("prd"), prd1)
    np.testing.assert_array_equal(s.download("prd1"), prd1)
