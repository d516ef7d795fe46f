"""GPU tests of the FP64 CG as two kernels an iteration (SULI_NO_COOP=1, and devices or contexts that refuse
the cooperative launch): its iterations run in a device-side loop, without the host between them, and
give the bits of the same kernels launched one by one (SULI_EAGER_LOOPS=1)."""
import numpy as np
import pytest

from helpers import load_state, seeded_state, small_params

pytestmark = pytest.mark.gpu


def _solve(pkg, p, monkeypatch, eager):
    monkeypatch.setenv("SULI_NO_COOP", "1")
    monkeypatch.setenv("SULI_EAGER_LOOPS", eager)
    with pkg.Solver(p) as s:
        load_state(s, seeded_state(p, 3))
        s.heaviside()
        s.set_dt(1e-3)
        s.contorno(2)
        s.profile_enable(True)
        n, r = s.graddin()
        prof = s.profile_read()
        return n, r, s.download("prd1"), prof


# odd and even rows; solves that the divergence test resumes after odd and even numbers of iterations,
# and ones it does not
@pytest.mark.parametrize("shape", [(14, 12, 10), (13, 9, 7), (33, 20, 18)])
@pytest.mark.parametrize("tol,div_tol", [(1e-2, 1e-8), (2e-3, 1e-8), (5e-4, 1e-8), (1e-4, 0.0), (1e-8, 0.0)])
def test_loop_matches_single_launches(pkg, monkeypatch, shape, tol, div_tol):
    p = small_params(*shape)
    p.cg_stop, p.cg_tol, p.cg_maxit, p.div_tol = 1, tol, 20000, div_tol
    na, ra, a, prof = _solve(pkg, p, monkeypatch, "0")
    nb, rb, b, _ = _solve(pkg, p, monkeypatch, "1")
    assert (na, ra) == (nb, rb)
    assert np.array_equal(a, b)
    # the update kernels of the loop count as launched but are timed with the loop, as the product's:
    # at most one update a run of the loop is launched, and timed, by itself
    assert prof["cg_update"]["launches"] >= na
    assert prof["cg_update"]["ms"] < 0.2 * prof["cg_spmv"]["ms"]


@pytest.mark.parametrize("maxit", [0, 1, 2, 3])
def test_few_iterations(pkg, monkeypatch, maxit):
    p = small_params(14, 12, 10)
    p.cg_stop, p.cg_tol, p.cg_maxit = 1, 1e-12, maxit
    na, ra, a, _ = _solve(pkg, p, monkeypatch, "0")
    nb, rb, b, _ = _solve(pkg, p, monkeypatch, "1")
    assert na == nb == maxit and ra == rb
    assert np.array_equal(a, b)
