"""GPU tests of the mixed-precision solve after one that failed: a right-hand side beyond the FP32 range
makes the inner solve return SULI_ERR_NAN, and the context's next solve gives the bits of a fresh
context's, on the streaming and the vectorised level-0 kernels, from the graph and from the host."""
import numpy as np
import pytest

from helpers import load_state, seeded_state, small_params

pytestmark = pytest.mark.gpu


def _solve(s, p):
    load_state(s, seeded_state(p, 3))
    s.heaviside()
    s.set_dt(1e-3)
    s.contorno(2)
    n, _ = s.graddin()
    return n, s.download("prd1")


@pytest.mark.parametrize("eager", ["0", "1"])
@pytest.mark.parametrize("shape", [(32, 16, 16), (64, 20, 12), (40, 12, 16)])
def test_solve_after_overflow(pkg, monkeypatch, shape, eager):
    monkeypatch.setenv("SULI_EAGER_LOOPS", eager)
    p = small_params(*shape)
    p.precision, p.cg_stop, p.cg_tol, p.inner_tol, p.refine_maxit = 1, 1, 1e-8, 1e-3, 40
    with pkg.Solver(p) as s:
        want = _solve(s, p)
    with pkg.Solver(p) as s:
        load_state(s, seeded_state(p, 3))
        s.heaviside()
        s.set_dt(1e-3)
        s.upload("u", 1e39 * np.random.default_rng(1).standard_normal(s.shape("u")))
        with pytest.raises(pkg.SuliError) as ei:
            s.graddin()
        assert ei.value.code == pkg._abi.ERR_NAN
        got = _solve(s, p)
    assert got[0] == want[0]
    assert np.array_equal(got[1], want[1])
