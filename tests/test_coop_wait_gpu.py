"""GPU tests of the cooperative FP64 CG's grid-wide waits: a wait that runs out fails the solve and leaves
the context usable, and contexts that solve at the same time on their own streams and threads do
not disturb one another."""
import threading

import numpy as np
import pytest

from helpers import load_state, seeded_state, small_params

pytestmark = pytest.mark.gpu

WALLS = (2, 2, 2, 2, 2, 1)
PERIODIC = (0, 0, 0, 0, 0, 0)
# one sum an iteration, two sums in registers (clamped periodic faces), two passes over memory
KERNELS = [((25, 50, 45), WALLS), ((25, 50, 45), PERIODIC), ((66, 50, 48), WALLS)]


def _params(shape, bc):
    p = small_params(*shape, bc=bc)
    p.cg_stop, p.cg_tol, p.cg_maxit = 1, 1e-6, 2000
    if bc == PERIODIC:   # CG need not converge on the asymmetric operator: a fixed number of iterations
        p.cg_tol, p.cg_maxit = 1e-30, 100
    return p


def _solve(s, p, seed=3):
    load_state(s, seeded_state(p, seed))
    s.heaviside()
    s.set_dt(1e-3)
    s.contorno(2)
    n, _ = s.graddin()
    return n, s.download("prd1")


@pytest.mark.parametrize("shape,bc", KERNELS)
def test_wait_that_runs_out(pkg, monkeypatch, shape, bc):
    p = _params(shape, bc)
    with pkg.Solver(p) as s:
        want = _solve(s, p)
    with pkg.Solver(p) as s:
        monkeypatch.setenv("SULI_COOP_POLLS", "1")   # whoever arrives first gives up after one look
        with pytest.raises(pkg.SuliError) as ei:
            _solve(s, p)
        assert ei.value.code == pkg._abi.ERR_CUDA
        monkeypatch.delenv("SULI_COOP_POLLS")
        got = _solve(s, p)
    assert got[0] == want[0]
    assert np.array_equal(got[1], want[1])


@pytest.mark.parametrize("shape,bc", KERNELS)
def test_two_contexts_at_once(pkg, shape, bc):
    p = _params(shape, bc)
    want = {}
    for seed in (3, 4):
        with pkg.Solver(p) as s:
            want[seed] = _solve(s, p, seed)
    got, errors = {}, []
    start = threading.Barrier(2)

    def work(seed):
        try:
            with pkg.Solver(p) as s:
                start.wait(60)
                for _ in range(3):
                    got[seed] = _solve(s, p, seed)
        except Exception as e:   # noqa: BLE001 - reported by the main thread
            errors.append(e)

    threads = [threading.Thread(target=work, args=(seed,)) for seed in (3, 4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for seed in (3, 4):
        assert got[seed][0] == want[seed][0]
        assert np.array_equal(got[seed][1], want[seed][1])
