"""Level-set transport forms only the upwind WENO derivative of each axis: against the CPU oracle for
every sign of the velocity (and exact zeros), at tile edges and on grids where every cell sees the
boundary rules.  Tolerance as the level-set parity test's: 1e-12 of each field's scale."""
import numpy as np
import pytest

from helpers import OUT_FIELDS, load_state, rel_err, seeded_state, small_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bc", [(2, 2, 2, 2, 2, 1), (0, 0, 2, 2, 2, 1), (2, 4, 1, 1, 2, 1)])
@pytest.mark.parametrize("signs", ["plus", "minus", "mixed"])
@pytest.mark.parametrize("shape", [(4, 5, 6), (7, 6, 5), (32, 8, 8), (33, 9, 8)])
def test_upwind_side(pkg, orc, shape, signs, bc):
    p = small_params(*shape, bc=bc)
    g, o = pkg.Solver(p), orc.Oracle(p)
    st = seeded_state(p, 3)
    rng = np.random.default_rng(11)
    for f in ("u", "v", "w"):
        a = 0.2 * rng.random(st[f].shape)
        if signs == "minus":
            a = -a
        if signs == "mixed":
            a = np.where(rng.random(a.shape) < 0.3, 0.0, a - 0.1)
        st[f] = a
    for m in (g, o):
        load_state(m, st)
        m.level_set_ini()
        m.set_dt(2e-3)
        m.level_set()
    for f in OUT_FIELDS["level_set"]:
        a, b = g.download(f), o.download(f)
        assert rel_err(a, b) <= 1e-12, (f, rel_err(a, b))
