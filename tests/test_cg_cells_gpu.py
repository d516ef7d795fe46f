"""The register kernels of the cooperative FP64 CG at three and at four cells a thread: the largest
grid of the one on 148 SMs (64 x 48 x 37 = 113,664 cells) and one plane more, for the symmetric
operator (one sum an iteration) and the asymmetric one (periodic axes with the clamped end faces,
two sums).  Against two kernels an iteration, with the tolerances of test_cg_coop_gpu.py."""
import pytest

from helpers import rel_err, small_params
from test_cg_coop_gpu import PERIODIC, WALLS, _solve

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bc", [WALLS, PERIODIC])
@pytest.mark.parametrize("shape", [(5, 7, 22), (64, 48, 37), (64, 48, 38)])
def test_three_and_four_cells_a_thread(pkg, monkeypatch, shape, bc):
    p = small_params(nx=shape[0], ny=shape[1], nz=shape[2], bc=bc)
    p.cg_stop, p.cg_tol, p.cg_maxit = 1, 1e-30, 30
    na, ra, a = _solve(pkg, p, False, monkeypatch, twice=True)
    nb, rb, b = _solve(pkg, p, True, monkeypatch)
    assert na == nb == 30
    assert abs(ra - rb) <= 1e-9 * rb
    assert rel_err(a, b) <= 1e-9
