"""The streaming level-0 kernels on a periodic y axis (the wrapped row behind a tile's box) against the
vectorised level-0 kernels (SULI_NO_STREAM=1): per cell the same arithmetic, the FP64 dot products
grouped differently, so a step agrees within the solve's tolerance 1e-10: iteration counts within
2, velocities within 1e-9 of their scale."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("perz", [False, True])
@pytest.mark.parametrize("shape,chunk", [((128, 64, 64), None), ((64, 36, 24), None), ((32, 12, 16), None),
                                         ((48, 20, 32), None), ((128, 32, 64), "7"), ((32, 8, 16), None)])
def test_periodic_y_matches_vectorised(pkg, monkeypatch, shape, chunk, perz):
    # full tiles; rows that are no multiple of the 8-row tile; few rows; nx = 48 (vectorised
    # post-smoothing); a ring that wraps and a last CTA of one plane; 8 rows (vectorised throughout)
    if chunk:
        monkeypatch.setenv("SULI_STREAM_CHUNK", chunk)
    nx, ny, nz = shape
    res = {}
    for ns in ("1", "0"):
        monkeypatch.setenv("SULI_NO_STREAM", ns)
        p, init = pkg.cases.dam_break(nx=nx, ny=ny, nz=nz, dx=0.005, cg_tol=1e-10)
        p.precision, p.inner_tol, p.refine_maxit = 1, 1e-4, 30
        p.ccy0 = p.ccyf = 0
        if perz:   # one fluid without gravity (a dam across a periodic z axis is no valid problem)
            p.ccz0 = p.cczf = 0
            p.rho_f1, p.mi_f1, p.gz = p.rho_f2, p.mi_f2, 0.0
        s = pkg.Solver(p)
        init(s)
        v = s.download("v")
        j, k = np.meshgrid(np.arange(v.shape[1]), np.arange(v.shape[2]), indexing="ij")
        v += 0.1 * np.sin(2 * np.pi * (j - 1) / ny) * np.cos(np.pi * k / nz)   # flow across the wrap
        s.upload("v", np.asfortranarray(v))
        s.contorno(1)
        steps = [s.step(1)]
        assert all(st["status"] == 0 for st in steps)
        res[ns] = ([sum(st["cg_iters"]) for st in steps], {f: s.download(f) for f in ("u", "v", "w")})
        s.close()
    (i1, v1), (i0, v0) = res["1"], res["0"]
    assert all(abs(a - b) <= 2 for a, b in zip(i1, i0)), (i1, i0)
    vs = max(float(np.abs(b).max()) for b in v1.values())
    for f in v1:
        assert float(np.abs(v1[f] - v0[f]).max()) <= 1e-9 * vs, f
