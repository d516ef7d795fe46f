"""GPU test of gradients taken by two networks on two threads at once: each keeps what it asked the device
about its kernels, so the bits are those of one network after the other."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _gradient(pkg, shape, seed):
    torch = pytest.importorskip("torch")
    nx, ny, nz = shape
    rng = np.random.default_rng(seed)
    x3 = torch.from_numpy(rng.standard_normal((nx * ny * nz, 3)).astype(np.float32)).to("cuda:0")
    t = torch.from_numpy(rng.standard_normal(nx * ny * nz).astype(np.float32)).to("cuda:0")
    torch.cuda.synchronize()
    net = pkg.learned.Net(nx, ny, nz, params=pkg.learned.init_params(seed, head_scale=1.0))
    out = [net.loss_grad(x3, t)[1] for _ in range(3)]
    net.close()
    assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])
    return out[0]


def test_two_threads(pkg):
    jobs = [((24, 40, 72), 3), ((40, 24, 16), 4)]
    got, errors = {}, []
    start = threading.Barrier(len(jobs))

    def work(shape, seed):
        try:
            start.wait(60)
            got[seed] = _gradient(pkg, shape, seed)
        except Exception as e:   # noqa: BLE001 - reported by the main thread
            errors.append(e)

    threads = [threading.Thread(target=work, args=job) for job in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for shape, seed in jobs:
        assert np.array_equal(got[seed], _gradient(pkg, shape, seed))
