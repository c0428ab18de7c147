"""Short characteristics at every width of the upstream patch's staging copies (16, 8
and 4 bytes: the frequencies' count and the work array's alignment decide), tiles cut
off in x, y and frequency, and a chain of many planes, bit for bit against the oracle."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _work(rng, nf, nx, ny, nz, dt=np.float32):
    w = np.empty((3, nz + 2, ny, nx, nf), dt)
    w[0] = 10.0 ** rng.uniform(-9.0, -6.0, w[0].shape)
    w[1:] = rng.uniform(0.1, 2.0, w[1:].shape)
    return w


@pytest.mark.parametrize("nf", [1, 2, 3, 4, 30, 31, 32, 33, 34, 36, 65])
@pytest.mark.parametrize("shape", [(8, 8, 2), (17, 9, 23), (1, 1, 5), (5, 30, 7)])
@pytest.mark.parametrize("dir", [1, -1])
def test_short_char_shapes(m3d, oracle, nf, shape, dir):
    nx, ny, nz = shape
    rng = np.random.default_rng(nf + 100 * nx)
    vec = np.array([0.31, -0.22, dir * math.sqrt(1 - 0.31**2 - 0.22**2)])
    ds = [1.2e7, 1.0e7, 0.8e7]
    work = _work(rng, nf, nx, ny, nz)
    out = {}
    for mod in (oracle, m3d):
        w = work.copy()
        p = [np.zeros((nz, ny, nx, nf), np.float32) for _ in range(3)]
        slab = mod.make_slab(nf, nx, ny, nz, dir, ds, vec, get_psi=True, split_rates=True)
        mod.formal_solve(mod.SHORT_LINEAR, slab, w, psi=p[0], irem=p[1], escape=p[2])
        out[mod] = [w] + p
    for a, b in zip(out[m3d], out[oracle]):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("offset", [1, 2, 3])
def test_short_char_unaligned_work(m3d, oracle, offset):
    """A device work array that starts between 16-byte boundaries."""
    import torch
    nf, nx, ny, nz = 32, 10, 9, 6
    rng = np.random.default_rng(3)
    vec = np.array([-0.2, 0.35, math.sqrt(1 - 0.04 - 0.35**2)])
    ds = [1.2e7, 1.0e7, 0.8e7]
    work = _work(rng, nf, nx, ny, nz)
    ref = work.copy()
    oracle.formal_solve(oracle.SHORT_LINEAR, oracle.make_slab(nf, nx, ny, nz, 1, ds, vec), ref)
    buf = torch.empty(work.size + offset, dtype=torch.float32, device="cuda")
    w = buf[offset:].view(work.shape)
    w.copy_(torch.from_numpy(work))
    m3d.formal_solve(m3d.SHORT_LINEAR, m3d.make_slab(nf, nx, ny, nz, 1, ds, vec), w)
    np.testing.assert_array_equal(w.cpu().numpy(), ref)


@pytest.mark.parametrize("nf", [5, 6, 32])
def test_short_char_double(m3d, oracle, nf):
    nx, ny, nz = 11, 9, 7
    rng = np.random.default_rng(nf)
    vec = np.array([0.25, 0.4, math.sqrt(1 - 0.0625 - 0.16)])
    ds = [1.2e7, 1.0e7, 0.8e7]
    work = _work(rng, nf, nx, ny, nz, np.float64)
    out = []
    for mod in (oracle, m3d):
        w = work.copy()
        mod.formal_solve(mod.SHORT_LINEAR, mod.make_slab(nf, nx, ny, nz, 1, ds, vec), w)
        out.append(w)
    np.testing.assert_allclose(out[1], out[0], rtol=1e-12)
