"""The LTE pass at every form of its line-opacity kernel: window sizes at the edges
of the register counts (8, 16, 32, 48, 64 frequencies a lane, then 2, 4, 8, 16 lanes a
cell) and below them, rays sharing a launch, and one cell column; bit for bit against
the oracle."""
import numpy as np
import pytest

from dispatch_b200 import synth

pytestmark = pytest.mark.gpu


def _case(nf, nray, size=None):
    atm, _, _, vec, wmu = synth.lte_config("mini", nf=16)
    llam, nu = synth.frequency_grid(5000.5, 5000.5 + 0.01 * nf, nf)
    # one ray leaning in x and y among them: the sheared planes of the sweep
    pick = [0, 5, 12][:nray]
    return atm, nu, llam, np.ascontiguousarray(vec[pick]), np.ascontiguousarray(wmu[pick])


@pytest.mark.parametrize("nf", [2, 7, 8, 9, 15, 16, 17, 31, 33, 45, 48, 49, 63, 64, 65, 66, 127, 128, 129, 250, 257,
                                513, 1000])
def test_window_sizes(m3d, oracle, nf):
    from oracle import pipeline as P
    atm, nu, llam, vec, wmu = _case(nf, 1 if nf > 128 else 3)
    ie, flux, top = m3d.lte_synthesis(atm, nu, llam, vec, wmu, return_itop=True)
    oie, oflux, otop = P.lte_synthesis(atm, nu, llam, vec, wmu)
    assert np.array_equal(top, otop)
    np.testing.assert_allclose(flux, oflux, rtol=2e-6)
    chi, S = m3d.lte_transfer_units(atm, nu, llam, vec[0])
    ochi, oS = P.transfer_units(atm, nu, llam, vec[0])
    assert np.array_equal(chi, ochi) and np.array_equal(S, oS)


@pytest.mark.parametrize("nf,fp64", [(32, False), (45, False), (32, True), (20, True)])
def test_rays_together_equal_one_by_one(m3d, nf, fp64):
    """A ray's results do not depend on the rays that share its launch."""
    atm, nu, llam, _, _ = _case(nf, 1)
    vec, wmu = synth.lobatto_rays(4, 4)
    ie, flux, top = m3d.lte_synthesis(atm, nu, llam, vec, wmu, fp64=fp64, return_itop=True)
    for r in (0, 4, 12):
        ie1, _, top1 = m3d.lte_synthesis(atm, nu, llam, vec[r:r + 1], wmu[r:r + 1], fp64=fp64, return_itop=True)
        assert np.array_equal(top[r], top1[0]) and np.array_equal(ie[r], ie1[0])


@pytest.mark.parametrize("nf", [2, 3, 5, 8, 9, 16, 17, 31, 33, 64, 65, 100, 257])
def test_double_window_sizes(m3d, oracle, nf):
    """The plain FP64 pass at the edges of its register counts (4, 8, 16, 32 frequencies
    a lane, then several lanes a cell), to 1e-11: the device's double exp and log."""
    from oracle import pipeline as P
    atm, nu, llam, vec, _ = _case(nf, 3)
    for v in vec[:1] if nf > 64 else vec:
        chi, S = m3d.lte_transfer_units(atm, nu, llam, v, fp64=True)
        ochi, oS = P.transfer_units(atm, nu, llam, v, fp64=True)
        np.testing.assert_allclose(chi, ochi, rtol=1e-11, atol=0)
        np.testing.assert_allclose(S, oS, rtol=1e-11, atol=0)
