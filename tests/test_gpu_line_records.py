"""The lane kernels' packed line records, every law and mark they carry, and the launch
form of few units, bit for bit against the oracle and against launches of more units."""
import numpy as np
import pytest

from dispatch_b200 import synth

pytestmark = pytest.mark.gpu


def _laws(atm, which):
    rng = np.random.default_rng(5)
    out = dict(atm, species=[])
    for k, sp0 in enumerate(atm["species"]):
        sp = dict(sp0)
        n = sp["llam0"].size
        if which == "inactive" or (which == "mixed" and k == 0):
            sp["active"] = (rng.random(n) < 0.6).astype(np.uint8)
            sp["gpref"] = np.where(sp["active"] == 1, sp["gpref"], np.float32(np.nan)).astype(np.float32)
        if which in ("laws", "mixed"):
            sp["unsold"] = (rng.random(n) < 0.4).astype(np.uint8)
            sp["gw1"] = np.where(rng.random(n) < 0.7, 1e-20 * rng.random(n), 0.0).astype(np.float32)
            sp["gw2"] = np.where(sp["unsold"] == 1, np.float32(np.nan), 0.3 * rng.random(n)).astype(np.float32)
            sp["gstk"] = (np.abs(sp["gstk"]) * rng.choice([-1.0, 1.0], n)).astype(np.float32)
        out["species"].append(sp)
    if which == "none":
        out["species"] = [dict(sp, active=np.zeros(sp["llam0"].size, np.uint8)) for sp in out["species"]]
    return out


@pytest.mark.parametrize("which", ["laws", "inactive", "mixed", "none"])
@pytest.mark.parametrize("nf", [20, 32, 70])
def test_laws_and_marks(m3d, oracle, which, nf):
    from oracle import pipeline as P
    atm, _, _, vec, _ = synth.lte_config("mini", nf=16)
    llam, nu = synth.frequency_grid(5000.5, 5000.5 + 0.01 * nf, nf)
    atm = _laws(atm, which)
    chi, S = m3d.lte_transfer_units(atm, nu, llam, vec[5])
    ochi, oS = P.transfer_units(atm, nu, llam, vec[5])
    assert np.array_equal(chi, ochi) and np.array_equal(S, oS)


def test_few_units_equal_many(m3d):
    """24^3 cells: two rays are 864 units of 32 cells, six are 2592, to either side of
    the 2368 that one round of 16 warps an SM holds."""
    atm, nu, llam, _, _ = synth.lte_config("mini", nf=32, size=24)
    vec, wmu = synth.lobatto_rays(4, 4)
    _, _, many = m3d.lte_synthesis(atm, nu, llam, vec[:6], wmu[:6], return_itop=True)
    _, _, few = m3d.lte_synthesis(atm, nu, llam, vec[:2], wmu[:2], return_itop=True)
    assert np.array_equal(many[:2], few)


@pytest.mark.parametrize("nwin", [8, 300])
def test_few_window_units(m3d, nwin):
    """A column's windows, 3 units each, to either side of the 16-warp form, against
    one synthesis per window."""
    atm, _, _, vec, wmu = synth.lte_config("c0", nf=32)
    llam, nu = synth.frequency_grid(5000.5, 5000.5 + 0.005 * 32 * nwin, 32 * nwin)
    llam, nu = np.ascontiguousarray(llam).reshape(nwin, 32), np.ascontiguousarray(nu).reshape(nwin, 32)
    _, _, top = m3d.lte_synthesis_windows(atm, nu, llam, vec, wmu, return_itop=True)
    for w in (0, nwin // 2, nwin - 1):
        _, _, one = m3d.lte_synthesis(atm, nu[w], llam[w], vec, wmu, return_itop=True)
        assert np.array_equal(np.asarray(top).reshape(len(wmu), -1)[:, 32 * w:32 * w + 32],
                              np.asarray(one).reshape(len(wmu), -1))
