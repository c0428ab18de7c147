"""An adjoint that is not finite at one frequency of the window: a line whose own part of
the window leaves that frequency out, in every cell and for every ray, keeps the gradient
it has without it."""
import numpy as np
import pytest

from dispatch_b200 import synth

pytestmark = pytest.mark.gpu

NLINE = 8


@pytest.fixture(scope="module")
def case(m3d):
    """Eight lines on a coarse window, so that each covers a part of it, and by line the
    frequencies whose opacity it changes in any cell for any ray."""
    atm, _, _, vec, wmu, raw = synth.lte_config_c4(size=(8, 6, 32), nline_per_species=20, window=100)
    llam, nu = synth.frequency_grid(6000.0, 6050.0, 32)
    sp = dict(atm["species"][0])
    # eight lines spread over the window, weak enough to reach a few points of it
    for k in ("llam0", "lower_ev", "gpref", "grad", "gw1", "gw2", "gstk", "unsold"):
        sp[k] = np.ascontiguousarray(np.asarray(sp[k])[:NLINE])
    sp["llam0"] = np.ascontiguousarray(llam[2:30:4][:NLINE - 1].tolist() + [llam[30]], np.float64)
    sp["gpref"] = (sp["gpref"] - 4.0).astype(np.float32)
    for k in ("active", "reach_in"):
        sp.pop(k, None)

    def atm_of(lines):
        s = {k: (v[lines] if k in ("llam0", "lower_ev", "gpref", "grad", "gw1", "gw2", "gstk", "unsold") else v)
             for k, v in sp.items()}
        return dict(atm, species=[{k: np.ascontiguousarray(v) for k, v in s.items()}])

    cover = np.zeros((NLINE, 32), bool)
    for v in vec:
        none = m3d.lte_transfer_units(dict(atm, species=[]), nu, llam, v)[0]
        for j in range(NLINE):
            chi = m3d.lte_transfer_units(atm_of([j]), nu, llam, v)[0]
            cover[j] |= (chi != none).any(axis=0)
    return atm_of(list(range(NLINE))), nu, llam, vec, wmu, cover


@pytest.mark.parametrize("bad", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("f0", [0, 13, 17, 31])
def test_lines_that_leave_a_frequency_out(m3d, case, f0, bad):
    atm, nu, llam, vec, wmu, cover = case
    near = cover.copy()             # a point more on either side: a window's edge adds little
    near[:, 1:] |= cover[:, :-1]
    near[:, :-1] |= cover[:, 1:]
    apart = ~near[:, f0] & cover.any(axis=1)
    assert apart.any() and not apart.all()
    g = np.linspace(0.5, 1.5, 32).astype(np.float32)
    g[f0] = 0.0
    want = m3d.lte_synthesis_adjoint(atm, nu, llam, vec, wmu, g)["gpref"]
    g[f0] = bad
    got = m3d.lte_synthesis_adjoint(atm, nu, llam, vec, wmu, g)["gpref"]
    assert np.all(want[apart] != 0.0)
    # the order of the cells' sums is free: float32 sums of 1536 cells and 13 rays
    np.testing.assert_allclose(got[apart], want[apart], rtol=1e-3, atol=1e-6 * np.abs(want).max())
