"""sample_interpolate_ll where a cell's Doppler factor is infinite, undefined, zero or
far beyond the table: the bracket's walk ends on the table for every value, and each
cell gets what it gets on its own, bit for bit the oracle's, whichever of its
neighbours it shares a warp with."""
import numpy as np
import pytest

import optab_cases as oc

pytestmark = pytest.mark.gpu


def _shifts(n, seed):
    """Ordinary shifts with an extreme one in every second to fifth cell."""
    rng = np.random.default_rng(seed)
    vp = rng.normal(0.0, 1e-4, n).astype(np.float32)
    ext = np.array([-np.inf, np.inf, np.nan, -1.0, -2.0, 3.0, 1e30, -1e30], np.float32)
    k = np.cumsum(rng.integers(2, 6, n))
    k = k[k < n]
    vp[k] = ext[np.arange(k.size) % ext.size]
    return vp


@pytest.mark.parametrize("with_scat", [True, False])
@pytest.mark.parametrize("nnu", [2, 3, 500])
@pytest.mark.parametrize("ncell", [1, 3, 5, 161])
def test_sample_ll_extreme_shifts(m3d, oracle, nnu, ncell, with_scat):
    from dispatch_b200.optab import SampleOptab
    from oracle import optab
    c = oc.cells()
    tab = oc.table("linelist", nnu=nnu, cells_=c)
    q = np.linspace(4050.0, 8950.0, 45)
    T = SampleOptab.from_dict(tab)
    for seed in range(8 if ncell < 8 else 1):
        f = {k: np.ascontiguousarray(c[k].ravel()[:ncell]) for k in ("temp", "ne", "chi500")}
        vp = _shifts(ncell, seed)
        if ncell < 8:       # the extreme value in each place of the warp's cells
            vp[seed % ncell] = [-np.inf, np.inf, np.nan, -1.0, -np.inf, 1e30, -1e30, -2.0][seed]
        base = [np.random.default_rng(7 + k).random((ncell, q.size)).astype(np.float32) for k in range(3)]
        out = {}
        for name in ("g", "o"):
            x, e, s = (b.copy() for b in base)
            cs = s if with_scat else None
            if name == "g":
                T.interpolate_ll(f["temp"], f["ne"], f["chi500"], x, e, q, vp, cs)
            else:
                optab.sample_ll(tab, f["temp"], f["ne"], f["chi500"], vp, q, x, e, cs)
            out[name] = (x, e, s)
        for a, b in zip(out["g"], out["o"]):
            np.testing.assert_array_equal(a, b)
        ok = np.isfinite(vp) & (np.abs(vp) < 1e-2)
        assert np.isfinite(out["g"][0][ok]).all()
    T.close()
