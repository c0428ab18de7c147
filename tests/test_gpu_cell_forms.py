"""Cell counts on both sides of the line that parts the one-cell and the grouped form of
the continuum, groups left short among them, and windows of many table rows: bit for bit
against the oracle."""
import numpy as np
import pytest

from dispatch_b200 import synth

pytestmark = pytest.mark.gpu

SMS = 148
CONT = SMS * 64                  # the continuum's line


def _exact_comps(comps):
    """The kinds without a platform exp or log, as in the continuum's own tests."""
    from dispatch_b200 import continuum as cn
    return [c for c in comps if c["kind"] not in (cn.H_FF, cn.REGULAR) and not (c["ilogl"] and not c["log_table"])
            and not (c["tt"].size == 1 and c["ilogl"])]


def _continuum(comps, lam, nu, cells, ncell):
    from dispatch_b200 import continuum as cn
    from oracle import continuum as oc
    cells = {k: v for k, v in cells.items() if k not in ("nHI", "partHI")}
    beta = np.random.default_rng(9).uniform(1e-6, 0.8, (ncell, lam.size)).astype(np.float32)
    xo, so = oc.continuum_opacities(comps, lam, nu, cells, beta=beta)
    xg, sg = cn.continuum_opacities(comps, lam, nu, cells, beta=beta)
    np.testing.assert_array_equal(xg, xo)
    np.testing.assert_array_equal(sg, so)


@pytest.mark.parametrize("ncell", [CONT - 1, CONT, CONT + 1, CONT + 2, CONT + 31])
def test_continuum_counts(m3d, oracle, ncell):
    comps, lam, nu, cells = synth.continuum_case(ncell=ncell, nlam=33)
    _continuum(_exact_comps(comps), lam, nu, cells, ncell)


def _refined(c, nnu):
    """The component's table on nnu wavelength nodes."""
    if c["tt"].size < 2:
        return c
    lam = np.geomspace(c["lam"][0], c["lam"][-1], nnu)
    xk = np.stack([np.interp(lam, c["lam"], r) for r in c["xkap"].reshape(c["tt"].size, -1)]).astype(np.float32)
    ld = np.zeros(nnu, bool)
    ld[nnu // 3] = True
    return dict(c, lam=lam, xkap=xk, ldisk=ld)


@pytest.mark.parametrize("ncell", [3, 33, CONT + 5])
@pytest.mark.parametrize("nnu,ncomp", [(50, 12), (120, 28), (150, 64), (400, 64), (1100, 20)])
def test_continuum_table_rows(m3d, oracle, ncell, nnu, ncomp):
    """Windows that read so many table rows, for so many components, that a block's shared
    memory decides the form, up to the most components a call takes, with all rows staged,
    some left in global memory, and none that fits."""
    comps, lam, nu, cells = synth.continuum_case(ncell=ncell, nlam=40)
    base = [_refined(c, nnu) for c in _exact_comps(comps)]
    comps = (base * (ncomp // len(base) + 1))[:ncomp]
    _continuum(comps, lam, nu, cells, ncell)
