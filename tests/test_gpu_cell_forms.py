"""Cell counts on both sides of the lines that part the one-cell and the grouped forms of
the continuum and of the table samplers, groups left short among them: bit for bit
against the oracle.  Below the lines the grouped forms, which the small counts of other
tests no longer reach, are not taken."""
import numpy as np
import pytest

import optab_cases as ocases
from dispatch_b200 import synth

pytestmark = pytest.mark.gpu

SMS = 148
CONT = SMS * 32 + 1              # the continuum's line
BG, ROUND = SMS * 8 * 8, SMS * 2 * 8 * 4      # the samplers': a block of groups an SM, a round


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


@pytest.mark.parametrize("ncell", [ROUND * 19 // 20, ROUND * 19 // 20 + 1, BG - 1, BG, BG + 1, BG + 7,
                                   2 * ROUND * 19 // 20, 2 * ROUND * 19 // 20 + 1, 2 * ROUND + 1,
                                   5 * ROUND, 5 * ROUND + 1, 5 * ROUND + 3])
def test_table_counts(m3d, oracle, ncell):
    from dispatch_b200.optab import SampleOptab
    from oracle import optab
    c = ocases.cells(seed=3, nx=40, ny=40, nz=36)
    tab = ocases.table("linelist", nnu=120, cells_=c)
    c = {k: np.ascontiguousarray(v[:ncell]) for k, v in c.items()}
    assert c["temp"].size == ncell
    q = np.sort(np.concatenate([tab["lam"][20:60:10], np.linspace(3900.0, 9100.0, 29)]))
    T = SampleOptab.from_dict(tab)
    for g, o in zip(T.interpolate(c["temp"], c["ne"], c["chi500"], q),
                    optab.sample(tab, c["temp"], c["ne"], c["chi500"], q)):
        np.testing.assert_array_equal(g, o)
    vp = (c["vproj"] * 40.0).astype(np.float32)
    vp[::97] = np.float32(-np.inf)
    rng = np.random.default_rng(5)
    base = [rng.random((ncell, q.size)).astype(np.float32) for _ in range(3)]
    gpu, ref = [b.copy() for b in base], [b.copy() for b in base]
    T.interpolate_ll(c["temp"], c["ne"], c["chi500"], gpu[0], gpu[1], q, vp, chi_scat=gpu[2])
    optab.sample_ll(tab, c["temp"], c["ne"], c["chi500"], vp, q, ref[0], ref[1], ref[2])
    for g, o in zip(gpu, ref):
        np.testing.assert_array_equal(g, o)
    T.close()
