"""Kernels whose warps take several neighbouring cells: cell counts that leave a group
short, and neighbours that share nothing (the continuum's four cells a warp, the table
samplers' eight and four), bit for bit against the oracle."""
import numpy as np
import pytest

import optab_cases as ocases
from dispatch_b200 import synth

pytestmark = pytest.mark.gpu

COUNTS = [1, 2, 3, 4, 5, 7, 8, 9, 31, 33]


@pytest.mark.parametrize("ncell", COUNTS)
@pytest.mark.parametrize("nlam", [1, 31, 33, 64])
def test_continuum_groups(m3d, oracle, ncell, nlam):
    from dispatch_b200 import continuum as cn
    from oracle import continuum as oc
    comps, lam, nu, cells = synth.continuum_case(ncell=ncell, nlam=max(nlam, 2))
    lam, nu = lam[:nlam], nu[:nlam]
    # the kinds without a platform exp or log, as in the continuum's own tests
    comps = [c for c in comps if c["kind"] not in (cn.H_FF, cn.REGULAR) and not (c["ilogl"] and not c["log_table"])
             and not (c["tt"].size == 1 and c["ilogl"])]
    cells = {k: v for k, v in cells.items() if k not in ("nHI", "partHI")}
    beta = np.random.default_rng(9).uniform(1e-6, 0.8, (ncell, nlam)).astype(np.float32)
    xo, so = oc.continuum_opacities(comps, lam, nu, cells, beta=beta)
    xg, sg = cn.continuum_opacities(comps, lam, nu, cells, beta=beta)
    np.testing.assert_array_equal(xg, xo)
    np.testing.assert_array_equal(sg, so)


@pytest.mark.parametrize("ncell", COUNTS)
@pytest.mark.parametrize("nf", [1, 32, 70])
@pytest.mark.parametrize("shuffled", [False, True])
def test_table_groups(m3d, oracle, ncell, nf, shuffled):
    from dispatch_b200.optab import SampleOptab
    from oracle import optab
    c = ocases.cells()
    pick = np.random.default_rng(ncell).permutation(c["temp"].size)[:ncell] if shuffled else np.arange(ncell)
    c = {k: np.ascontiguousarray(v[pick]) for k, v in c.items() if np.ndim(v)}
    tab = ocases.table("background", nnu=120, cells_=ocases.cells())
    # half the queries on nodes, some beyond both ends
    q = np.sort(np.concatenate([tab["lam"][:nf // 2], np.linspace(3900.0, 9100.0, nf - nf // 2)]))
    T = SampleOptab.from_dict(tab)
    for g, o in zip(T.interpolate(c["temp"], c["ne"], c["chi500"], q),
                    optab.sample(tab, c["temp"], c["ne"], c["chi500"], q)):
        np.testing.assert_array_equal(g, o)
    vp = (c["vproj"] * 40.0).astype(np.float32)
    rng = np.random.default_rng(5)
    base = [rng.random((ncell, q.size)).astype(np.float32) for _ in range(3)]
    gpu, ref = [b.copy() for b in base], [b.copy() for b in base]
    T.interpolate_ll(c["temp"], c["ne"], c["chi500"], gpu[0], gpu[1], q, vp, chi_scat=gpu[2])
    optab.sample_ll(tab, c["temp"], c["ne"], c["chi500"], vp, q, ref[0], ref[1], ref[2])
    for g, o in zip(gpu, ref):
        np.testing.assert_array_equal(g, o)
    T.close()
