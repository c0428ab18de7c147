"""The LTE pass where a cell's velocity, or a line's place, is infinite, undefined or far
beyond the grid: the line then lies outside every window by more steps than an int
counts.  Every form of the line-opacity kernels returns, and the cells (the lines) that
are sound get what they get without the others."""
import numpy as np
import pytest

from dispatch_b200 import synth

pytestmark = pytest.mark.gpu

BAD = [np.inf, -np.inf, np.nan, 3e38, -3e38, 1e30]


def _case(nf, shape=(16, 12, 13), nline=40):
    """2496 cells: more than the warp-per-cell kernel takes of one ray."""
    nx, ny, nz = shape
    cube = synth.cube_atmosphere(5, nx, ny, nz)
    temp, nH, ne = cube["temp"], cube["nH"], cube["ne"]
    lines = synth.random_linelist(np.random.default_rng(4), nline, 5000.0, 5002.0)
    sp = synth.species_arrays(lines, temp, 10.0 ** (7.5 - 12.0) * nH)
    llam, nu = synth.frequency_grid(5000.5, 5000.5 + 0.01 * nf, nf)
    code = tuple(d / 1e8 for d in cube["ds_cm"])
    flat = lambda a: np.ascontiguousarray(a, np.float32).ravel()
    atm = {"nx": nx, "ny": ny, "nz": nz, "slab_nz": [nz], "ds_cm": cube["ds_cm"], "ds_code": code,
           "pivot_z": nz * code[2], "ray_offset": (0.0, 0.0), "temp": flat(temp), "chi_c": flat(cube["chi_c"]),
           "vx": np.zeros(temp.size, np.float32), "vy": np.zeros(temp.size, np.float32), "vz": flat(cube["vz"]),
           "species": [{k: (np.ascontiguousarray(v).ravel() if k in ("inv_df", "vbar2", "lnbase") else np.asarray(v))
                        for k, v in sp.items()}]}
    atm.update({k: flat(v) for k, v in synth.cell_fields(temp, nH, ne).items()})
    return atm, nu, llam


V = np.array([0.3, -0.4, np.sqrt(0.75)])


@pytest.mark.parametrize("nf,fp64", [(nf, False) for nf in (7, 8, 16, 20, 32, 33, 45, 64, 65, 100, 300, 1000)]
                         + [(nf, True) for nf in (4, 8, 20, 32, 45, 200)])
def test_velocities(m3d, nf, fp64):
    atm, nu, llam = _case(nf)
    chi0, S0 = m3d.lte_transfer_units(atm, nu, llam, V, fp64=fp64)
    vz = atm["vz"].copy()
    at = np.arange(5, vz.size, 11)
    vz[at] = np.array(BAD, np.float32)[np.arange(at.size) % len(BAD)]
    chi, S = m3d.lte_transfer_units(dict(atm, vz=vz), nu, llam, V, fp64=fp64)
    sound = np.ones(vz.size, bool)
    sound[at] = False
    assert np.isfinite(chi0).all() and np.array_equal(chi[sound], chi0[sound]) and np.array_equal(S[sound], S0[sound])
    # infinitely far from every line: the continuum alone
    none, _ = m3d.lte_transfer_units(dict(atm, species=[]), nu, llam, V, fp64=fp64)
    far = at[np.isinf(vz[at])]
    np.testing.assert_allclose(chi[far], none[far], rtol=1e-6)


@pytest.mark.parametrize("nf,fp64", [(20, False), (32, False), (45, False), (100, False), (45, True)])
def test_line_places(m3d, nf, fp64):
    atm, nu, llam = _case(nf)
    sp = atm["species"][0]
    keep = np.arange(sp["llam0"].size) % 4 != 1
    per_line = ("llam0", "lower_ev", "gpref", "grad", "gw1", "gw2", "gstk", "unsold")
    some = {k: (np.ascontiguousarray(v[keep]) if k in per_line else v) for k, v in sp.items()}
    want = m3d.lte_transfer_units(dict(atm, species=[some]), nu, llam, V, fp64=fp64)
    ll = sp["llam0"].copy()
    ll[~keep] = np.array([np.inf, -np.inf, 1e300, -1e300])[np.arange((~keep).sum()) % 4]
    got = m3d.lte_transfer_units(dict(atm, species=[dict(sp, llam0=ll)]), nu, llam, V, fp64=fp64)
    np.testing.assert_allclose(got[0], want[0], rtol=1e-6)
    np.testing.assert_allclose(got[1], want[1], rtol=1e-6)


def test_windows_and_gradient(m3d):
    atm, nu, llam = _case(96, (1, 1, 40))
    vec, wmu = synth.gauss_rays(3)
    atm["vz"][[3, 17]] = np.inf, -np.inf
    m3d.lte_synthesis_windows(atm, nu.reshape(3, 32), llam.reshape(3, 32), vec, wmu)
    atm, nu, llam = _case(32)
    vec, wmu = synth.lobatto_rays(2, 4)
    atm["vz"][[30, 700, 1500]] = np.inf, -np.inf, 3e38
    g = m3d.lte_synthesis_adjoint(atm, nu, llam, vec, wmu, np.ones(32, np.float32))
    assert set(g) == {"temp", "chi_c", "e_kT", "inv_df", "lnbase", "gpref"}
