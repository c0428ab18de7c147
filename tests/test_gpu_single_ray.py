"""One ray of a small atmosphere, which the warp-per-cell kernel takes up to one round of
its warps (16 an SM) and 128 frequencies: on both sides of the two lines, the ray bit for
bit what it is among others (the lane kernel), and the oracle's."""
import numpy as np
import pytest

from dispatch_b200 import synth

pytestmark = pytest.mark.gpu

CELLS = 16 * 148


def _case(shape, nf, lines=40):
    nx, ny, nz = shape
    cube = synth.cube_atmosphere(7, nx, ny, nz)
    rng = np.random.default_rng(11)
    atm, _, _, vec, wmu = synth.lte_config("mini", nf=16)
    llam, nu = synth.frequency_grid(5000.5, 5000.5 + 0.01 * nf, nf)
    temp, nH, ne = cube["temp"], cube["nH"], cube["ne"]
    sp = synth.species_arrays(synth.random_linelist(rng, lines, 5000.0, 5002.5), temp, 10.0 ** (7.5 - 12.0) * nH)
    code = tuple(d / 1e8 for d in cube["ds_cm"])
    flat = lambda a: np.ascontiguousarray(a, np.float32).ravel()
    atm = {"nx": nx, "ny": ny, "nz": nz, "slab_nz": [nz], "ds_cm": cube["ds_cm"], "ds_code": code,
           "pivot_z": nz * code[2], "ray_offset": (0.0, 0.0), "temp": flat(temp), "chi_c": flat(cube["chi_c"]),
           "vx": np.zeros(temp.size, np.float32), "vy": np.zeros(temp.size, np.float32), "vz": flat(cube["vz"]),
           "species": [{k: (np.ascontiguousarray(v).ravel() if k in ("inv_df", "vbar2", "lnbase") else v)
                        for k, v in sp.items()}]}
    atm.update({k: flat(v) for k, v in synth.cell_fields(temp, nH, ne).items()})
    return atm, nu, llam, vec, wmu


@pytest.mark.parametrize("shape", [(1, 1, 2), (1, 1, 80), (8, 8, 37), (1, 23, 103)])
@pytest.mark.parametrize("nf", [8, 31, 32, 64, 65, 128, 129])
def test_one_ray(m3d, oracle, shape, nf):
    from oracle import pipeline as P
    assert (8 * 8 * 37, 23 * 103) == (CELLS, CELLS + 1)
    atm, nu, llam, vec, wmu = _case(shape, nf)
    pick = [5, 0]
    one = m3d.lte_synthesis(atm, nu, llam, vec[pick[:1]], wmu[pick[:1]], return_itop=True)
    two = m3d.lte_synthesis(atm, nu, llam, vec[pick], wmu[pick], return_itop=True)
    # (two planes' depths leave the synthetic fields undefined: the same NaN everywhere)
    np.testing.assert_array_equal(one[2][0], two[2][0])
    np.testing.assert_array_equal(one[0][0], two[0][0])
    _, _, otop = P.lte_synthesis(atm, nu, llam, vec[pick[:1]], wmu[pick[:1]])
    np.testing.assert_array_equal(one[2], otop)
    chi, S = m3d.lte_transfer_units(atm, nu, llam, vec[5])
    ochi, oS = P.transfer_units(atm, nu, llam, vec[5])
    np.testing.assert_array_equal(chi, ochi)
    np.testing.assert_array_equal(S, oS)
