"""The register rows of lineq_no_pivot with the collision rates formed in the kernel, at
the level counts where a form ends and the next begins.  An even count pads the matrix's
columns, which the sorted electron pairs and the records' element list then have to
follow: the bits of one warp per cell (whose columns are not padded), and those of the
update that reads m3d_collision_rates' rates."""
import numpy as np
import pytest

from dispatch_b200 import synth

pytestmark = pytest.mark.gpu

H_RECIPES = ("drawin", "drawin", "takeda")


@pytest.mark.parametrize("nlevel", [16, 17, 24, 25, 32, 33, 48, 49, 64])
@pytest.mark.parametrize("form", ["fused", "hydrogen", "gencol"])
def test_rates_in_kernel(m3d, nlevel, form):
    from dispatch_b200 import stateq as se
    nb = nlevel - 1
    kw = {"fused": {}, "hydrogen": {"h_recipes": H_RECIPES}, "gencol": {"h_recipes": H_RECIPES, "gencol": True}}[form]
    atom, inp = synth.se_config("small", ncell=333, nbound=nb, nline=min(3 * nb, nb * (nb - 1) // 2), **kw)
    cells = {} if form == "fused" else {k: inp[k] for k in ("nh1", "lsaha", "colliders")}
    cup = se.collision_rates(atom, inp["temp"], inp["ne"], inp["e_kT"], nstar=inp["nstar"], **cells)
    out = []
    for warp, rates in ((False, None), (True, None), (False, cup), (True, cup)):
        b = inp["b"].copy()
        res, lvl = se.stateq_update(atom, b, inp["nstar"], inp["totn"], inp["e_kT"], inp["gamma_ij"], inp["gamma_ji"],
                                    temp=inp["temp"], ne=inp["ne"], cup=rates, warp_per_cell=warp, **cells)
        assert res.pop("team") == (32 if warp or nlevel <= 32 else 64)
        out.append((b, res, lvl))
    for b, res, lvl in out[1:]:
        assert np.array_equal(b, out[0][0]) and res == out[0][1] and np.array_equal(lvl, out[0][2])
    assert out[0][1]["maxerr"] != 0
