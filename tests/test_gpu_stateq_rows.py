"""lineq_no_pivot with a thread per matrix row, at the edges of its forms (rows of 16,
24, 32, 48 and 64 registers, a warp or a block per cell): the update bit for bit against
the oracle, with the collision rates given and without collisions."""
import numpy as np
import pytest

from dispatch_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nlevel", [3, 8, 9, 16, 17, 24, 25, 32, 33, 40, 48, 49, 57, 63, 64])
@pytest.mark.parametrize("collisions", [True, False])
def test_rows_bitexact(oracle, m3d, nlevel, collisions):
    from oracle import stateq as sq
    from dispatch_b200 import stateq as se
    nb = nlevel - 1
    # without collisions every level needs a transition: the continua give each one
    atom, inp = synth.se_config("small", ncell=157, nbound=nb, nline=min(3 * nb, nb * (nb - 1) // 2))
    kw = {} if collisions else {"cswitch": 0.0, "max_update": 1e8}
    cup = sq.collision_rates(atom, inp["temp"], inp["ne"], inp["e_kT"])
    bo = inp["b"].copy()
    ro, lo, rc = sq.stateq_update(atom, bo, inp["nstar"], inp["totn"], inp["e_kT"], inp["gamma_ij"], inp["gamma_ji"],
                                  temp=inp["temp"], cup=cup, **kw)
    assert rc == 0 and ro["nclamp"] == 0
    bg = inp["b"].copy()
    rg, lg = se.stateq_update(atom, bg, inp["nstar"], inp["totn"], inp["e_kT"], inp["gamma_ij"], inp["gamma_ji"],
                              temp=inp["temp"], ne=inp["ne"], cup=cup, **kw)
    assert rg.pop("team") == (32 if nlevel <= 32 else 64)
    assert np.array_equal(bg, bo) and rg == ro and np.array_equal(lg, lo)


def test_singular_cell_reported(m3d):
    """A cell whose equations have no finite solution keeps its populations, and the
    call names it; the others are updated."""
    from dispatch_b200 import stateq as se
    atom, inp = synth.se_config("small", ncell=64, nbound=20, nline=60)
    gij, gji = inp["gamma_ij"].copy(), inp["gamma_ji"].copy()
    gij[:, 37] = np.nan
    b = inp["b"].copy()
    with pytest.raises(se.NonFiniteSolution) as e:
        se.stateq_update(atom, b, inp["nstar"], inp["totn"], inp["e_kT"], gij, gji, temp=inp["temp"], ne=inp["ne"])
    assert "cell 37" in str(e.value)
    assert np.array_equal(b[:, 37], inp["b"][:, 37]) and not np.array_equal(b[:, 36], inp["b"][:, 36])
