"""Cell counts on both sides of the lines that part the forms of the model atom's kernels:
the continuum rates with eight cells or one a warp (a block of tiles an SM, two for long
continua), the line opacities with the lines' constants formed ahead or at every point (2
Mi points), the line rates by their lines' points; bit for bit against the oracle."""
import numpy as np
import pytest

from dispatch_b200 import synth

pytestmark = pytest.mark.gpu


def _cells(ncell, transitions, nper, seed=11):
    atom, inp = synth.se_config("small", ncell=ncell)
    win = synth.atom_window(atom, nper=nper, transitions=[k if k >= 0 else atom["nline"] - k - 1 for k in transitions])
    rng = np.random.default_rng(seed)
    c = {"b": inp["b"], "nstar": inp["nstar"], "pop_ratio": np.ones(ncell), "e_kT": inp["e_kT"],
         "inv_df": (1.8e5 * (1 + 0.1 * rng.standard_normal(ncell))).astype(np.float32),
         "vproj": (1e-5 * rng.standard_normal(ncell)).astype(np.float32),
         "adamp": rng.uniform(1e-3, 0.1, (max(win["nline"], 1), ncell)).astype(np.float32)}
    return win, c, rng


@pytest.mark.parametrize("ncell,ncont,nper", [(1, 1, 37), (9, 3, 37), (9464, 1, 37), (9465, 1, 37), (9471, 1, 37),
                                              (472, 20, 5), (473, 20, 5), (592, 16, 5), (1185, 8, 5),
                                              (944, 20, 30), (945, 20, 30), (1184, 16, 30)])
@pytest.mark.parametrize("precond", [True, False])
@pytest.mark.parametrize("cut_x", [70.0, 15.0])
def test_bf_rates_tiles(m3d, oracle, ncell, ncont, nper, precond, cut_x):
    from dispatch_b200 import nlte as gn
    from oracle import nlte as nl
    win, c, rng = _cells(ncell, [-1 - k for k in range(ncont)], nper)
    win["cut_x"] = cut_x            # 15: some cells leave the transition out
    assert win["ncont"] == ncont and win["nline"] == 0
    J, P = (rng.random((ncell, win["nf"])).astype(np.float32) for _ in range(2))
    beta = rng.uniform(1e-3, 0.6, (ncell, win["nf"])).astype(np.float32)
    res = []
    for mod in (nl, gn):
        g = [np.full((ncont, ncell), 0.25, np.float32) for _ in range(2)]
        mod.bf_rates(win, c["b"], c["nstar"], c["e_kT"], J, P, beta, *g, preconditioning=precond)
        res.append(g)
    for o, g in zip(*res):
        np.testing.assert_array_equal(g, o)


@pytest.mark.parametrize("ncell", [3, 10485, 10486])
@pytest.mark.parametrize("lte", [False, True])
def test_bb_opacity_points(m3d, oracle, ncell, lte):
    from dispatch_b200 import nlte as gn
    from oracle import nlte as nl
    win, c, rng = _cells(ncell, range(0, 40, 5), 25)
    assert win["nf"] == 200
    x, e = (1e-8 * (1 + rng.random((ncell, 200), np.float32)) for _ in range(2))
    res = []
    for mod in (nl, gn):
        xh, eh, sp = x.copy(), e.copy(), gn.new_split(ncell, 200)
        mod.bb_opacity(win, c["b"], c["nstar"], c["pop_ratio"], c["e_kT"], c["inv_df"], c["vproj"], c["adamp"], xh,
                       eh, lte=lte, split=sp)
        res.append((xh, eh, *sp.values()))
    for o, g in zip(*res):
        np.testing.assert_array_equal(g, o)
    assert not np.array_equal(res[0][0], x)


@pytest.mark.parametrize("nper", [25, 32, 33, 70])
@pytest.mark.parametrize("split_rates", [True, False])
@pytest.mark.parametrize("precond", [True, False])
def test_bb_rates_line_points(m3d, oracle, nper, split_rates, precond):
    """The line rates with ten and with eight blocks an SM: lines of up to and beyond one
    round of the lanes."""
    from dispatch_b200 import nlte as gn
    from oracle import nlte as nl
    n = 61
    win, c, rng = _cells(n, range(0, 40, 5), nper)
    nf = win["nf"]
    f32 = lambda lo, hi: rng.uniform(lo, hi, (n, nf)).astype(np.float32)
    beta = f32(1e-3, 0.6)
    ids = lambda: rng.integers(0, 12, (n, nf)).astype(np.int32)
    split = {"opac_L": f32(0, 1), "opac_R": f32(0, 1), "id": ids(), "chi_L": f32(0, 1), "chi_R": f32(0, 1),
             "chi_id": ids()}
    kw = dict(work1=f32(0.1, 1), psi=f32(0, 1), irem=f32(0, 1), escape=f32(0, 1), split=split,
              split_rates=split_rates, preconditioning=precond, wmu=0.3)
    kw["psi"][rng.random((n, nf)) < 0.05] = 0.0
    inu, Bnu = f32(0, 1), beta / (1 - beta)
    res = []
    for mod in (nl, gn):
        g = [np.full((win["nline"], n), 0.25, np.float32) for _ in range(2)]
        mod.bb_rates(win, c["b"], c["nstar"], c["pop_ratio"], c["e_kT"], c["inv_df"], c["vproj"], c["adamp"], inu,
                     beta, Bnu, *g, **kw)
        res.append(g)
    for o, g in zip(*res):
        np.testing.assert_array_equal(g, o)
    assert np.abs(res[0][0]).max() > 0.25
