"""Calls where the device memory is nearly full.  The rays that share a launch, the lines'
constants of the NLTE opacity and a column plan's windows side by side take more memory
than a call needs: where it can't be had the call runs with less and gives the same
results, at every amount that is left.  Each runs in a thread, with a library context of
its own that holds nothing yet."""
import threading

import numpy as np
import pytest

from dispatch_b200 import synth

pytestmark = pytest.mark.gpu

MB = 1 << 20


def _in_thread(fn, *args):
    """fn's result from a thread with its own library context."""
    import dispatch_b200 as m
    out = {}

    def run():
        try:
            m.init(0)
            out["r"] = fn(*args)
        except BaseException as e:      # noqa: BLE001 -- raised again below
            out["e"] = e
        finally:
            m.synchronize()
            m.free()

    t = threading.Thread(target=run)
    t.start()
    t.join()
    if "e" in out:
        raise out["e"]
    return out["r"]


class _Full:
    """All of the device's free memory but `leave` bytes held."""

    def __init__(self, leave):
        import torch
        torch.cuda.synchronize()
        free, _ = torch.cuda.mem_get_info()
        self.block = torch.empty(max(free - leave, 0), dtype=torch.uint8, device="cuda")

    def __enter__(self):
        return self

    def __exit__(self, *exc):
        import torch
        del self.block
        torch.cuda.empty_cache()


def _device(atm):
    import torch
    up = lambda v: torch.as_tensor(np.ascontiguousarray(v), device="cuda") if isinstance(v, np.ndarray) else v
    out = {k: up(v) if k not in ("slab_nz", "species") else v for k, v in atm.items()}
    out["species"] = [{k: up(v) for k, v in sp.items()} for sp in atm["species"]]
    return out


def test_rays_one_by_one(m3d):
    """96 x 96 x 24 cells: five rays a launch hold 2 x 142 MB of transfer units, one 2 x 28."""
    import torch
    atm, nu, llam, vec, wmu = synth.lte_config(
        "mini", nf=32, cube=synth.cube_atmosphere(3, 96, 96, 24), lines=None)
    atm.update(nx=96, ny=96, nz=24, slab_nz=[12, 12], pivot_z=24 * atm["ds_code"][2])
    a, dn, dl = _device(atm), *(torch.as_tensor(x, device="cuda") for x in (nu, llam))
    run = lambda: [t.cpu() for t in m3d.lte_synthesis(a, dn, dl, vec, wmu, return_itop=True, device=True)]
    want = _in_thread(run)
    for leave in range(100, 360, 20):
        with _Full(leave * MB):
            got = _in_thread(run)
        for g, w in zip(got, want):
            assert torch.equal(g, w), leave


def test_gradient_rays_one_by_one(m3d):
    """32^3 cells: thirteen rays a group hold 430 MB of work arrays, one 33."""
    import torch
    atm, nu, llam, vec, wmu, _ = synth.lte_config_c4(size=(32, 32, 32), nline_per_species=10, window=100)
    a, dn, dl = _device(atm), *(torch.as_tensor(x, device="cuda") for x in (nu, llam))
    g = torch.linspace(0.5, 1.5, 32, device="cuda")
    run = lambda: {k: v.cpu() for k, v in
                   m3d.lte_synthesis_adjoint(a, dn, dl, vec, wmu, g, device=True).items()}
    want = _in_thread(run)
    for leave in (90, 120, 180, 240, 300, 360, 420):
        with _Full(leave * MB):
            got = _in_thread(run)
        for k in ("temp", "chi_c", "e_kT", "inv_df", "lnbase"):     # the rays' sums in their order
            assert torch.equal(got[k], want[k]), (leave, k)
        # the lines' sums over the cells in any order
        np.testing.assert_allclose(got["gpref"], want["gpref"], rtol=1e-4, atol=1e-6 * float(want["gpref"].abs().max()))


def test_line_constants_at_every_point(m3d):
    """106000 cells x 20 lines: 64 MB of the lines' constants where there is room for them,
    formed at every point where there is not."""
    import torch
    from dispatch_b200 import nlte
    nc = 106000
    atom, inp = synth.se_config("small", ncell=nc)
    win = synth.atom_window(atom, nper=5, transitions=list(range(20)))
    rng = np.random.default_rng(3)
    s = {"b": inp["b"], "nstar": inp["nstar"], "pop_ratio": np.ones(nc), "e_kT": inp["e_kT"],
         "inv_df": (1.8e5 * (1 + 0.1 * rng.standard_normal(nc))).astype(np.float32),
         "vproj": (1e-5 * rng.standard_normal(nc)).astype(np.float32),
         "adamp": rng.uniform(1e-3, 0.1, (win["nline"], nc)).astype(np.float32)}
    up = [torch.as_tensor(np.ascontiguousarray(v), device="cuda") for v in s.values()]
    base = [torch.full((nc, win["nf"]), 1e-9, device="cuda") for _ in range(2)]

    def run(x, e):
        nlte.bb_opacity(win, *up, x, e)
        m3d.synchronize()

    want, got = [b.clone() for b in base], [b.clone() for b in base]
    _in_thread(run, *want)
    with _Full(40 * MB):
        _in_thread(run, *got)
    for g, w, b in zip(got, want, base):
        assert torch.equal(g, w) and not torch.equal(g, b)
