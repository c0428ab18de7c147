"""A column plan whose windows outnumber the slots they are swept in: a window reuses the
arrays of an earlier one, in streams of its own, and the captured sweep still gives the
direct launches' bits, replay after replay.  And what a plan takes of the memory that is
free."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SMS = 148


def _slots(ncol, nwin):
    """Windows side by side: four rounds of four blocks an SM."""
    return min(nwin, -(-16 * SMS // (2 * ncol)))


def _departures(A):
    import torch
    gen = torch.Generator(device="cuda").manual_seed(5)
    A.b.copy_(torch.exp(0.1 * torch.randn(A.b.shape, generator=gen, device="cuda", dtype=torch.float64)))
    A.iter = 1
    return A


def _sweep(A):
    A.gamma_ij.zero_()
    A.gamma_ji.zero_()
    A.sweep()
    J, P = A.fields()
    return [t.cpu().numpy() for t in (A.gamma_ij, A.gamma_ji, J, P)]


@pytest.mark.parametrize("ncol,nwin,slots", [(600, 5, 2), (600, 4, 2), (400, 8, 3), (200, 7, 6), (1200, 3, 1)])
def test_slots_reused(m3d, ncol, nwin, slots):
    from dispatch_b200 import ali
    assert _slots(ncol, nwin) == slots < nwin
    cols, atom, wins, mu, wmu = ali.column_problem(ncol=ncol, depth=(4, 10), nwin=nwin, nbound=8, nline=16, nper=9)
    direct = _departures(ali.AliColumns(cols, atom, wins, mu, wmu, use_graph=False))
    want = _sweep(direct)
    graph = _departures(ali.AliColumns(cols, atom, wins, mu, wmu, use_graph=True))
    assert graph.shape["fused_windows"] == nwin
    assert np.abs(want[0]).max() > 0
    for _ in range(4):
        for g, w in zip(_sweep(graph), want):
            np.testing.assert_array_equal(g, w)
    direct.close()
    graph.close()


def test_plan_leaves_memory(m3d):
    """Eight windows of 18 MB a slot with 240 MB free: the plan takes a quarter of them at
    the most beyond its first slot, where eight slots would take 144 MB, and the sweep is
    the one of a plan with all its slots."""
    import torch
    from dispatch_b200 import ali
    cols, atom, wins, mu, wmu = ali.column_problem(ncol=40, depth=(50, 60), nz=64, nbound=20, nline=60, nwin=8)
    A = _departures(ali.AliColumns(cols, atom, wins, mu, wmu))
    want = _sweep(A)
    A.close()
    del A
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    block = torch.empty(free - (240 << 20), dtype=torch.uint8, device="cuda")
    try:
        before, _ = torch.cuda.mem_get_info()
        A = _departures(ali.AliColumns(cols, atom, wins, mu, wmu))
        after, _ = torch.cuda.mem_get_info()
        assert before - after <= 110 << 20
        for _ in range(2):
            for g, w in zip(_sweep(A), want):
                np.testing.assert_array_equal(g, w)
        A.close()
    finally:
        del block
        torch.cuda.empty_cache()
