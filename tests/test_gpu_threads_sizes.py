"""Calls of different sizes from two threads: a kernel's shared-memory limit belongs to the
kernel, so a small call of one thread must not lower it for a large one of the other.
By turns for the kernels whose threads used to remember the limit they had set, and side by
side for all of them; each call gives what it gives alone."""
import queue
import threading

import numpy as np
import pytest

from dispatch_b200 import synth

pytestmark = pytest.mark.gpu


class _Worker:
    """A thread with a library context of its own that runs what it is handed."""

    def __init__(self):
        self.todo, self.done = queue.Queue(), queue.Queue()
        self.t = threading.Thread(target=self._run, daemon=True)
        self.t.start()

    def _run(self):
        import dispatch_b200 as m
        m.init(0)
        while True:
            f = self.todo.get()
            if f is None:
                break
            try:
                self.done.put((f(), None))
            except BaseException as e:      # noqa: BLE001 -- raised again by result()
                self.done.put((None, e))
        m.free()

    def start(self, f):
        self.todo.put(f)

    def result(self):
        r, e = self.done.get(timeout=120)
        if e is not None:
            raise e
        return r

    def close(self):
        self.todo.put(None)
        self.t.join()


@pytest.fixture
def workers(m3d):
    w = (_Worker(), _Worker())
    yield w
    for k in w:
        k.close()


def _ray(m, nf):
    atm, _, _, vec, wmu = synth.lte_config("mini", nf=16)
    llam, nu = synth.frequency_grid(5000.5, 5000.5 + 0.01 * nf, nf)
    return lambda: m.lte_synthesis(atm, nu, llam, vec[:1], wmu[:1], return_itop=True)[2]


def _gradient(m, nline):
    atm, nu, llam, vec, wmu, _ = synth.lte_config_c4(size=(4, 4, 16), nline_per_species=nline, window=100)
    g = np.ones(32, np.float32)
    return lambda: m.lte_synthesis_adjoint(atm, nu, llam, vec[:3], wmu[:3], g)["inv_df"]


def _update(m, nb, solver, warp=False):
    from dispatch_b200 import stateq as se
    atom, inp = synth.se_config("small", ncell=40, nbound=nb, nline=2 * nb)

    def run():
        b = inp["b"].copy()
        se.stateq_update(atom, b, inp["nstar"], inp["totn"], inp["e_kT"], inp["gamma_ij"], inp["gamma_ji"],
                         temp=inp["temp"], ne=inp["ne"], solver=solver, warp_per_cell=warp)
        return b
    return run


def _continuum(m, rep):
    from dispatch_b200 import continuum as cn
    comps, lam, nu, cells = synth.continuum_case(ncell=40, nlam=64)
    comps = comps * rep
    return lambda: cn.continuum_opacities(comps, lam, nu, cells)[0]


def _same(a, b):
    np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("make,large,small", [(_ray, (128,), (8,)), (_gradient, (100,), (5,))])
def test_by_turns(m3d, workers, make, large, small):
    jobs = [make(m3d, *large), make(m3d, *small)]
    want = None
    for turn in (0, 1, 0, 1, 0):
        workers[turn].start(jobs[turn])
        got = workers[turn].result()
        if turn == 0:
            want = got if want is None else want
            _same(got, want)


@pytest.mark.parametrize("make,large,small", [(_ray, (128,), (8,)), (_gradient, (100,), (5,)),
                                              (_update, (63, 1), (40, 1)), (_update, (60, 0), (40, 0)),
                                              (_update, (63, 0, True), (40, 0, True)), (_continuum, (4,), (2,))])
def test_side_by_side(m3d, workers, make, large, small):
    jobs = [make(m3d, *large), make(m3d, *small)]
    want = [j() for j in jobs]
    for _ in range(25):
        for w, j in zip(workers, jobs):
            w.start(j)
        for w, r in zip(workers, want):
            _same(w.result(), r)
