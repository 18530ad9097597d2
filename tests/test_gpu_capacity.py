"""Groups of batches that do not fit the particle queues.

Batches that each fit the queues must run whatever the handle ran before and
however many batches the engine would transport together: a group that
overflows is undone and its batches run in smaller wavefronts.  Nothing of the
first try may stay: sums, sums of squares, energies, counters and per-history
tallies equal those of an engine with ample queues (FP64: the chunking
tolerance of the parity tests, the order of the FP64 atomics).  A batch that
does not fit by itself is still refused.
"""
import numpy as np
import pytest

import egsnrc_gb300 as eg
from egsnrc_gb300 import workloads as W

pytestmark = pytest.mark.gpu
TOL = 1e-12


def electrons():
    return eg.ParallelBeam(charge=-1, energy=20.0, position=(0.0, 0.0, -1.0), rectangle=(-3, 3, -3, 3))


def photons(energy):
    return eg.ParallelBeam(charge=0, energy=energy, position=(0.0, 0.0, -1.0), rectangle=(-3, 3, -3, 3))


def engine(n=20, **cfg):
    e = eg.DoseEngine([W.WATER], ecut=0.521, pcut=0.01, precision=64, **cfg)
    e.set_geometry(W.centred_geometry(n, 30.0 / n))
    return e


def results(e, n, nb, seed):
    e.reset()
    e.set_history_tally(0, n)
    e.run(n, nbatch=nb, seed=seed)
    s, s2, _ = e.tallies()
    t = e.totals()
    return [s, s2, e.history_tally()] + [np.float64(t[k]) for k in ("deposited", "escaped", "steps")]


def agree(got, want):
    for g, w in zip(got, want):
        assert np.max(w) > 0
        assert np.allclose(g, w, rtol=TOL, atol=TOL * np.max(w))


@pytest.mark.parametrize("graph", [0, 1, 2])
@pytest.mark.parametrize("n,nb", [(1000, 10), (1007, 10), (1009, 3)])
def test_batches_that_fit_one_at_a_time_run(graph, n, nb):
    """The estimate has a floor of 1024 histories, more than these queues hold."""
    big = engine()
    big.set_source(photons(6.0))
    want = results(big, n, nb, 5)
    peak = 4 * (n // nb + nb)        # a batch's photons, and its electrons above 10 keV
    e = engine(capacity=peak, use_graph=graph)
    e.set_source(photons(6.0))
    for _ in range(3):               # the later runs with groups that were made smaller
        agree(results(e, n, nb, 5), want)


@pytest.mark.parametrize("nb", [10, 1])
def test_a_chunk_tuned_on_lighter_particles(nb):
    e = engine(capacity=1 << 14)
    e.set_source(photons(0.06))
    e.run(200000, nbatch=1, seed=1)
    assert e.profile()["chunk"] >= 4000
    e.set_source(electrons())
    big = engine()
    big.set_source(electrons())
    n = 20000
    want = results(big, n, nb, 8)
    for _ in range(3):
        agree(results(e, n, nb, 8), want)


def test_several_phantoms():
    probs = [dict(geometry=W.centred_geometry(10 + k, 0.5), source=photons(0.05) if k < 2 else electrons(),
                  seed=70 + k, histories=h) for k, h in enumerate((1500, 900, 601))]
    out = []
    for cfg in ({}, {"capacity": 450}):
        e = eg.DoseEngine([W.WATER], ecut=0.521, pcut=0.01, precision=64, **cfg)
        e.set_phantoms(probs)
        e.run_phantoms(nbatch=10)
        s, s2, _ = e.tallies()
        t = e.totals()
        out.append([s, s2, np.float64(t["deposited"]), np.float64(t["escaped"])])
        e.close()
    agree(out[1], out[0])


def test_a_batch_too_large_by_itself_is_refused_and_leaves_the_handle_usable():
    e = engine(capacity=300)
    e.set_source(photons(6.0))
    with pytest.raises(eg.EGSError) as ex:
        e.run(4000, nbatch=10, seed=5)
    assert ex.value.code == 5
    big = engine()
    big.set_source(photons(6.0))
    agree(results(e, 300, 10, 5), results(big, 300, 10, 5))


def test_batch_slots_leave_a_nearly_full_device_its_memory():
    """With 3 GiB free the slots of ten batches (1.1 GB at 240^3 voxels) are not
    taken: batches run one at a time, with the same result."""
    import torch
    g = W.centred_geometry(240, 0.125)
    out = []
    for fill in (False, True):
        e = eg.DoseEngine([W.WATER], ecut=0.7, pcut=0.01, precision=64, capacity=1 << 16)
        e.set_geometry(g)
        e.set_source(photons(2.0))
        e.run(100, nbatch=1, seed=2)     # queues and kernels are in place
        e.reset()
        torch.cuda.synchronize()
        keep = torch.empty(torch.cuda.mem_get_info()[0] - (3 << 30), dtype=torch.uint8, device="cuda") if fill else None
        free = torch.cuda.mem_get_info()[0]
        e.run(4000, nbatch=20, seed=2)
        torch.cuda.synchronize()
        taken = free - torch.cuda.mem_get_info()[0]
        del keep
        torch.cuda.empty_cache()
        if fill:
            assert taken <= free // 6 + (64 << 20)
        out.append(e.tallies()[:2])
        e.close()
    agree(out[1], out[0])
