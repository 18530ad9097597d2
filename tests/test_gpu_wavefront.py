"""The wavefront: batches transported together, sparse launches, the generator window.

Batches transported together (one tally slot each) against batches run one at
a time: sum and sum of squares over batches.  A slot's deposits are added in
another order (FP64 atomics), so the two agree to the chunking tolerance of the
parity tests: about 1e3 additions of FP64 values per voxel, 1e3 * 2^-53 < 1e-12.
FP32 runs may also merge the deposits of two particles of one history in FP32
(6e-8 of one deposit), hence their 2e-5 bound, the scheduling tolerance there.
"""
import numpy as np
import pytest

import egsnrc_gb300 as eg
from egsnrc_gb300 import workloads as W

pytestmark = pytest.mark.gpu
TOL = {64: 1e-12, 32: 2e-5}


def ranges(n, nb):
    per = n // nb
    return [(b * per, per if b < nb - 1 else n - b * per) for b in range(nb)]


def one_by_one(e, n, nb, seed):
    s = s2 = 0
    for first, cnt in ranges(n, nb):
        e.reset()
        e.run(cnt, nbatch=1, seed=seed, first=first)
        d = e.tallies()[0]
        s, s2 = s + d, s2 + d * d
    return s, s2


# chunk 0: all batches in one group; 300: groups of two whose wavefronts are
# cut inside a batch; 40: smaller than a batch, so each batch runs alone
@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("n,nb,cfg", [(1003, 7, {}), (1003, 7, {"chunk": 300}), (1003, 7, {"chunk": 40}),
                                      (20, 20, {}), (1003, 7, {"use_graph": 1}), (1003, 7, {"use_graph": 2}),
                                      (1003, 7, {"use_graph": 1, "chunk": 300}), (501, 1, {})])
def test_grouped_batches_equal_single_batches(n, nb, cfg, precision):
    wl = W.slab64(16)
    def engine(**kw):
        e = eg.DoseEngine(wl["media"], ecut=wl["ecut"], pcut=wl["pcut"], precision=precision, **kw)
        e.set_geometry(wl["geometry"])
        e.set_source(wl["source"])
        return e
    want = one_by_one(engine(), n, nb, 5)
    e = engine(**cfg)
    for _ in range(2):            # a second run finds every slot cleared
        e.reset()
        e.run(n, nbatch=nb, seed=5)
        got = e.tallies()[:2]
        for g, w in zip(got, want):
            assert w.sum() > 0
            assert np.allclose(g, w, rtol=TOL[precision], atol=TOL[precision] * w.max())
    # a smaller geometry and fewer batches on the same handle
    e.set_geometry(W.slab64(8)["geometry"])
    e.run(60, nbatch=3, seed=6)
    f = engine()
    f.set_geometry(W.slab64(8)["geometry"])
    for g, w in zip(e.tallies()[:2], one_by_one(f, 60, 3, 6)):
        assert np.allclose(g, w, rtol=TOL[precision], atol=TOL[precision] * w.max())


@pytest.mark.parametrize("cfg", [{}, {"chunk": 200}, {"use_graph": 2}])
def test_grouped_batches_of_several_phantoms(cfg):
    nb = 3
    def phantoms(counts):
        return [dict(W.batch_problem(k, edge=(8 + 3 * k, 8 + 3 * k)), histories=c) for k, c in enumerate(counts)]
    counts = [100, 3, 331, 0, 57]
    e = eg.DoseEngine(W.BATCH_MEDIA, ecut=0.7, pcut=0.01, precision=64, **cfg)
    e.set_phantoms(phantoms(counts))
    e.run_phantoms(nbatch=nb)
    for k, c in enumerate(counts):
        s, s2 = e.phantom_tallies(k)
        if not c:
            assert not s.any()
            continue
        ph = phantoms(counts)[k]
        f = eg.DoseEngine(W.BATCH_MEDIA, ecut=0.7, pcut=0.01, precision=64)
        f.set_geometry(ph["geometry"])
        f.set_source(ph["source"])
        for g, w in zip((s, s2), one_by_one(f, c, nb, ph["seed"])):
            assert np.allclose(g, w, rtol=TOL[64], atol=TOL[64] * max(w.max(), 1e-30))


# the sparse launch's edges: fewer particles than warps, one or two per warp, a
# few more than the grid has lanes (about 1e5), and requeue on a sparse launch
@pytest.mark.parametrize("n,requeue", [(1, 0), (33, 0), (5000, 0), (120000, 0), (60000, 24)])
def test_sparse_launches_take_every_particle_once(n, requeue):
    wl = W.water30(10)
    t = []
    for cfg in ({}, {"chunk": 1009, "block_size": 32, "ctas_per_sm": 1, "requeue_lanes": requeue}):
        e = eg.DoseEngine(wl["media"], ecut=wl["ecut"], pcut=wl["pcut"], precision=32, **cfg)
        e.set_geometry(wl["geometry"])
        e.set_source(wl["source"])
        e.run(n, nbatch=1, seed=9)
        t.append((e.tallies()[0], e.totals()))
        e.close()
    assert t[0][1]["steps"] == t[1][1]["steps"] > 0
    assert t[0][1]["deposited"] + t[0][1]["escaped"] == pytest.approx(2.0 * n, rel=1e-6)
    assert np.allclose(t[0][0], t[1][0], rtol=TOL[32], atol=TOL[32] * t[0][0].max())


def test_requeue_on_a_sparse_launch_makes_progress():
    wl = W.water30(10)
    t = []
    for requeue in (0, 24):
        e = eg.DoseEngine(wl["media"], ecut=wl["ecut"], pcut=wl["pcut"], precision=32, requeue_lanes=requeue)
        e.set_geometry(wl["geometry"])
        e.set_source(wl["source"])
        e.run(60000, nbatch=1, seed=9)
        t.append(e.totals()["steps"])
        e.close()
    assert t[0] == t[1] > 0


def test_positrons_follow_the_oracle_one_by_one():
    """A Bhabha positron below the cut-off annihilates on its own stream, drawing
    through the thread's one generator window between two draws of its parent.
    20 MeV histories do not fork in 0.8 cm voxels, so nearly all 4000 must agree
    (a parent that read the other stream's numbers: 2 in 1000 histories)."""
    from oracle.oracle_binding import Oracle
    n = 4000
    g = W.centred_geometry(15, 1.0, (np.arange(15 ** 3) % 7 == 0).astype(np.int32))
    src = eg.ParallelBeam(charge=1, energy=10.0, position=(0.0, 0.0, -1.0), rectangle=(-3, 3, -3, 3))
    e = eg.DoseEngine([W.WATER, W.BONE], ecut=0.521, pcut=0.01, precision=64)
    o = Oracle([W.WATER, W.BONE], ecut=0.521, pcut=0.01)
    for x in (e, o):
        x.set_geometry(g)
        x.set_source(src)
        x.set_history_tally(0, n)
    e.run(n, nbatch=1, seed=3)
    o.run(n, nbatch=1, seed=3, threads=8)
    hg, ho = e.history_tally(), o.history_tally()
    assert np.sum(np.abs(hg - ho) > 1e-6 * np.maximum(1e-12, np.abs(ho))) <= 2
