"""Runs on a caller's stream that does not wait for the default stream.

The engine clears tallies and uploads on the default stream; a run on a
non-blocking stream (every torch.cuda.Stream is one) must wait for that work,
and the clearing of batch slots must come before the deposits.  The same
histories on either stream deposit the same energy: FP64 runs agree to the
order of the FP64 atomics (the chunking tolerance of the parity tests), and a
run's sums add up to the energy it counted as deposited, FP32 deposits being
rounded once per addition (1e-6 relative).
"""
import numpy as np
import pytest

import egsnrc_gb300 as eg
from egsnrc_gb300 import workloads as W

pytestmark = pytest.mark.gpu
TOL = 1e-12


def side_stream():
    import torch
    return torch.cuda.Stream()


def beam(half=5.0):
    return eg.ParallelBeam(charge=0, energy=2.0, position=(0.0, 0.0, -1.0), rectangle=(-half, half, -half, half))


def test_batch_slots_on_a_side_stream():
    """256^3 voxels: ten slots are 1.3 GB to clear, while the first deposits of
    1e4 histories come after tens of microseconds."""
    s = side_stream()
    g = W.centred_geometry(256, 0.1)
    sums = []
    for stream in (None, s.cuda_stream):
        e = eg.DoseEngine([W.WATER], ecut=0.7, pcut=0.01, precision=64)
        e.set_geometry(g)
        e.set_source(beam())
        for _ in range(2):       # the second time after a new upload
            e.run(10000, nbatch=10, seed=4, stream=stream)
            t = e.totals()
            sums.append(e.tallies()[0])
            assert sums[-1].sum() == pytest.approx(t["deposited"], rel=1e-6)
            e.set_geometry(g)
            e.reset()
        e.close()
    for x in sums[1:]:
        assert np.allclose(x, sums[0], rtol=TOL, atol=TOL * sums[0].max())


@pytest.mark.parametrize("precision", [64, 32])
def test_reset_and_uploads_are_ordered_before_a_side_stream(precision):
    s = side_stream()
    g = [W.centred_geometry(160, 0.15), W.centred_geometry(96, 0.25)]
    e = eg.DoseEngine([W.WATER], ecut=0.7, pcut=0.01, precision=precision)
    e.set_source(beam())
    want = {}
    for stream in (None, s.cuda_stream, s.cuda_stream):
        for k, geom in enumerate(g):
            e.set_geometry(geom)
            e.reset()
            e.run(3000, nbatch=1, seed=7, stream=stream)
            e.reset()
            e.run(3000, nbatch=5, seed=7, stream=stream)
            got = e.tallies()[0]
            assert got.sum() == pytest.approx(e.totals()["deposited"], rel=1e-6)
            w = want.setdefault(k, got)
            tol = TOL if precision == 64 else 2e-5
            assert np.allclose(got, w, rtol=tol, atol=tol * w.max())
    e.close()


def test_phantoms_and_noalloc_on_a_side_stream():
    import torch
    s = side_stream()
    probs = [dict(W.batch_problem(k, edge=(20 + k, 20 + k)), histories=200 + 7 * k) for k in range(3)]
    sums = []
    for stream in (None, s.cuda_stream):
        e = eg.DoseEngine(W.BATCH_MEDIA, ecut=0.7, pcut=0.01, precision=64)
        e.set_phantoms(probs)
        e.run_phantoms(nbatch=5, stream=stream)
        sums.append(e.tallies()[:2])
        e.close()
    for a, b in zip(*sums):
        assert a.sum() > 0 and np.allclose(a, b, rtol=TOL, atol=TOL * a.max())
    g = W.centred_geometry(96, 0.25)
    dose = torch.empty(g.nvox, dtype=torch.float64, device="cuda")
    out = []
    for stream in (None, s.cuda_stream):
        e = eg.DoseEngine([W.WATER], ecut=0.7, pcut=0.01, precision=64)
        e.set_geometry(g)
        e.set_source(beam())
        torch.cuda.synchronize()
        e.run_noalloc(dose.data_ptr(), 500, seed=3, stream=stream)
        out.append(dose.cpu().numpy().copy())
        e.close()
    assert out[0].sum() > 0 and np.allclose(out[0], out[1], rtol=TOL, atol=TOL * out[0].max())
