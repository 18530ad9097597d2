"""Where launches change from an even share per warp to fetching, and parking.

A launch takes an even share of its queue per warp when the queue holds no more
particles than the grid has lanes.  One CTA of one warp per SM makes that number
small and known: wavefronts one particle below it, at it, one above it and well
above it, against one dense wavefront of all histories.  Parking survivors
(requeue_lanes) works on queues of at least 32768.  FP64 runs agree to the order
of the FP64 atomics (the chunking tolerance of the parity tests).
"""
import numpy as np
import pytest

import egsnrc_gb300 as eg
from egsnrc_gb300 import workloads as W

pytestmark = pytest.mark.gpu
TOL = 1e-12


def transport(n, source=None, **cfg):
    wl = W.water30(10)
    e = eg.DoseEngine(wl["media"], ecut=wl["ecut"], pcut=wl["pcut"], precision=64, **cfg)
    e.set_geometry(wl["geometry"])
    e.set_source(source or wl["source"])
    e.run(n, nbatch=1, seed=9)
    s, t = e.tallies()[0], e.totals()
    e.close()
    return s, t


def agree(a, b):
    assert a[1]["steps"] == b[1]["steps"] > 0
    assert a[0].sum() > 0 and np.allclose(a[0], b[0], rtol=TOL, atol=TOL * a[0].max())
    assert a[1]["deposited"] == pytest.approx(b[1]["deposited"], rel=TOL)


def lanes():
    import torch
    return 32 * torch.cuda.get_device_properties(0).multi_processor_count


# photons fill the photon queue, electrons the electron queue
@pytest.mark.parametrize("charge", [0, -1])
@pytest.mark.parametrize("off", [-1, 0, 1])
def test_shares_and_fetches_meet_at_the_grid_s_lanes(off, charge):
    L = lanes()
    n = 2 * (L + off) + 3
    src = None if charge == 0 else eg.ParallelBeam(charge=-1, energy=3.0, position=(0.0, 0.0, -1.0))
    small = transport(n, src, chunk=L + off, block_size=32, ctas_per_sm=1)
    agree(small, transport(n, src, chunk=n, block_size=32, ctas_per_sm=1))
    agree(small, transport(n, src, chunk=n))


# 40000: a share per warp by default, but parking keeps the fetch; 400000: more than the grid's lanes
@pytest.mark.parametrize("n", [40000, 400000])
@pytest.mark.parametrize("requeue", [8, 24])
def test_parked_particles_resume_with_the_same_result(n, requeue):
    agree(transport(n, chunk=n, requeue_lanes=requeue), transport(n, chunk=n))
