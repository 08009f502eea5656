"""Batches in which rooms of a few images stand between dense ones.

Dense rooms take the moment kernel; a room of fewer than 64 images in reach keeps its taps, with the
same bits as in a batch without the dense rooms, and tail and RIRs agree with the FP64 oracle
(early part 1e-6 relative L2, as the other tests of both kernels; tails 1e-4, FP32 envelope and noise).
"""
import numpy as np
import pytest

import oracle
from conftest import rel_l2

pytestmark = pytest.mark.gpu

FS = 16000.0


def _room(rng, size, n_img, ns, nr, tail):
    size = np.array(size)
    inside = lambda n: (0.1 * size + rng.random((n, 3)) * 0.8 * size).astype(np.float32)
    return dict(room_sz=size.astype(np.float32), beta=rng.uniform(0.7, 0.95, 6).astype(np.float32), pos_src=inside(ns),
                pos_rcv=inside(nr), nb_img=n_img, Tmax=0.15, Tdiff=0.07 if tail else 0.15)


def _rooms(tail):
    rng = np.random.default_rng(3)
    dense = lambda ns, nr: _room(rng, [2.0, 2.2, 2.4], [30, 28, 26], ns, nr, tail)
    few = lambda n, ns, nr: _room(rng, [6.0, 5.0, 3.0], n, ns, nr, tail)
    return [few([1, 1, 1], 2, 3), dense(2, 3), few([2, 2, 2], 1, 2), dense(1, 5), dense(3, 2), few([3, 3, 3], 2, 1)]


@pytest.mark.parametrize("tail", [False, True])
def test_few_images_between_dense_rooms(built, tail):
    import torch
    import gpurir_gb300 as G
    from gpurir_gb300 import batch as B
    rooms = _rooms(tail)
    small = [k for k, r in enumerate(rooms) if np.prod(r["nb_img"]) < 64]
    sim = G.Simulator(seed=21)
    flat, _ = B.simulate_batch(rooms, FS, sim=sim)
    assert sim.last_moment_rirs() == sum(len(r["pos_src"]) * len(r["pos_rcv"]) for k, r in enumerate(rooms) if k not in small)
    out = B.unpack(flat.cpu().numpy(), rooms, FS)
    alone = B.simulate_batch([rooms[k] for k in small], FS, sim=sim)[0].cpu().numpy()
    assert sim.last_moment_rirs() == 0
    alone = B.unpack(alone, [rooms[k] for k in small], FS)
    n = oracle.n_samples(rooms[0]["Tdiff"], FS)
    for k, a in zip(small, alone):
        assert np.array_equal(out[k][..., :n], a[..., :n])
    plan = B.BatchPlan(rooms, FS, sim=sim)   # the same launches in a graph, replayed twice
    for _ in range(2):
        again = B.unpack(plan.launch().cpu().numpy(), rooms, FS)
        for x, y in zip(out, again):
            assert np.array_equal(x[..., :n], y[..., :n])
    torch.cuda.synchronize()
    base = 0
    for r, v in zip(rooms, out):
        ref = oracle.simulate_rir(r["room_sz"], r["beta"], r["pos_src"], r["pos_rcv"], r["nb_img"], r["Tmax"], FS,
                                  r["Tdiff"], seed=21, offset=0, rir_base=base)
        for s in range(v.shape[0]):
            for m in range(v.shape[1]):
                assert rel_l2(v[s, m, :n], ref[s, m, :n]) <= 1e-6
                assert rel_l2(v[s, m, n:], ref[s, m, n:]) <= 1e-4
        base += v.shape[0] * v.shape[1]
