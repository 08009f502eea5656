"""The moment kernel's edges with images enough that it runs, which every case asserts.

test_gpu_moments.py names most of these edges too, but its rooms there have fewer images than
the line from which a launch takes this kernel, and are summed tap by tap.  Tolerance as there:
relative L2 <= 1e-6 of the FP64 sum.
"""
import numpy as np
import pytest

import oracle
from conftest import rel_l2

pytestmark = pytest.mark.gpu

TOL = 1e-6


def _inside(rng, n, room):
    room = np.asarray(room)
    return (0.1 * room + rng.random((n, 3)) * 0.8 * room).astype(np.float32)


def _check(room, beta, ps, pr, nb, T, fs, pairs=None, Td=None, pooled=False, **pat):
    import gpurir_gb300 as G
    sim = G.Simulator(seed=5)
    out = sim.simulate_rir(room, beta, ps, pr, pat.get("orV_src"), pat.get("orV_rcv"),
                           G.polar_patterns[pat.get("spkr", "omni")], G.polar_patterns[pat.get("mic", "omni")], nb,
                           Td or T, T, fs)
    assert sim.last_moment_rirs() == len(ps) * len(pr)
    pairs = pairs or [(s, r) for s in range(len(ps)) for r in range(len(pr))]
    got, want = [], []
    for s, r in pairs:
        o = pat.get("orV_src"), pat.get("orV_rcv")
        ref, parts = oracle.simulate_rir(room, beta, ps[s:s + 1], pr[r:r + 1], nb, T, fs, Td or T,
                                         pat.get("spkr", "omni"), pat.get("mic", "omni"),
                                         None if o[0] is None else o[0][s:s + 1], None if o[1] is None else o[1][r:r + 1],
                                         seed=5, offset=0, return_parts=True, rir_base=s * len(pr) + r)
        n = parts["n_ism"]
        if Td:   # FP32 envelope and noise
            assert rel_l2(out[s, r, n:], ref[0, 0, n:]) <= 1e-4
        got.append(out[s, r, :n])
        want.append(ref[0, 0, :n])
        assert pooled or rel_l2(got[-1], want[-1]) <= TOL, (s, r, rel_l2(got[-1], want[-1]))
    assert rel_l2(np.stack(got), np.stack(want)) <= TOL


@pytest.mark.parametrize("n", [2, 160, 162, 510, 512, 514, 1022, 1024, 1026, 1184, 1188, 2048, 2210])
def test_segment_edges(built, n):
    """Early parts that end at, just before and just after a segment or a tile of outputs; a cubic
    box small enough for 3000 images in reach.  (The error is taken over all pairs: a few samples
    of one can nearly cancel.)"""
    rng = np.random.default_rng(n)
    edge = 0.1118 * (n + 64) * 343.0 / 16000.0
    room = [edge, edge, edge]
    _check(room, rng.uniform(0.6, 0.95, 6).astype(np.float32), _inside(rng, 3, room), _inside(rng, 4, room),
           [21, 22, 23], n / 16000.0, 16000.0, pooled=True)


@pytest.mark.parametrize("n_rir", [(1, 1), (19, 17)])   # parts of the image rows; whole items
@pytest.mark.parametrize("fs", [6000.0, 6125.0])        # the shortest windows: 48 samples, an odd one
def test_shortest_windows(built, fs, n_rir):
    room = [3.4, 3.1, 2.5]
    rng = np.random.default_rng(int(fs))
    ps, pr = _inside(rng, n_rir[0], room), _inside(rng, n_rir[1], room)
    _check(room, rng.uniform(0.6, 0.95, 6).astype(np.float32), ps, pr, [24, 25, 31], 0.11, fs,
           pairs=[(0, 0), (n_rir[0] - 1, n_rir[1] - 1)], spkr="subcard", mic="hypcard",
           orV_src=rng.standard_normal((len(ps), 3)).astype(np.float32),
           orV_rcv=rng.standard_normal((len(pr), 3)).astype(np.float32))


@pytest.mark.parametrize("gap", [1e-4, 0.01, 0.049])
def test_source_next_to_the_receiver(built, gap):
    rng = np.random.default_rng(7)
    room = [3.0, 4.0, 2.5]
    pr = _inside(rng, 2, room)
    ps = pr + np.array([gap, 0, 0], np.float32)
    _check(room, rng.uniform(0.6, 0.95, 6).astype(np.float32), ps, pr, [31, 24, 37], 0.13, 16000.0)


def test_source_outside_the_room(built):
    """Image rows are then not in order of distance."""
    rng = np.random.default_rng(10)
    room = [3.0, 4.0, 2.5]
    ps = np.array([[-1.7, 5.2, 6.1], [4.4, 2.0, -3.3]], np.float32)
    _check(room, rng.uniform(0.6, 0.95, 6).astype(np.float32), ps, _inside(rng, 2, room), [31, 24, 37], 0.13, 16000.0)


def test_absorbing_walls(built):
    """beta = 0 on some walls: images of zero amplitude, one row of them left."""
    rng = np.random.default_rng(11)
    room = [3.0, 4.0, 2.5]
    _check(room, np.array([0.0, 0.0, 0.0, 0.0, 0.9, 0.8], np.float32), _inside(rng, 2, room), _inside(rng, 2, room),
           [31, 24, 37], 0.13, 16000.0)


@pytest.mark.parametrize("fs", [8000.0, 16000.0, 24000.0])   # 24 kHz: the most cells of the small blocks
@pytest.mark.parametrize("tail", [False, True])
def test_launches_of_many_segments(built, fs, tail):
    """Three blocks per SM, with the tail that their last items write."""
    rng = np.random.default_rng(int(fs))
    room = [3.5, 3.0, 2.6]
    _check(room, rng.uniform(0.6, 0.95, 6).astype(np.float32), _inside(rng, 40, room), _inside(rng, 36, room),
           [16, 16, 17], 0.3 if tail else 0.2, fs, pairs=[(0, 0), (17, 20), (39, 35)], Td=0.15 if tail else None)
