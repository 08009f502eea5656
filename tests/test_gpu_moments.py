"""The moment kernel (ism_moment.cu) at the sizes where it can go wrong, against the FP64 oracle.

Tolerance: an RIR of the FP32 path is within 3e-7 relative L2 of the FP64 sum (delays and
amplitudes of each image to ~1e-7, the filter's tables 4e-8, FP32 sums of ~200 terms 1e-7);
1e-6 leaves a factor of three.
"""
import numpy as np
import pytest

import oracle
from conftest import rel_l2

pytestmark = pytest.mark.gpu

TOL = 1e-6


def _scene(seed, room, ns, nr):
    rng = np.random.default_rng(seed)
    room = np.asarray(room)
    inside = lambda n: (0.1 * room + rng.random((n, 3)) * 0.8 * room).astype(np.float32)
    return inside(ns), inside(nr), rng.uniform(0.6, 0.95, 6).astype(np.float32)


def _check(room, beta, ps, pr, nb, T, fs, pairs=None, spkr="omni", mic="omni", os_=None, or_=None, tol=TOL):
    import gpurir_gb300 as G
    sim = G.Simulator()
    args = (room, beta, ps, pr, os_, or_, G.polar_patterns[spkr], G.polar_patterns[mic], nb, T, T, fs)
    out = sim.simulate_rir(*args).copy()
    assert np.array_equal(out, sim.simulate_rir(*args))   # any order of the atomics, the same bits
    for s, r in pairs or [(s, r) for s in range(len(ps)) for r in range(len(pr))]:
        ref = oracle.simulate_rir(room, beta, ps[s:s + 1], pr[r:r + 1], nb, T, fs, spkr_pattern=spkr, mic_pattern=mic,
                                  orV_src=None if os_ is None else os_[s:s + 1],
                                  orV_rcv=None if or_ is None else or_[r:r + 1])
        assert rel_l2(out[s, r], ref[0, 0]) <= tol, (s, r, rel_l2(out[s, r], ref[0, 0]))
    return out


@pytest.mark.parametrize("n", [2, 160, 162, 510, 512, 514, 1022, 1026, 1184, 1188, 2048, 2210])
def test_segment_edges(built, n):
    """Early parts that end at, just before and just after a segment or a tile of outputs."""
    ps, pr, beta = _scene(n, [3.0, 2.6, 2.4], 1, 2)
    _check([3.0, 2.6, 2.4], beta, ps, pr, [9, 10, 11], n / 16000.0, 16000.0)


@pytest.mark.parametrize("n_rir", [(1, 1), (19, 17)])   # parts of the image rows; whole items
@pytest.mark.parametrize("fs", [6000.0, 8000.0, 11025.0, 22050.0, 44100.0, 50000.0])
def test_window_lengths(built, fs, n_rir):
    """The shortest and longest window of the kernel, odd windows, windows that end inside a cell."""
    ps, pr, beta = _scene(int(fs), [3.4, 3.1, 2.5], *n_rir)
    last = (n_rir[0] - 1, n_rir[1] - 1)
    rng = np.random.default_rng(1)
    _check([3.4, 3.1, 2.5], beta, ps, pr, [21, 22, 27], 0.09, fs, pairs=[(0, 0), last], spkr="subcard", mic="hypcard",
           os_=rng.standard_normal((len(ps), 3)).astype(np.float32),
           or_=rng.standard_normal((len(pr), 3)).astype(np.float32))


def test_rows_past_one_batch(built):
    """More image rows than a block takes at once, in one item per segment."""
    ps, pr, beta = _scene(5, [2.0, 2.2, 6.0], 18, 18)
    _check([2.0, 2.2, 6.0], beta, ps, pr, [41, 38, 14], 0.1, 16000.0, pairs=[(0, 0), (17, 17), (3, 11)])


def test_symmetric_scene(built):
    """Source and receiver at the centre of a cube: up to 48 images of one delay."""
    c = np.full((1, 3), 1.5, np.float32)
    _check([3.0] * 3, np.full(6, 0.9, np.float32), c, c + np.float32(0.0078125), [24] * 3, 0.1, 16000.0)


def test_more_images_per_cell_than_the_sums_hold(built):
    """A small box with images to 25 m and RIRs enough that no segment is dealt out: cells of
    5000 images, past the 2048 of the first scale."""
    room = [0.5, 0.5, 0.5]
    ps, pr, _ = _scene(6, room, 20, 16)
    _check(room, np.full(6, 0.97, np.float32), ps, pr, [101, 101, 101], 0.073, 16000.0, pairs=[(0, 0), (19, 15)])


@pytest.mark.parametrize("centred", [False, True])   # True: many images of one delay, cells past the packed sums
@pytest.mark.parametrize("edge", [3.0, 2.0, 1.5, 1.2, 1.0])
def test_packed_sums(built, edge, centred):
    """Cells of 15 to 400 images: each width of the packed sums, both sides of the last one."""
    room = [edge, edge, edge] if centred else [edge, 1.1 * edge, 0.9 * edge]
    ps, pr, beta = _scene(int(10 * edge), room, 20, 16)
    if centred:
        ps[0] = pr[0] = 0.5 * edge
        pr[0, 0] += np.float32(0.06)
    n = int(2 * 27.0 / edge) + 3
    _check(room, beta, ps, pr, [n, n, n + 4], 0.08, 16000.0, pairs=[(0, 0), (19, 15)])


@pytest.mark.parametrize("gap", [1e-4, 0.01, 0.049])
def test_source_next_to_the_receiver(built, gap):
    """Direct paths below the 5 cm of the first scale: the loud list."""
    room = [3.0, 4.0, 2.5]
    _, pr, beta = _scene(7, room, 1, 2)
    ps = pr + np.array([gap, 0, 0], np.float32)
    _check(room, beta, ps, pr, [9, 9, 9], 0.08, 16000.0)


def test_more_loud_images_than_the_list_holds(built):
    """A 4 cm box: dozens of images within 5 cm, so the segment is done again at the true bound."""
    room = [0.04, 0.04, 0.04]
    ps, pr, beta = _scene(8, room, 1, 2)
    _check(room, beta, ps, pr, [15, 15, 15], 0.02, 16000.0)


def test_walls_that_amplify(built):
    """beta above one: the scale follows the indices that each segment reaches."""
    room = [3.0, 4.0, 2.5]
    ps, pr, _ = _scene(9, room, 1, 2)
    _check(room, np.array([1.3, 0.9, 1.1, 1.2, 0.8, 1.4], np.float32), ps, pr, [17, 15, 21], 0.12, 16000.0)


def test_source_outside_the_room(built):
    """Image rows are then not in order of distance."""
    import gpurir_gb300 as G
    room = [3.0, 4.0, 2.5]
    _, pr, beta = _scene(10, room, 1, 2)
    ps = np.array([[-1.7, 5.2, 6.1], [4.4, 2.0, -3.3]], np.float32)
    _check(room, beta, ps, pr, [9, 8, 11], 0.1, 16000.0)


def test_absorbing_walls(built):
    """beta = 0 on some walls: images of zero amplitude, one row of them left."""
    room = [3.0, 4.0, 2.5]
    ps, pr, _ = _scene(11, room, 2, 2)
    _check(room, np.array([0.0, 0.0, 0.0, 0.0, 0.9, 0.8], np.float32), ps, pr, [9, 9, 15], 0.1, 16000.0)


@pytest.mark.parametrize("fs,n_img", [(8000.0, 9), (16000.0, 9), (24000.0, 9), (16000.0, 64)])   # 24 kHz: the widest window
@pytest.mark.parametrize("tail", [False, True])
def test_launches_of_many_segments(built, fs, n_img, tail):
    """Launches large enough for three blocks per SM, with the tail that their last items write;
    64 images per axis: tables of nearly 200 entries."""
    import gpurir_gb300 as G
    room = [3.5, 3.0, 2.6]
    ps, pr, beta = _scene(int(fs), room, 40, 36)
    T, Td = 0.3 if tail else 0.2, 0.2
    sim = G.Simulator(seed=5)
    nb = [n_img, n_img, n_img + 1]
    out = sim.simulate_rir(room, beta, ps, pr, None, None, 0, 0, nb, Td, T, fs)
    for s, r in [(0, 0), (17, 20), (39, 35)]:
        ref, parts = oracle.simulate_rir(room, beta, ps[s:s + 1], pr[r:r + 1], nb, T, fs, Td, seed=5, offset=0,
                                         return_parts=True, rir_base=s * 36 + r)
        n = parts["n_ism"]
        assert rel_l2(out[s, r, :n], ref[0, 0, :n]) <= TOL
        assert not tail or rel_l2(out[s, r, n:], ref[0, 0, n:]) <= 1e-4   # FP32 envelope and noise
