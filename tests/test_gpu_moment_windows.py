"""Quiet stretches of an RIR by the moment kernel: every 128 samples against the FP64 oracle.

The norm of a whole RIR is that of its first images, and hides what happens to samples that are
a thousand times weaker within one segment of 1024.  Here the error of 128 samples is held
against what the images that reach them amount to: the root of the sum of their taps' squares, each
tap at the size that a delay between two samples gives it.  (Of a lone image whose delay is nearly
a whole sample the far taps almost vanish, and the rounding of its delay shows in them, in any
FP32 evaluation.)  Per image: the fraction of its delay to 2^-24 sample, 1.9e-7 of such a tap at
most; its amplitude 1e-7; tables and sums 1e-7.  Together 2.4e-7; 1e-6 leaves a factor of four.
At the last tap on either side, where the window ends inside a cell of two samples, the tables are
good to 2e-8 of the image's largest tap instead: as if that tap were 0.02.
"""
import numpy as np
import pytest

import oracle
from conftest import rel_l2

pytestmark = pytest.mark.gpu

TOL = 1e-6
W = 128


def _scene(seed, dist, n_rcv=3):
    """Receivers near the middle of a 5 x 4 x 3 m room, the first one dist from the source."""
    rng = np.random.default_rng(seed)
    pr = (1.3 + rng.random((n_rcv, 3)) * 0.5).astype(np.float32)
    d = rng.standard_normal(3)
    return (pr[:1] + dist * d / np.linalg.norm(d)).astype(np.float32), pr


def _counts(T, room=(5.0, 4.0, 3.0)):
    return [int(np.ceil(2 * (T + 0.02) * 343.0 / v)) for v in room]


def _beta(walls):
    """One coefficient for every wall, or two reverberant walls between four dull ones."""
    return np.array([0.99, 0.99, 0.1, 0.1, 0.1, 0.1] if walls == "flutter" else [walls] * 6, np.float32)


def _images(room, beta, ps, pr, nb, fs):
    """Delays in samples and wall factors (their size) of every image of one pair, and distances."""
    d2, att = np.zeros((1, 1, 1)), np.ones((1, 1, 1))
    for a in range(3):
        k = np.arange(nb[a]) - nb[a] // 2
        c, odd = (k + 1) // 2, k % 2
        v = 2.0 * c * room[a] + (1 - 2 * odd) * float(ps[a]) - float(pr[a])
        shape = [-1 if b == a else 1 for b in range(3)]
        d2 = d2 + (v * v).reshape(shape)
        f = float(beta[2 * a]) ** np.abs(c - odd) * float(beta[2 * a + 1]) ** np.abs(c)
        att = att * f.reshape(shape)
    d = np.sqrt(d2.ravel())
    return d * fs / 343.0, att.ravel(), d


def _reach(tau, amp, n, fs):
    """Per sample, the sum of the squares of the taps that images at these delays have on it."""
    H = round(0.008 * fs) // 2
    p = np.bincount(np.minimum(tau.astype(int), n + H), weights=amp ** 2, minlength=n + H + 1)[:n + H]
    k = np.arange(-H, H + 2)
    size = 0.5 * (1 + np.cos(np.pi * np.minimum(np.abs(k), H) / H)) / np.maximum(1.0, np.pi * np.abs(k))
    size[[0, 1, -2, -1]] = 0.02
    return np.convolve(p, size ** 2)[H:H + n]


def _worst_window(out, ref, reach):
    first = int(np.nonzero(np.abs(ref) > 1e-3 * np.abs(ref).max())[0][0])
    e2 = (out.astype(np.float64) - ref) ** 2
    return max(np.sqrt(e2[t:t + W].sum() / reach[t:t + W].sum()) for t in range(first, len(ref) - W + 1, W))


@pytest.mark.parametrize("walls", [0.02, 0.1, 0.3, 0.6, "flutter"])
@pytest.mark.parametrize("dist", [1.0, 0.3, 0.06])
@pytest.mark.parametrize("fs,T", [(8000.0, 0.2), (16000.0, 0.13), (48000.0, 0.06)])
def test_windows(built, fs, T, dist, walls):
    import gpurir_gb300 as G
    room, nb, beta = [5.0, 4.0, 3.0], _counts(T), _beta(walls)
    ps, pr = _scene(3, dist)
    sim = G.Simulator()
    out = sim.simulate_rir(room, beta, ps, pr, None, None, 0, 0, nb, T, T, fs)
    assert sim.last_moment_rirs() == 3
    ref = oracle.simulate_rir(room, beta, ps, pr, nb, T, fs)
    for r in range(3):
        tau, att, d = _images(room, beta, ps[0], pr[r], nb, fs)
        assert _worst_window(out[0, r], ref[0, r], _reach(tau, att / (4 * np.pi * d), ref.shape[2], fs)) <= TOL


def test_crowded_cells(built):
    """The same where cells hold thousands of images: more than the sums' first scale, rows past one batch."""
    import gpurir_gb300 as G
    room, nb, fs, T = [0.3, 0.33, 0.27], [71, 67, 79], 16000.0, 0.03
    rng = np.random.default_rng(6)
    ps, pr = [(0.1 * np.array(room) + rng.random((n, 3)) * 0.8 * np.array(room)).astype(np.float32) for n in (20, 16)]
    beta = _beta(0.6)
    sim = G.Simulator()
    out = sim.simulate_rir(room, beta, ps, pr, None, None, 0, 0, nb, T, T, fs)
    assert sim.last_moment_rirs() == 320
    for s, r in ((0, 0), (19, 15)):
        ref = oracle.simulate_rir(room, beta, ps[s:s + 1], pr[r:r + 1], nb, T, fs)[0, 0]
        tau, att, d = _images(room, beta, ps[s], pr[r], nb, fs)
        assert _worst_window(out[s, r], ref, _reach(tau, att / (4 * np.pi * d), len(ref), fs)) <= TOL


@pytest.mark.parametrize("walls", [0.1, 0.3])
def test_tail_level(built, walls):
    """The diffuse tail's level comes from the last 10 ms of an early part of one segment."""
    import gpurir_gb300 as G
    room, fs, Td, T = [2.0, 1.7, 1.5], 16000.0, 0.06, 0.2
    rng = np.random.default_rng(4)
    ps, pr = (0.3 + rng.random((1, 3))).astype(np.float32), (0.3 + rng.random((2, 3))).astype(np.float32)
    nb = _counts(Td, room)
    sim = G.Simulator(seed=9)
    out = sim.simulate_rir(room, _beta(walls), ps, pr, None, None, 0, 0, nb, Td, T, fs)
    assert sim.last_moment_rirs() == 2
    ref, p = oracle.simulate_rir(room, _beta(walls), ps, pr, nb, T, fs, Td, seed=9, offset=0, return_parts=True)
    n = p["n_ism"]
    for r in range(2):
        assert rel_l2(out[0, r, n - 160:n], ref[0, r, n - 160:n]) <= 2 * TOL
        assert rel_l2(out[0, r, n:], ref[0, r, n:]) <= 1e-4   # FP32 envelope and noise


def test_amplitudes_past_float32(built):
    """Walls that amplify until their factors overflow: the samples before the first infinite image
    are what they are without it, and the overflow shows from its first tap on."""
    import gpurir_gb300 as G
    room, fs, T = [3.0, 4.0, 2.5], 16000.0, 0.13
    rng = np.random.default_rng(5)
    ps, pr = (0.5 + rng.random((1, 3))).astype(np.float32), (0.5 + rng.random((1, 3))).astype(np.float32)
    nb, beta = _counts(T, room), np.full(6, 1e5, np.float32)   # eight reflections are past 3.4e38
    sim = G.Simulator()
    out = sim.simulate_rir(room, beta, ps, pr, None, None, 0, 0, nb, T, T, fs)[0, 0]
    assert sim.last_moment_rirs() == 1
    ref = oracle.simulate_rir(room, beta, ps, pr, nb, T, fs)[0, 0]
    tau, att, _ = _images(room, beta, ps[0], pr[0], nb, fs)
    bad = int(np.nonzero(~np.isfinite(out))[0][0])
    assert 0 <= tau[att > 3.4e38].min() - 64 - bad <= 8   # its window, to the filter's groups of four cells
    assert rel_l2(out[:bad], ref[:bad]) <= 1e-6
