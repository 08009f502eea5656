"""workloads.images_and_samples against a count image by image."""
import numpy as np

from gpurir_gb300 import workloads


def test_images_and_samples():
    rng = np.random.default_rng(2)
    room, nb, fs, T = np.array([3.0, 2.6, 2.4]), [5, 4, 3], 8000.0, 0.02
    ps, pr = rng.random((2, 3)) * room, rng.random((3, 3)) * room
    n, H = workloads.n_samples(T, fs), 32.0
    images = samples = 0
    for s in ps:
        for r in pr:
            last = 0.0
            for m in np.ndindex(*nb):
                k = np.array(m) - np.array(nb) // 2
                v = 2 * np.ceil(k / 2.0) * room + np.where(k % 2, -s, s) - r
                tau = np.linalg.norm(v) * fs / 343.0
                images += tau < n + H
                last = max(last, tau)
            samples += min(last + H, n)
    got = workloads.images_and_samples(dict(room_sz=room, nb_img=nb, fs=fs, Tmax=T, pos_src=ps, pos_rcv=pr))
    assert got[0] == images < 6 * np.prod(nb) and abs(got[1] - samples) <= 2   # (whole samples per source)
