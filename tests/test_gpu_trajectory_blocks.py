"""The trajectory adjoint in blocks of lags (traj_adjoint_blk_kernel), against the FP64 oracle.

Tolerance as in test_gpu_trajectory_adjoint.py: relative L2 <= 2e-6 (float32 FFTs).  Cases: rows
just past one 2048-point problem, lengths that leave the last block partly or nearly empty,
odd lengths, the longest segment of the path and one past it (whole rows), uneven and empty
segments, one point and one receiver.
"""
import numpy as np
import pytest

import oracle
from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P,R,L,seg", [
    (3, 2, 2001, 48),      # two blocks: L + S - 1 = 2048 is one problem, 2049 is not (below)
    (3, 2, 2002, 48),
    (1, 1, 4097, 1),       # a segment of one sample
    (5, 3, 3333, 250),     # odd, the last block short
    (2, 1, 12801, 400),
    (4, 2, 2500, 1024),    # longest segment
    (4, 2, 2500, 1025),    # whole rows
])
def test_block_adjoint_matches_oracle(built, P, R, L, seg):
    import torch
    from gpurir_gb300.trajectory import simulate_trajectory_torch
    rng = np.random.default_rng(P * 1000 + L + seg)
    n = P * seg
    sig = rng.standard_normal(n).astype(np.float32)
    rir = (rng.standard_normal((P, R, L)) * np.exp(-4 * np.arange(L) / L)).astype(np.float32)
    ts = torch.from_numpy(sig).cuda().requires_grad_(True)
    tr = torch.from_numpy(rir).cuda().requires_grad_(True)
    y = simulate_trajectory_torch(ts, tr)
    G = rng.standard_normal(tuple(y.shape))
    y.backward(torch.from_numpy(G).cuda())
    gs, gr = oracle.trajectory_adjoint(sig, rir, G, None, None)
    assert rel_l2(ts.grad.cpu().numpy(), gs) < 2e-6
    assert rel_l2(tr.grad.cpu().numpy(), gr) < 2e-6


def test_block_adjoint_uneven_segments_and_a_bad_receiver(built):
    """Custom time stamps with an empty segment; then a NaN in one receiver's gradient leaves the
    other receivers' RIR gradients as they were."""
    import torch
    from gpurir_gb300.trajectory import simulate_trajectory_torch
    rng = np.random.default_rng(4)
    fs, stamps, n, P, R, L = 1000.0, [0.0, 0.13, 0.13, 0.5, 0.71], 1000, 5, 3, 3000
    sig = rng.standard_normal(n).astype(np.float32)
    rir = rng.standard_normal((P, R, L)).astype(np.float32)
    G = rng.standard_normal((n + L - 1, R))

    def grads(g):
        ts = torch.from_numpy(sig).cuda().requires_grad_(True)
        tr = torch.from_numpy(rir).cuda().requires_grad_(True)
        simulate_trajectory_torch(ts, tr, stamps, fs).backward(torch.from_numpy(g).cuda())
        return ts.grad.cpu().numpy(), tr.grad.cpu().numpy()

    s, r = grads(G)
    # (the oracle's correlations take no empty segment: it runs without that point, whose RIR
    # gradient is zero)
    full = [0, 2, 3, 4]
    gs, gr4 = oracle.trajectory_adjoint(sig, rir[full], G, [stamps[k] for k in full], fs)
    gr = np.zeros(rir.shape)
    gr[full] = gr4
    assert rel_l2(s, gs) < 2e-6 and rel_l2(r, gr) < 2e-6
    bad = G.copy()
    bad[700, 1] = np.nan
    _, r2 = grads(bad)
    assert np.array_equal(r2[:, 0], r[:, 0]) and np.array_equal(r2[:, 2], r[:, 2])
    assert np.isnan(r2[:, 1]).any()
