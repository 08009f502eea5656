"""The cases that the autotuner times have to reach the kernels whose shape they choose."""
import os
import re

from gpurir_gb300 import tune

CSRC = os.path.join(os.path.dirname(os.path.abspath(tune.__file__)), "csrc")


def test_trajectory_adjoint_case_takes_whole_rows():
    """Segments up to kBlkMaxSeg take the adjoint in blocks of lags, which the knob does not change."""
    text = open(os.path.join(CSRC, "conv.cu")).read()
    longest = int(re.search(r"constexpr int kBlkMaxSeg = (\d+);", text).group(1))
    points, receivers, rir_len, segment = tune.TRAJ_ADJOINT
    assert longest < segment and segment + rir_len - 1 <= 16384   # (its FFT's longest problem)
