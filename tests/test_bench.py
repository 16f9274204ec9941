"""CPU tests of the benchmark's bookkeeping."""
import os
import sys

import numpy as np

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)
import bench  # noqa: E402


def test_phase_figures_count_real_frames_only():
    """The products, sums and sweeps of a ragged fraction leave padding frames out: its phases are credited with the work of the real
    frames, the same as an unpadded fraction of as many frames and sequences."""
    layers = [dict(type="input", size=10), dict(type="feedforward_tanh", size=16), dict(type="blstm", size=32), dict(type="lstm", size=8),
              dict(type="sse", size=8)]
    ragged, even = np.array([100, 60, 20, 20], np.int32), np.array([50] * 4, np.int32)
    work = bench.phase_work(layers, ragged)
    assert work == bench.phase_work(layers, even)
    assert work["lstm_proj_gemm"] == ("flops", 8.0 * 200 * (32 * 16 + 8 * 32))
    assert work["lstm_dw_rec_gemm"] == ("flops", 8.0 * 196 * (32 * 16 + 8 * 8))
    assert work["lstm_vector_grads"] == ("bytes", 20.0 * 200 * 40)
