"""The diagonal-layout sweeps of kcig_eikods at the edges of their rows (16
entries), warps (32 rows), skipping blocks (16 diagonals) and unskew windows,
with more sources than resident blocks, and on grids longer than 1024 blocks
of 16: equal to the sweep oracle, bit for bit."""
import os
import sys

import numpy as np
import pytest

import kirch_datuming_b200 as kd

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.join(os.path.dirname(HERE), "oracle"))
import oracle as O  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nz,nx,order,nshot", [
    (3, 3, 2, 2), (13, 40, 2, 2), (14, 5, 1, 2), (15, 33, 2, 2), (31, 16, 2, 2), (32, 17, 1, 2), (33, 64, 2, 2),
    (62, 15, 2, 2), (640, 40, 2, 1), (641, 33, 2, 1), (20, 24, 2, 700), (4, 17000, 1, 1)])
def test_layout_edges(nz, nx, order, nshot):
    import torch
    rng = np.random.default_rng(nz * nx)
    d = 0.01
    v = (1.5 + np.linspace(0, 1.5, nz)[None, :] + 0.6 * rng.random((nx, nz))).astype(np.float32)
    shots = np.zeros((nshot, 3), np.float32)
    shots[:, 0] = rng.uniform(0, (nz - 1) * d, nshot) * (np.arange(nshot) % 2)
    shots[:, 1] = rng.uniform(0, (nx - 1) * d, nshot)
    got = kd.eikods(torch.from_numpy(v).cuda(), d, d, shots, order=order, grads=True)
    ref = O.eikods(v, d, d, shots, method=1, grads=True, order=order)
    np.testing.assert_array_equal(got["sweeps"], ref["sweeps"])
    for k in ("time", "tdl1", "tds1", "gradz", "gradx"):
        np.testing.assert_array_equal(got[k].cpu().numpy(), ref[k], err_msg=k)
    only = kd.eikods(torch.from_numpy(v).cuda(), d, d, shots, order=order, derivs=False)
    assert torch.equal(only["time"], got["time"])
