"""Traveltime tables on grids of unequal spacings (each axis' reciprocals told
apart) and around a point that no front reaches (negative squared slowness:
its time stays FLT_MAX, whose difference over a squared spacing below 1
overflows): equal to the sweep oracle, bit for bit."""
import os
import sys

import numpy as np
import pytest

import kirch_datuming_b200 as kd

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.join(os.path.dirname(HERE), "oracle"))
import oracle as O  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hole", [False, True])
@pytest.mark.parametrize("dz,dx,order,l", [(0.5, 0.7, 2, 1), (0.7, 0.5, 1, 0), (0.01, 0.03, 2, 1), (12.5, 5.0, 2, 0), (3.0, 8.0, 1, 1)])
def test_spacings_equal_oracle(dz, dx, order, l, hole):
    import torch
    nz, nx = 37, 53
    rng = np.random.default_rng(int(100 * dz) + order)
    dz, dx = float(np.float32(dz)), float(np.float32(dx))
    s2 = (0.04 * (1 + 0.3 * rng.random((nx, nz)))).astype(np.float32)
    if hole:
        if min(dz, dx) < 0.4:
            pytest.skip("the slope times FLT_MAX overflows too: no fixed point, here and in the oracle")
        s2[30, 20] = -1e-4
    shots = np.zeros((3, 3), np.float32)
    shots[:, 1] = np.float32(dx) * np.float32([3.0, 25.3, 50.0])
    shots[1, 0] = np.float32(dz) * np.float32(7.6)
    got = kd.eikods(torch.from_numpy(s2).cuda(), dz, dx, shots, order=order, l=l, vel_is_slowness2=True, grads=True)
    ref = O.eikods(s2, dz, dx, shots, method=1, grads=True, order=order, l=l, vel_is_s2=True)
    assert (ref["time"] == np.finfo(np.float32).max).sum() == (3 if hole else 0)
    np.testing.assert_array_equal(got["sweeps"], ref["sweeps"])
    for k in ("time", "tdl1", "tds1", "gradz", "gradx"):
        np.testing.assert_array_equal(got[k].cpu().numpy(), ref[k], err_msg=k)
