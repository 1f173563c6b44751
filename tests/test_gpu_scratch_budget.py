"""The scratch budget of a plan holds for prepared shots whatever tile the
autotuner picks: shots are batched so that the largest variant's lists fit."""
import numpy as np
import pytest

import kirch_datuming_b200 as kd

pytestmark = pytest.mark.gpu


def test_autotuned_shots_stay_within_scratch():
    import torch
    ns = nh = 768
    nz = nx = nt = 101
    f = lambda v: float(np.float32(v))  # noqa: E731
    d = 0.01
    npos = 26
    z = torch.arange(nz, device="cuda", dtype=torch.float64)[None, :] * d
    x = torch.arange(nx, device="cuda", dtype=torch.float64)[:, None] * d
    T = torch.stack([(torch.sqrt((x - 0.04 * k) ** 2 + z * z) / 2.0).float() for k in range(npos)])
    D = torch.zeros_like(T)
    geom = kd.geometry(nt=nt, nh=1, ns=1, t0=0.0, dt=f(0.01), h0=0.0, dh=0.0, s0=0.0, ds=0.0, nz=nz, nx=nx, z0=0.0, dz=f(d),
                       x0=0.0, dx=f(d), sny=npos, sy0=0.0, sdy=f(0.04), rny=npos, ry0=0.0, rdy=f(0.04))
    kp = kd.params("cig=0", "cmp=0", "type=linear")
    data = torch.randn((ns, nh, nt), generator=torch.Generator(device="cuda").manual_seed(1), device="cuda")
    shots = [dict(sx=f(1.0 * k / ns), h0=0.0, dh=f(1.0 / nh), data=data[k]) for k in range(ns)]
    # what the shots need in one batch with tiles of 128 points, to a megabyte: 64-point tiles take 90 MB more
    tiles = -(-nz // 16) * -(-nx // 8)
    lists = tiles * ((ns + nh) * 16 + ns // 2 * (4 + 4 * nh))
    budget = (ns + nh) * 24 * nz * nx + ns * nh * (16 * nt + 48) + lists + (1 << 20)
    warm = kd.Plan(kp, geom, 64 << 20)  # loads the kernels
    warm.set_tables(T, D, T, D)
    img = torch.zeros((1, nx, nz), device="cuda")
    warm.prepare_shots(shots[:4])
    warm.autotune()
    warm.migrate_prepared(img)
    warm.close()
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    plan = kd.Plan(kp, geom, budget)
    plan.set_tables(T, D, T, D)
    plan.prepare_shots(shots)
    plan.autotune()
    plan.migrate_prepared(img)
    held = free - torch.cuda.mem_get_info()[0]
    plan.close()
    # the shots' samples beside the scratch; 2 MB of rounding for each of its dozen buffers
    assert held <= data.numel() * 4 + budget + (28 << 20), (held - data.numel() * 4 - budget) >> 20
    assert img.norm() > 0
