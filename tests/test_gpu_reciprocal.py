"""Surveys that shoot from their own stations (cmp=0, shots on receivers):
reciprocal traces are added and migrated once, and the shots' leg fields are
the receivers'.  Against the FP64 oracle (1e-5, as the other migrations) at
shot counts around the groups of four, shots before, on and past the spread,
weights that are and are not reciprocal, small scratch and shot ranges."""
import numpy as np
import pytest

import _cases
import kirch_datuming_b200 as kd
import oracle

pytestmark = pytest.mark.gpu

TAIL = ["direct_mute=1", "direct_mute_slope=0.5", "direct_mute_intercept=0", "direct_mute_taper=0.05"]
ANGLE = ["cig=1", "mode=angle", "angle_min=0", "angle_max=60", "angle_step=1", "angle_n=61"]


def _run(golden, tokens, ns, nh, off, scratch=0, first=0, count=-1):
    import torch
    geom = golden.geometry_dict("base")
    d = float(np.float32(0.03125))  # station positions exact in float
    geom.update(nt=golden.meta["nt"], ns=ns, nh=nh, ds=d, dh=d, h0=4 * d, s0=(4 + off) * d)
    kp = kd.params("adj=1", "cmp=0", *tokens)
    axis = kd.output_axis(kp, kd.geometry(**geom))
    op = _cases.oracle_params(kp, geom, axis)
    T, D = golden.tables()
    rng = np.random.default_rng(ns * 100 + nh + off)
    data = np.cumsum(rng.standard_normal((ns, nh, geom["nt"])), axis=2).astype(np.float32) * 0.1
    plan = kd.Plan(kp, kd.geometry(**geom), scratch)
    dT, dD = torch.from_numpy(T).cuda(), torch.from_numpy(D).cuda()
    plan.set_tables(dT, dD, dT, dD)
    plan.set_shot_range(first, count)
    img = torch.zeros((axis[0], geom["nx"], geom["nz"]), dtype=torch.float32, device="cuda")
    sub = data if count < 0 else data[first:first + count]
    plan.migrate(torch.from_numpy(np.ascontiguousarray(sub)).cuda(), img)
    launches = plan.stats()["launches"]
    plan.close()
    ref_data = data.copy()
    if count >= 0:
        ref_data[:first] = 0
        ref_data[first + count:] = 0
    ref = oracle.migrate_adj(op, ref_data, T, D, T, D, fp64=True)
    assert np.linalg.norm(ref) > 0
    return oracle.rel_l2(img.cpu().numpy(), ref), launches


@pytest.mark.parametrize("ns,nh,off", [(8, 8, 0), (9, 9, 0), (11, 14, 2), (16, 12, 0), (14, 12, -3), (13, 21, 8), (5, 7, 1), (4, 4, 0), (17, 6, -4)])
def test_shots_on_receivers(golden, ns, nh, off):
    err, _ = _run(golden, ANGLE + TAIL, ns, nh, off)
    assert err <= 1e-5, err


@pytest.mark.parametrize("tokens", [
    ["cig=0"] + TAIL, ["cig=1", "mode=offset"] + TAIL, ANGLE + ["angle_interp=0", "diff=1", "type=linear", "antialias=0.5"],
    ANGLE + ["half_angle=1", "aperture=50", "aperture_taper=10"], ANGLE + TAIL + ["aperture_trace=9", "aperture_trace_taper=5"]])
def test_options(golden, tokens):
    err, _ = _run(golden, tokens, 13, 17, 2)
    assert err <= 1e-5, err


@pytest.mark.parametrize("scratch", [1 << 20, 3 << 20, 6 << 20])
def test_small_scratch(golden, scratch):
    err, _ = _run(golden, ANGLE + TAIL, 18, 20, 1, scratch=scratch)
    assert err <= 1e-5, err


def test_shot_range(golden):
    for first, count in ((0, 7), (7, 10), (17, 1)):
        err, _ = _run(golden, ANGLE + TAIL, 18, 20, 1, first=first, count=count)
        assert err <= 1e-5, (first, count, err)
