"""The lists of pairs that may reach a tile (k_leg_bounds, k_cull) where they
leave most pairs out: short records, narrow or offset angle axes, fine bins,
tight apertures, receiver counts around the warp's 32 and shot counts around
the blocks' 4 and 2, ragged shots.  A pair dropped by mistake shows against
the FP64 oracle (1e-5, as the other migrations)."""
import numpy as np
import pytest

import _cases
import kirch_datuming_b200 as kd
import oracle

pytestmark = pytest.mark.gpu

A = ["cig=1", "mode=angle"]


@pytest.mark.parametrize("tokens,cmp,ns,nh,nt", [
    (A + ["angle_min=0", "angle_max=60", "angle_n=61"], 0, 5, 33, 121),
    (A + ["angle_min=20", "angle_max=30", "angle_n=11"], 0, 7, 31, 301),
    (A + ["angle_min=5", "angle_max=9", "angle_step=0.01", "angle_n=401"], 0, 4, 40, 301),
    (A + ["angle_min=30", "angle_max=60", "angle_step=2", "angle_n=16", "angle_interp=0"], 0, 9, 64, 200),
    (A + ["angle_min=0", "angle_max=12", "angle_n=13", "half_angle=1"], 1, 5, 33, 150),
    (A + ["angle_min=0", "angle_max=60", "angle_n=61", "aperture=20", "aperture_taper=4"], 1, 6, 21, 301),
    (A + ["angle_min=0", "angle_max=60", "angle_n=61", "aperture_trace=4", "aperture_trace_taper=0"], 0, 6, 35, 301),
    (["cig=0", "aperture=15", "aperture_taper=0"], 0, 3, 32, 90), (["cig=1", "mode=offset", "tau=-0.05"], 0, 3, 9, 160)])
def test_regular_cube_vs_oracle(golden, tokens, cmp, ns, nh, nt):
    import torch
    geom = golden.geometry_dict("base")
    geom.update(nt=nt, ns=ns, nh=nh, ds=float(np.float32(0.09)), s0=float(np.float32(0.1)), dh=float(np.float32(0.02)),
                h0=float(np.float32(-0.3 if cmp else 0.05)))
    kp = kd.params("adj=1", "cmp=%d" % cmp, *tokens)
    axis = kd.output_axis(kp, kd.geometry(**geom))
    op = _cases.oracle_params(kp, geom, axis)
    T, D = golden.tables()
    data = np.random.default_rng(nh).standard_normal((ns, nh, nt)).astype(np.float32)
    dT, dD = torch.from_numpy(T).cuda(), torch.from_numpy(D).cuda()
    plan = kd.Plan(kp, kd.geometry(**geom))
    plan.set_tables(dT, dD, dT, dD)
    img = torch.zeros((axis[0], geom["nx"], geom["nz"]), dtype=torch.float32, device="cuda")
    plan.migrate(torch.from_numpy(data).cuda(), img)
    plan.close()
    ref = oracle.migrate_adj(op, data, T, D, T, D, fp64=True)
    assert np.linalg.norm(ref) > 0
    assert oracle.rel_l2(img.cpu().numpy(), ref) <= 1e-5


def test_ragged_shots_every_tile_variant(golden):
    """Each autotuned tile shape with its own lists gives the sum of the one-shot images."""
    import torch
    geom = golden.geometry_dict("base")
    geom.update(nt=301, nh=1, ns=1, ds=0.0, dh=float(np.float32(0.02)), h0=0.0, s0=0.0)
    kp = kd.params("adj=1", "cmp=0", *A, "angle_min=0", "angle_max=40", "angle_n=41")
    axis = kd.output_axis(kp, kd.geometry(**geom))
    T, D = golden.tables()
    rng = np.random.default_rng(2)
    shots, ref = [], 0.0
    for k in range(7):
        nh, nt, sx = int(rng.integers(1, 50)), int(rng.integers(60, 302)), float(np.float32(0.1 * k + 0.05))
        h0 = float(np.float32(0.02 * rng.integers(0, 10)))
        x = rng.standard_normal((nh, nt)).astype(np.float32)
        shots.append(dict(sx=sx, h0=h0, dh=geom["dh"], data=x))
        op = _cases.oracle_params(kp, dict(geom, nt=nt, nh=nh, h0=h0, s0=sx), axis)
        ref = ref + oracle.migrate_adj(op, x[None], T, D, T, D, fp64=True)
    plan = kd.Plan(kp, kd.geometry(**geom))
    dT, dD = torch.from_numpy(T).cuda(), torch.from_numpy(D).cuda()
    plan.set_tables(dT, dD, dT, dD)
    img = torch.zeros((axis[0], geom["nx"], geom["nz"]), dtype=torch.float32, device="cuda")
    for tuned in (False, True):
        plan.prepare_shots(shots)
        if tuned:
            plan.autotune()
        plan.migrate_prepared(img.zero_())
        assert oracle.rel_l2(img.cpu().numpy(), ref) <= 1e-5
    plan.close()
