"""The walks of the summation -- every receiver, or lists of the pairs that may
reach a tile, each whole or in parts -- as a sample of the survey's pairs picks
them: short records and narrow angle axes leave most pairs out (lists), long
ones few (every receiver).  Surveys large enough to be sampled (24e6 pairs x
points), with and without parts (shots up to and beyond 64 blocks), receivers
shared, of their own and ragged; launches tell which walk ran, and the image is
held against the FP64 oracle (1e-5, as the other migrations)."""
import numpy as np
import pytest

import _cases
import kirch_datuming_b200 as kd
import oracle

pytestmark = pytest.mark.gpu

A = ["cig=1", "mode=angle"]
PARTS, WHOLE = (90, 97), (310, 26)


def _geometry(golden, cmp, ns, nh, nt):
    g = golden.geometry_dict("base")
    g.update(nt=nt, ns=ns, nh=nh, ds=float(np.float32(1.6 / ns)), s0=float(np.float32(0.013)),
             dh=float(np.float32((0.6 if cmp else 1.5) / nh)), h0=float(np.float32(-0.3 if cmp else 0.05)))
    assert ns * nh * g["nz"] * g["nx"] >= 24e6
    return g


def _run(golden, tokens, cmp, ns, nh, nt, dt=None):
    import torch
    geom = _geometry(golden, cmp, ns, nh, nt)
    if dt:
        geom["dt"] = float(np.float32(dt))
    kp = kd.params("adj=1", "cmp=%d" % cmp, *tokens)
    axis = kd.output_axis(kp, kd.geometry(**geom))
    T, D = golden.tables()
    data = np.random.default_rng(nh).standard_normal((ns, nh, nt)).astype(np.float32)
    dT, dD = torch.from_numpy(T).cuda(), torch.from_numpy(D).cuda()
    plan = kd.Plan(kp, kd.geometry(**geom))
    plan.set_tables(dT, dD, dT, dD)
    img = torch.full((axis[0], geom["nx"], geom["nz"]), 5.0, dtype=torch.float32, device="cuda")
    plan.migrate(torch.from_numpy(data).cuda(), img)
    launches = plan.stats()["launches"]
    plan.close()
    ref = oracle.migrate_adj(_cases.oracle_params(kp, geom, axis), data, T, D, T, D, fp64=True)
    assert np.linalg.norm(ref) > 0
    return oracle.rel_l2(img.cpu().numpy(), ref), launches


@pytest.mark.parametrize("ns,nh", [PARTS, WHOLE])
@pytest.mark.parametrize("cmp", [0, 1])
@pytest.mark.parametrize("tokens", [
    A + ["angle_min=0", "angle_max=180", "angle_n=181"], A + ["angle_max=60", "angle_n=31", "angle_interp=0"],
    ["cig=0"], ["cig=1", "mode=offset"]])
def test_short_and_long_records(golden, tokens, cmp, ns, nh):
    launches = {}
    for nt, dt in ((40, 0.002), (301, 0.02)):  # 0.08 s: few pairs end within it; 6 s: all do
        err, launches[nt] = _run(golden, tokens, cmp, ns, nh, nt, dt)
        assert err <= 1e-5, (nt, err)
    narrow = "angle_max=60" in tokens  # the axis alone may leave enough pairs out
    assert launches[40] - launches[301] in ((0, 2) if narrow else (2,)), launches


@pytest.mark.parametrize("ns,nh", [PARTS, WHOLE])
@pytest.mark.parametrize("tokens,cmp,nt", [
    (A + ["angle_min=20", "angle_max=30", "angle_n=11"], 0, 201),
    (A + ["angle_min=5", "angle_max=9", "angle_step=0.01", "angle_n=401"], 0, 201),
    (A + ["angle_min=0", "angle_max=12", "angle_n=13", "half_angle=1"], 1, 150),
    (A + ["angle_min=0", "angle_max=60", "angle_n=61", "aperture=20", "aperture_taper=4"], 1, 201),
    (A + ["angle_min=0", "angle_max=60", "angle_n=61", "aperture_trace=4", "aperture_trace_taper=2"], 0, 201)])
def test_few_pairs_contribute(golden, tokens, cmp, nt, ns, nh):
    err, _ = _run(golden, tokens, cmp, ns, nh, nt)
    assert err <= 1e-5, err


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("count,nhmax", [(90, 180), (200, 80)])
def test_ragged_shots(golden, count, nhmax, graph):
    import torch
    geom = golden.geometry_dict("base")
    geom.update(nt=301, nh=1, ns=1, ds=0.0, dh=float(np.float32(0.02)), h0=0.0, s0=0.0)
    T, D = golden.tables()
    dT, dD = torch.from_numpy(T).cuda(), torch.from_numpy(D).cuda()
    launches = []
    for nt, ang in ((60, 40), (301, 180)):
        kp = kd.params("adj=1", "cmp=0", *A, "angle_min=0", "angle_max=%d" % ang, "angle_n=%d" % (ang + 1))
        g = dict(geom, dt=float(np.float32(0.002 if nt == 60 else 0.02)))
        axis = kd.output_axis(kp, kd.geometry(**g))
        rng = np.random.default_rng(count)
        shots, ref, pairs = [], 0.0, 0
        for k in range(count):
            nh, n = int(rng.integers(nhmax // 2, nhmax)), int(rng.integers(nt // 2, nt + 1))
            sx, h0 = float(np.float32(1.5 * k / count + 0.03)), float(np.float32(0.001 * rng.integers(0, 20)))
            dh = float(np.float32(1.5 / nhmax))
            x = rng.standard_normal((nh, n)).astype(np.float32)
            shots.append(dict(sx=sx, h0=h0, dh=dh, data=x))
            pairs += nh
            op = _cases.oracle_params(kp, dict(g, nt=n, nh=nh, h0=h0, dh=dh, s0=sx), axis)
            ref = ref + oracle.migrate_adj(op, x[None], T, D, T, D, fp64=True)
        assert pairs * g["nz"] * g["nx"] >= 24e6
        plan = kd.Plan(kp, kd.geometry(**g))
        plan.set_tables(dT, dD, dT, dD)
        plan.prepare_shots(shots)
        img = torch.zeros((axis[0], g["nx"], g["nz"]), dtype=torch.float32, device="cuda")
        if graph:
            plan.set_graph(True)
            plan.migrate_prepared(img)  # direct run, then the capture keeps its walk
            img.fill_(2.0)
        plan.migrate_prepared(img)
        launches.append(plan.stats()["launches"])
        plan.close()
        assert np.linalg.norm(ref) > 0
        assert oracle.rel_l2(img.cpu().numpy(), ref) <= 1e-5
    if not graph:
        assert launches[0] - launches[1] == 2, launches


def test_many_plans_at_once(golden):
    """More plans alive than the library has slots for their samples."""
    import torch
    geom = _geometry(golden, 0, *PARTS, 40)
    kp = kd.params("adj=1", "cmp=0", *A, "angle_max=60", "angle_n=31")
    ng = kd.output_axis(kp, kd.geometry(**geom))[0]
    dT, dD = (torch.from_numpy(a).cuda() for a in golden.tables())
    data = torch.randn((PARTS[0], PARTS[1], 40), generator=torch.Generator(device="cuda").manual_seed(1), device="cuda")
    plans, want = [], None
    for rounds in range(2):
        for k in range(70):
            plan = kd.Plan(kp, kd.geometry(**geom))
            plan.set_tables(dT, dD, dT, dD)
            img = torch.full((ng, geom["nx"], geom["nz"]), 5.0, device="cuda")
            plan.migrate(data, img)
            want = img.clone() if want is None else want
            assert torch.equal(img, want)
            plans.append(plan)
        for plan in plans[::2] + plans[1::2]:
            plan.close()
        plans = []
    assert want.norm() > 0
