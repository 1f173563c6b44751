"""One plan taken through different kinds of migration: what an earlier call
left in it (the needed-blocks map of its legs) must not reach a later one."""
import numpy as np
import pytest

import kirch_datuming_b200 as kd

pytestmark = pytest.mark.gpu


def _line(nz, nx, npos, step):
    """Straight-ray tables of v = 2 + 0.2 z at stations 0, step, ..."""
    import torch
    d = 0.01
    z = torch.arange(nz, device="cuda", dtype=torch.float64)[None, :] * d
    x = torch.arange(nx, device="cuda", dtype=torch.float64)[:, None] * d
    T = torch.empty((npos, nx, nz), device="cuda")
    D = torch.empty_like(T)
    for k in range(npos):
        r = torch.sqrt((x - step * k) ** 2 + z * z)
        T[k] = (r / (2.0 + 0.2 * z)).float()
        D[k] = (-(x - step * k) / r.clamp(min=1e-9) / (2.0 + 0.2 * z)).float()
    return T, D


@pytest.mark.parametrize("ds", [0.25, 0.125])
def test_surrogate_after_tables(ds):
    """Tables on a survey longer than its records reach (blocks of points that
    no pair reaches are left out), then a surrogate of a faster medium on the
    same plan: the image of a plan that never saw the tables' map, bit for bit,
    with the shots on the receivers (0.25) and between them (0.125)."""
    import torch
    nz, nx, nt, ns, nh, npos = 601, 1201, 401, 40, 48, 49
    T, D = _line(nz, nx, npos, 0.25)
    f = lambda v: float(np.float32(v))  # noqa: E731
    geom = kd.geometry(nt=nt, nh=nh, ns=ns, t0=0.0, dt=f(0.004), h0=0.0, dh=f(0.25), s0=f(0.0625 if ds < 0.2 else 0.5),
                       ds=f(ds), nz=nz, nx=nx, z0=0.0, dz=f(0.01), x0=0.0, dx=f(0.01), sny=npos, sy0=0.0, sdy=f(0.25),
                       rny=npos, ry0=0.0, rdy=f(0.25))
    kp = kd.params("cig=1", "mode=angle", "cmp=0", "angle_max=60", "angle_n=61")
    data = torch.randn((ns, nh, nt), generator=torch.Generator(device="cuda").manual_seed(4), device="cuda")
    net = kd.Surrogate((0.0, 0.0, 0.0), (12.0, 6.0, 12.0), fmax=2.0, vref=4.0, zsrc=0.0, seed=3)
    images = []
    for tables_first in (True, False):
        plan = kd.Plan(kp, geom, 24 << 30)
        plan.set_tables(T, D, T, D)
        img = torch.full((plan.ng, nx, nz), 7.0, device="cuda")
        if tables_first:
            plan.migrate(data, img)
        plan.set_surrogate(net, net, angle="network")
        plan.migrate(data, img)
        plan.close()
        images.append(img)
    net.close()
    assert images[1].norm() > 0
    assert torch.equal(images[0], images[1])


@pytest.mark.parametrize("own", [False, True])
def test_graph_keeps_its_scratch(golden, own):
    """A graph over prepared shots (kcig_graph, or the plan's own) replays the
    same image after calls that need more scratch than the shots did: the
    autotuner's larger lists, a migration and a modelling of the whole cube.
    What they free, if anything, is overwritten before the replay."""
    import torch
    import _cases
    kp, geom, axis, _, _ = _cases.case_setup(golden, "base")
    kp.direct_mute = 0  # kcig_model takes none
    tT, tD = (torch.from_numpy(a).cuda() for a in golden.tables())
    cube = torch.from_numpy(golden.data("base")).cuda()
    ns, nh, nt = cube.shape
    dh = float(np.float32(geom["dh"]))
    shot = dict(sx=float(np.float32(geom["s0"])), h0=float(np.float32(geom["h0"])), dh=dh, data=cube[0, :5].contiguous())
    plan = kd.Plan(kp, kd.geometry(**geom))
    plan.set_tables(tT, tD, tT, tD)
    plan.prepare_shots([shot])
    img, other, data = (torch.zeros(s, device="cuda") for s in ((axis[0], geom["nx"], geom["nz"]),) * 2 + (cube.shape,))
    if own:
        plan.set_graph(True)
        plan.migrate_prepared(img)
    else:
        graph = kd.Graph([plan], [img])
    replay = (lambda: plan.migrate_prepared(img)) if own else graph.launch
    replay()
    torch.cuda.synchronize()
    want = img.clone()
    assert want.norm() > 0
    steps = [lambda: plan.migrate(cube, other), lambda: plan.model(want, data)]
    if not own:  # the autotuner drops the plan's own graph
        steps.insert(0, plan.autotune)
    for step in steps:
        step()
        waste = [torch.full((n << 18,), float("nan"), device="cuda") for n in (1, 2, 4, 8, 16, 32, 64)]
        torch.cuda.synchronize()
        img.fill_(3.0)
        replay()
        torch.cuda.synchronize()
        assert torch.equal(img, want)
        del waste
        torch.cuda.empty_cache()
    if not own:
        graph.close()
    plan.close()
