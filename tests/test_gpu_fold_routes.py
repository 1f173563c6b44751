"""Routes of a survey's migration that share work between its sides, where the
fields come from elsewhere than device tables: reciprocal traces migrated once
with a surrogate and with streamed tables, and the map of needed blocks against
the FP64 oracle."""
import numpy as np
import pytest

import _cases
import kirch_datuming_b200 as kd
import oracle

pytestmark = pytest.mark.gpu

ANGLE = ["cig=1", "mode=angle", "angle_min=0", "angle_max=60", "angle_step=1", "angle_n=61"]


def _survey(golden, ns, nh, off):
    geom = golden.geometry_dict("base")
    d = float(np.float32(0.03125))  # station positions exact in float
    geom.update(nt=golden.meta["nt"], ns=ns, nh=nh, ds=d, dh=d, h0=4 * d, s0=(4 + off) * d)
    data = np.random.default_rng(ns).standard_normal((ns, nh, geom["nt"])).astype(np.float32)
    return geom, data


@pytest.mark.parametrize("angle", ["network", "fd"])
@pytest.mark.parametrize("ns,nh,off", [(13, 17, 2), (9, 12, -3), (16, 16, 0)])
def test_fold_with_surrogate(golden, ns, nh, off, angle):
    """One surrogate for both sides (folded) against two equal ones (not)."""
    import torch
    geom, data = _survey(golden, ns, nh, off)
    kp = kd.params("adj=1", "cmp=0", *ANGLE)
    dev = torch.from_numpy(data).cuda()
    nets = [kd.Surrogate((0.0, 0.0, 0.0), (2.0, 1.0, 2.0), fmax=6.0, vref=1.8, zsrc=0.0, seed=5) for _ in range(2)]
    images = []
    for rcv in nets:
        plan = kd.Plan(kp, kd.geometry(**geom))
        T, D = (torch.from_numpy(a).cuda() for a in golden.tables())
        plan.set_tables(T, D, T, D)
        plan.set_surrogate(nets[0], rcv, angle=angle)
        img = torch.full((61, geom["nx"], geom["nz"]), 7.0, device="cuda")
        plan.migrate(dev, img)
        plan.close()
        images.append(img.double())
    for n in nets:
        n.close()
    assert images[1].norm() > 0
    assert (images[0] - images[1]).norm() <= 1e-6 * images[1].norm()


@pytest.mark.parametrize("ns,nh,off", [(13, 17, 2), (9, 12, -3), (16, 16, 0)])
def test_fold_with_streamed_tables(golden, ns, nh, off):
    """Tables in host memory (folded) against the FP64 oracle and, bit for bit, device tables."""
    geom, data = _survey(golden, ns, nh, off)
    kp = kd.params("adj=1", "cmp=0", *ANGLE)
    axis = kd.output_axis(kp, kd.geometry(**geom))
    T, D = golden.tables()
    images = []
    for stream in (True, False):
        plan = kd.Plan(kp, kd.geometry(**geom))
        plan.set_tables(T, D, T, D, stream=stream)
        img = np.full((61, geom["nx"], geom["nz"]), 7.0, np.float32)
        plan.migrate(data, img)
        plan.close()
        images.append(img)
    ref = oracle.migrate_adj(_cases.oracle_params(kp, geom, axis), data, T, D, T, D, fp64=True)
    assert oracle.rel_l2(images[0], ref) <= 1e-5
    np.testing.assert_array_equal(images[0], images[1])


@pytest.mark.parametrize("s0,ds", [(4.0, 0.5), (4.1, 0.25)])
def test_needed_blocks_vs_oracle(s0, ds):
    """A survey much longer than its records reach, on and off the receivers."""
    import torch
    nz, nx, nt, ns, nh, npos, d = 601, 1201, 151, 2, 48, 49, 0.01
    f = lambda v: float(np.float32(v))  # noqa: E731
    z, x = np.arange(nz)[None, :] * d, np.arange(nx)[:, None] * d
    T, D = np.empty((npos, nx, nz), np.float32), np.empty((npos, nx, nz), np.float32)
    for k in range(npos):
        r = np.sqrt((x - 0.25 * k) ** 2 + z * z)
        T[k] = r / (2.0 + 0.2 * z)
        D[k] = -(x - 0.25 * k) / np.maximum(r, 1e-9) / (2.0 + 0.2 * z)
    geom = dict(nt=nt, nh=nh, ns=ns, t0=0.0, dt=f(0.008), h0=0.0, dh=f(0.25), s0=f(s0), ds=f(ds), nz=nz, nx=nx, z0=0.0, dz=f(d),
                x0=0.0, dx=f(d), sny=npos, sy0=0.0, sdy=f(0.25), rny=npos, ry0=0.0, rdy=f(0.25))
    assert (ns + nh) * nz * nx >= 32 << 20  # mapped
    kp = kd.params("adj=1", "cmp=0", "cig=1", "mode=angle", "angle_max=60", "angle_n=13", "angle_step=5", "type=linear")
    axis = kd.output_axis(kp, kd.geometry(**geom))
    data = np.random.default_rng(3).standard_normal((ns, nh, nt)).astype(np.float32)
    plan = kd.Plan(kp, kd.geometry(**geom), 24 << 30)
    dT, dD = torch.from_numpy(T).cuda(), torch.from_numpy(D).cuda()
    plan.set_tables(dT, dD, dT, dD)
    img = torch.full((axis[0], nx, nz), 7.0, device="cuda")
    for _ in range(2):  # the second run finds the first one's fields in the left-out blocks
        plan.migrate(torch.from_numpy(data).cuda(), img)
    plan.close()
    ref = oracle.migrate_adj(_cases.oracle_params(kp, geom, axis), data, T, D, T, D, fp64=True)
    assert np.linalg.norm(ref) > 0
    assert oracle.rel_l2(img.cpu().numpy(), ref) <= 1e-5
