"""Leg fields only where a pair may end within the record: a survey much longer
than its records reach, migrated with one set of tables for both sides (the
blocks of points that no pair reaches are left out, and reciprocal traces
folded where the shots stand on receivers) against the same survey with a copy
of the tables for the receivers, which takes the general path (every block, no
folding).  The same pairs in FP32 sums of another grouping: 1e-6."""
import numpy as np
import pytest

import kirch_datuming_b200 as kd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nz,nx,nt,t0,tau,ds,interp", [
    (601, 1201, 401, 0.0, 0.0, 0.25, "h"), (601, 1201, 401, 0.0, 0.0, 0.125, "h"), (577, 1250, 301, 0.1, -0.05, 0.2, "l"),
    (601, 1201, 3, 0.0, 0.0, 0.25, "h")])
def test_survey_longer_than_its_records(nz, nx, nt, t0, tau, ds, interp):
    import torch
    d, ns, nh, npos = 0.01, 46, 48, 49
    z = torch.arange(nz, device="cuda", dtype=torch.float64)[None, :] * d
    x = torch.arange(nx, device="cuda", dtype=torch.float64)[:, None] * d
    T = torch.empty((npos, nx, nz), device="cuda")
    D = torch.empty_like(T)
    for k in range(npos):
        r = torch.sqrt((x - 0.25 * k) ** 2 + z * z)
        T[k] = (r / (2.0 + 0.2 * z)).float()
        D[k] = (-(x - 0.25 * k) / r.clamp(min=1e-9) / (2.0 + 0.2 * z)).float()
    f = lambda v: float(np.float32(v))  # noqa: E731
    geom = kd.geometry(nt=nt, nh=nh, ns=ns, t0=f(t0), dt=f(0.004), h0=0.0, dh=f(0.25), s0=f(ds * 2), ds=f(ds), nz=nz, nx=nx,
                       z0=0.0, dz=f(d), x0=0.0, dx=f(d), sny=npos, sy0=0.0, sdy=f(0.25), rny=npos, ry0=0.0, rdy=f(0.25))
    kp = kd.params("cig=1", "mode=angle", "cmp=0", "angle_max=60", "angle_n=61", "type=%s" % interp, "tau=%g" % tau)
    g = torch.Generator(device="cuda").manual_seed(nt)
    data = torch.randn((ns, nh, nt), generator=g, device="cuda")
    images = []
    for rT, rD in ((T, D), (T.clone(), D.clone())):
        plan = kd.Plan(kp, geom, 24 << 30)
        plan.set_tables(T, D, rT, rD)
        img = torch.full((plan.ng, nx, nz), 7.0, device="cuda")
        for _ in range(2):  # the second run finds the first one's fields in the left-out blocks
            plan.migrate(data, img)
        plan.close()
        images.append(img.double())
    a, b = images
    assert nt < 10 or b.norm() > 0
    assert (a - b).norm() <= 1e-6 * b.norm()
    assert torch.equal(a == 0, b == 0)
