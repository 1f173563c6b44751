"""Forward modelling (k_spray) at the edges of its 32 x 4 tiles, with records
of one sample interval to many, pairs that miss most tiles, and each of the
three weightings, against the FP64 oracle (1e-5, as the other forward cases)."""
import numpy as np
import pytest

import _cases
import kirch_datuming_b200 as kd
import oracle

pytestmark = pytest.mark.gpu

A = ["cig=1", "mode=angle", "angle_min=0", "angle_max=60", "angle_n=61"]


@pytest.mark.parametrize("tokens,nz,nx,ns,nh,nt", [
    (A, 32, 4, 2, 3, 301), (A, 33, 5, 1, 1, 301), (A, 31, 67, 3, 7, 121), (A, 3, 81, 2, 5, 301),
    (A + ["angle_interp=0"], 41, 81, 3, 5, 200), (["cig=0"], 40, 79, 2, 4, 90),
    (["cig=1", "mode=offset"], 39, 33, 2, 9, 160), (A + ["tau=-0.05", "aperture=15", "aperture_taper=4"], 41, 80, 2, 6, 2500),
    (["cig=1", "mode=angle", "angle_min=20", "angle_max=30", "angle_n=11"], 41, 81, 4, 9, 301)])
def test_model_tiles_vs_oracle(golden, tokens, nz, nx, ns, nh, nt):
    T, D = golden.tables()
    geom = golden.geometry_dict("base")
    full = (geom["sny"], geom["nx"], geom["nz"])
    T, D = (np.ascontiguousarray(t.reshape(full)[:, :nx, :nz]).reshape(-1) for t in (T, D))
    geom.update(nz=nz, nx=nx, nt=nt, ns=ns, nh=nh, ds=float(np.float32(0.09)), s0=float(np.float32(0.1)),
                dh=float(np.float32(0.02)), h0=float(np.float32(0.05)))
    kp = kd.params("adj=0", "cmp=0", *tokens)
    axis = kd.output_axis(kp, kd.geometry(**geom))
    op = _cases.oracle_params(kp, geom, axis)
    model = np.random.default_rng(nz + nh).standard_normal((axis[0], nx, nz)).astype(np.float32)
    plan = kd.Plan(kp, kd.geometry(**geom))
    plan.set_tables(T, D, T, D)
    out = np.zeros((ns, nh, nt), np.float32)
    plan.model(model, out)
    plan.close()
    ref = oracle.model_fwd(op, model, T, D, T, D, fp64=True)
    assert np.linalg.norm(ref) > 0
    assert oracle.rel_l2(out, ref) <= 1e-5
