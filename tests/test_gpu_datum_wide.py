"""Datuming of spreads so wide that one residue of operators by FFT (up to 64
frequencies of nh x nh terms) passes the memory a chunk may take: the call
stays within it, and the interior traces equal those of a short spread at the
same positions, taken by the FP64 oracle (1e-5 relative L2, as the other
datuming tests)."""
import os
import sys

import numpy as np
import pytest

import kirch_datuming_b200 as kd

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.join(os.path.dirname(HERE), "oracle"))
import datum as D  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nh", [1700, 3000])
def test_wide_spread_keeps_to_its_memory(nh):
    """Below (1700) and above (3000) the width at which the form changes."""
    import torch
    ns, nt, dt, dh, depth, aper = 1, 60, 0.004, 0.02, 0.1, 5
    ng, dg = 601, 0.1
    x = np.arange(ng) * dg
    table = (np.sqrt((x[:, None] - x[None, :]) ** 2 + depth ** 2) / 2.0).astype(np.float32)
    f = lambda v: float(np.float32(v))  # noqa: E731
    kw = dict(aperture=aper, taper=0, data_taper=0, cmp=0, antialias=1.0, length=f(dt * 50.5))

    def params(n, h0):
        return kd.datum_params(nt=nt, nh=n, ns=ns, dt=f(dt), h0=f(h0), dh=f(dh), s0=0.0, ds=f(dh), nsg=ng, nrg=ng, sg0=0.0,
                               dsg=f(dg), rg0=0.0, drg=f(dg), sdatum=f(depth), rdatum=f(depth), **kw)
    data = torch.randn((ns, nh, nt), generator=torch.Generator().manual_seed(nh)).numpy()
    small = np.ascontiguousarray(data[:, :8])
    kd.datum_freq(params(8, 0.0), table, table, small, np.empty_like(small))  # loads the kernels
    kd.datum_release()
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    out = np.empty_like(data)
    kd.datum_freq(params(nh, 0.0), table, table, data, out)
    held = free - torch.cuda.mem_get_info()[0]
    kd.datum_release()
    # a chunk's 1.5 GB, 12 bytes a term, and per trace four arrays of the transform's length: its spectrum,
    # the padded trace, its transform and cuFFT's work area; 64 MB for the rest
    nfft = kd.datum_sizes(params(nh, 0.0), table, table)[1]
    assert held < (1536 << 20) + 12 * nh * nh + 4 * nh * 4 * (nfft + 2) + (64 << 20), held >> 20
    # a window of the spread: its interior traces see the same neighbours
    n, first = 48, nh // 2
    o = D.Datum(nt, n, ns, f(dt), f(first * dh), f(dh), 0.0, f(dh), table, 0.0, f(dg), table, 0.0, f(dg),
                np.float32(depth), np.float32(depth), **kw)
    assert o.nfft == nfft
    want = o.run(data[:, first:first + n])[:, aper:-aper]
    got = out[:, first + aper:first + n - aper]
    assert np.linalg.norm(want) > 0
    assert np.linalg.norm(got - want) <= 1e-5 * np.linalg.norm(want)
