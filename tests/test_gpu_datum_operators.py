"""The datuming operators by short FFTs (8 to 64 points, and Horner's rule
beyond) and the cmp=1 sums, at the filter lengths where the form changes and
at gathers where several trace positions share a shot, against the FP64 oracle
(1e-5 relative L2: FP32 spectra and sums, the operators in FP64)."""
import os
import sys

import numpy as np
import pytest

import kirch_datuming_b200 as kd

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.join(os.path.dirname(HERE), "oracle"))
sys.path.insert(0, HERE)
import datum as D  # noqa: E402
from test_datum_oracle import GOLD, META, rel  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cmp,ns,nh,ds", [(0, 13, 37, 0.02), (1, 11, 13, 0.02), (1, 14, 9, 0.01), (1, 9, 11, 0.04)])
@pytest.mark.parametrize("samples", [1, 6, 7, 14, 15, 30, 31, 62, 63, 90])
def test_filter_lengths_vs_oracle(cmp, ns, nh, ds, samples):
    """samples + 1 filter samples: the last of a transform size, the first of
    the next; shots at, below and above the trace spacing."""
    t, G, dt, nt = META["table"], np.ascontiguousarray(GOLD["green"]), 0.004, 93
    h0, s0 = (-0.02 * (nh // 2), 0.22) if cmp else (0.02, 0.06)
    kw = dict(aperture=5, taper=3, data_taper=2, cmp=cmp, antialias=1.0, length=float(np.float32(dt * (samples + 0.5))))
    p = kd.datum_params(nt=nt, nh=nh, ns=ns, dt=dt, h0=h0, dh=0.02, s0=s0, ds=ds, nsg=G.shape[0], nrg=G.shape[0],
                        sg0=t["o"][2], dsg=t["d"][2], rg0=t["o"][2], drg=t["d"][2], sdatum=0.1, rdatum=0.1, **kw)
    x = np.random.default_rng(samples).standard_normal((ns, nh, nt)).astype(np.float32)
    out, im = np.empty_like(x), np.empty_like(x)
    kd.datum_freq(p, G, G, x, out, im)
    o = D.Datum(nt, nh, ns, dt, h0, 0.02, s0, ds, G, t["o"][2], t["d"][2], G, t["o"][2], t["d"][2],
                np.float32(0.1), np.float32(0.1), **kw)
    want, want_im = o.run(x, interm=True)
    assert np.linalg.norm(want) > 0
    assert rel(im, want_im) < 1e-5 and rel(out, want) < 1e-5, (rel(im, want_im), rel(out, want))
