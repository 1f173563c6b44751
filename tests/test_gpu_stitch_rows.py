"""The by-rows stitching kernel (at most two windows on a row) at the edges of
its row blocks (32) and column rounds (8), with rows kept, blended and covered
by no window, and non-finite samples on either side of an overlap: equal to
the oracle, bit for bit."""
import os
import sys

import numpy as np
import pytest

import kirch_datuming_b200 as kd

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.join(os.path.dirname(HERE), "oracle"))
import stitch as so  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("blend,aper,lateral", [(15, 0, False), (3, 4, True), (0, 1, True), (-1, 2, True), (1, 0, True)])
@pytest.mark.parametrize("n1,n2,n3,wins", [
    (31, 7, 1, [(0, 30)]), (33, 1, 9, [(1, 12), (8, 32)]), (64, 13, 5, [(0, 31), (30, 40), (40, 63)]),
    (97, 8, 1, [(0, 40), (21, 70), (60, 90)]), (150, 3, 2, [(5, 64), (33, 65), (65, 149)])])
def test_rows_equal_oracle(n1, n2, n3, wins, blend, aper, lateral):
    import torch
    rng = np.random.default_rng(n1 + n2 + blend)
    vols = [rng.standard_normal((n3, n2, e - s + 1)).astype(np.float32) for s, e in wins]
    scales = [1.0 + 0.25 * k for k in range(len(wins))]
    for v in vols:  # the oracle refuses non-finite windows: 0 there, not finite on the device
        v[n3 - 1, n2 - 1, 0] = v[0, 0, -1] = 0.0
    ref = so.stitch(n1, wins, vols, scales, blend, aper if lateral else 0, 0.7)
    for v in vols:
        v[n3 - 1, n2 - 1, 0], v[0, 0, -1] = np.inf, np.nan
    out = torch.full((n3, n2, n1), 7.0, dtype=torch.float32, device="cuda")
    bad = kd.stitch_windows(out, [torch.from_numpy(v).cuda() for v in vols], wins, blend, scales, lateral, aper, 0.7)
    got = out.cpu().numpy()
    assert bad == [2] * len(wins)
    assert np.array_equal(got.view(np.uint32), ref.view(np.uint32))
