"""Counts of non-finite samples of the stitching when a window's scale itself
is not finite: every sample of the window, none of the columns that a round of
the kernel reads past the end; equal to the window-by-window calls."""
import numpy as np
import pytest

import kirch_datuming_b200 as kd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [float("inf"), float("nan"), 3e38])
@pytest.mark.parametrize("n2,n3", [(1, 1), (7, 1), (8, 2), (13, 5), (17, 9)])
def test_scales_not_finite(n2, n3, scale):
    import torch
    n1, wins = 70, [(0, 40), (31, 69)]
    rng = np.random.default_rng(n2)
    vols = [torch.from_numpy((2 + rng.random((n3, n2, e - s + 1))).astype(np.float32)).cuda() for s, e in wins]
    for scales in ([scale, 1.0], [1.0, scale], [scale, scale]):
        out = torch.empty((n3, n2, n1), device="cuda")
        bad = kd.stitch_windows(out, vols, wins, 5, scales)
        assert bad == [v.numel() if not 2 * s < 3.4e38 else 0 for v, s in zip(vols, scales)]
        one, counts, prev = torch.zeros_like(out), [], -1
        for v, (a, b), s in zip(vols, wins, scales):
            counts.append(kd.stitch_window(one, v, a, b, prev, 5, s))
            prev = b
        assert counts == bad
        assert torch.equal(out, one)


def test_most_columns_accepted():
    """2^31 - 1 columns (17 GB with the window): the last ones are written by
    each form of the stitching -- by rows, by columns (three windows on a row)
    and window by window."""
    import torch
    n2 = 2 ** 31 - 1
    vol = torch.empty((1, n2, 1), device="cuda").uniform_(1.0, 2.0)
    out = torch.empty_like(vol)
    for layers in ([vol], [vol, vol, vol]):
        out.zero_()
        assert kd.stitch_windows(out, layers, [(0, 0)] * len(layers), 0) == [0] * len(layers)
        assert torch.equal(out, vol)
    out.zero_()
    assert kd.stitch_window(out, vol, 0, 0) == 0
    assert torch.equal(out, vol)
