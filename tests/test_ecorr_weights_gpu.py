"""The ecorr flush's weights at the ends of their range (GPU, against the sum over the placements' own
histograms): as small as a normal double holds them in FP64."""
import numpy as np
import pytest

from tests.test_ecorr_flush_gpu import _system

pytestmark = pytest.mark.gpu


def _flush(precision, sw):
    """(ecorr, histograms) of one call of unit-volume placements with weights sw."""
    n = len(sw)
    w, topo, bins, gpu = _system(300, 21.0, 7, {}, 0, precision)
    pos, cell = w.frame(0)
    pl = w.placements(0, n)
    tag = np.full(n, topo["nummol"], np.int32)
    gpu.frame(pos, cell)
    uv = gpu.placements(tag, pl, np.zeros(n), want_uvengy=True)["uvengy"][:, 1:]
    H = np.stack([np.bincount(np.searchsorted(bins["uvcrd"], u, side="left") - 1, minlength=gpu.ermax) for u in uv])
    gpu.engclear()
    gpu.placements(tag, pl, sw)
    got = gpu.accum()["ecorr"]
    gpu.close()
    return got, H.astype(float)


@pytest.mark.parametrize("scale", [1e-303, 1e-304, 1e-305, 3e-308])
def test_smallest_weights(gpu_lib, scale):
    sw = np.random.default_rng(4).uniform(1.0, 1.5, 64) * scale
    got, H = _flush("fp64", sw)
    want = (H * sw[:, None]).T @ H
    np.testing.assert_array_equal(got != 0.0, want != 0.0)
    np.testing.assert_allclose(got, want, rtol=1e-12)
