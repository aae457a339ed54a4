"""The ecorr flush's weights at the ends of their range (GPU, against the sum over the placements' own
histograms): as small as a normal double holds them in FP64, and 48-bit weights of 2^-12 of the
largest, the widest spread that the matrix kernels take; and a flush adds to an entry once, whatever
the number of its counts' digits."""
import numpy as np
import pytest

from tests.test_ecorr_flush_gpu import COARSE, _system

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


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_spread_weights_keep_48_bits(gpu_lib, precision):
    n = 64
    k = 2 ** 47 + np.random.default_rng(9).integers(0, 2 ** 46, n) * 2 + 1  # 48 bits, the last one set
    spread = 12 if precision == "mixed" else 10
    k_hi = k >> 24 << 24
    exps = np.full(n, -spread)
    exps[5] = 0
    scale = 2.0 ** (exps - 47.0)
    got, H = _flush(precision, k * scale)
    # the weights' halves of 24 bits: sums of exact products, rounded once when they are joined
    want = (H * (k_hi * scale)[:, None]).T @ H + (H * ((k - k_hi) * scale)[:, None]).T @ H
    # every weight is a multiple of the matrix kernels' unit, so only the joining rounds: twice
    np.testing.assert_allclose(got, want, rtol=2.0 ** -50)


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_one_addition_per_flush(gpu_lib, precision):
    """Counts of one and two 8-bit digits: two flushes give the sum of each by itself, rounded once."""
    w, topo, bins, gpu = _system(3000, 46.0, 15, COARSE, 0, precision)
    pos, cell = w.frame(0)
    gpu.frame(pos, cell)
    n = 64
    pl = w.placements(0, 2 * n)
    sw = np.random.default_rng(8).uniform(1.0, 2.0, 2 * n)
    tag = np.full(n, topo["nummol"], np.int32)
    parts = [(pl[:n], sw[:n]), (pl[n:], sw[n:])]
    alone = []
    for p, x in parts:
        gpu.engclear()
        gpu.placements(tag, p, x)
        alone.append(gpu.accum()["ecorr"])
    gpu.engclear()
    for p, x in parts:
        gpu.placements(tag, p, x)
    both = gpu.accum()["ecorr"]
    gpu.close()
    assert alone[0].max() > 2.0 * n * 256.0 ** 2
    np.testing.assert_array_equal(both, alone[0] + alone[1])
