"""The ecorr flush (GPU) against the sum over the placements' own histograms: rings below, at and
above the matrix kernels' least length, of one and several flushes and of more than one pass;
counts of one, two and three 8-bit digits; weights within their range of exponents, beyond it
(the walk), zero, and as large as they come; more active bins than they take.

Bounds: a flush keeps at least 44 bits (FP64 path 53) of every entry's terms, all positive, so
an entry is off by less than 2^-43 of itself per flush; 1e-11 (1e-12) covers the flushes of a
call and the reference's own rounding."""
import numpy as np
import pytest

from ermod_gb300 import setconf, synth

pytestmark = pytest.mark.gpu


def _system(nwater, box, lattice, hist, batch, precision):
    from ermod_gb300.engproc import EnergyRepresentation
    w = synth.Workload("flush", "refs", box, nwater, synth.methanol_like(),
                       synth._params(2, 32, corrcal=1, wgtslf=0, estype=1), 11, 1, 1, lattice)
    topo = setconf.setparam_topology(w.species(), slttype=2)
    bins = setconf.enginit_bins(topo["numslv"], dict(setconf.HIST_DEFAULT, ecdmin=-60.0, **hist))
    return w, topo, bins, EnergyRepresentation(w.params, topo, bins, precision=precision, batch=batch)


COARSE = dict(eclbin=5.0, ecfbin=0.05, ec0bin=0.2, finfac=4.0, pecore=20)
FINE = dict(eclbin=0.02, ecfbin=2.5e-4, ec0bin=2.0e-5, finfac=100.0, pecore=500)


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("n,nwater,box,lattice,hist,batch,weights", [
    (47, 300, 21.0, 7, {}, 0, "near"), (48, 300, 21.0, 7, {}, 0, "near"), (49, 300, 21.0, 7, {}, 16, "unit"),
    (700, 300, 21.0, 7, {}, 64, "near"), (1100, 120, 16.0, 5, {}, 512, "near"),
    (64, 3000, 46.0, 15, COARSE, 0, "near"), (48, 70000, 130.0, 42, COARSE, 0, "near"),
    (64, 300, 21.0, 7, {}, 0, "edge"), (64, 300, 21.0, 7, {}, 0, "wide"), (64, 300, 21.0, 7, {}, 0, "zero"),
    (64, 300, 21.0, 7, {}, 0, "huge"), (60, 3000, 46.0, 15, FINE, 0, "near")])
def test_flush_against_histograms(gpu_lib, n, nwater, box, lattice, hist, batch, weights, precision):
    w, topo, bins, gpu = _system(nwater, box, lattice, hist, batch, precision)
    rng = np.random.default_rng(n)
    sw = {"unit": np.ones(n), "near": rng.uniform(0.5, 1.5, n), "edge": 2.0 ** -(np.arange(n) % 13) * 1.3,
          "wide": 10.0 ** rng.uniform(-8, 8, n), "zero": rng.uniform(0.5, 1.5, n) * (np.arange(n) % 3 > 0),
          "huge": rng.uniform(0.5, 1.5, n) * 1e280}[weights]
    pos, cell = w.frame(0)
    pl = w.placements(0, n)
    gpu.frame(pos, cell)
    tag = np.full(n, topo["nummol"], np.int32)
    H = np.zeros((n, gpu.ermax))
    for p0 in range(0, n, 100):  # the same energies as the accumulating call's, in parts
        uv = gpu.placements(tag[p0:p0 + 100], pl[p0:p0 + 100], np.zeros(len(tag[p0:p0 + 100])), want_uvengy=True)["uvengy"]
        for p, u in enumerate(uv[:, 1:]):
            H[p0 + p] = np.bincount(np.searchsorted(bins["uvcrd"], u, side="left") - 1, minlength=gpu.ermax)
    gpu.engclear()
    gpu.placements(tag, pl, sw)
    got = gpu.accum()["ecorr"]
    want = (H * sw[:, None]).T @ H
    np.testing.assert_array_equal(got != 0.0, want != 0.0)
    np.testing.assert_allclose(got, want, rtol=1e-11 if precision == "mixed" else 1e-12)
    if weights == "unit":
        np.testing.assert_array_equal(got, want)
    if precision == "mixed":  # its kernels add one sum at both mirrored entries
        np.testing.assert_array_equal(got, got.T)
    gpu.close()
