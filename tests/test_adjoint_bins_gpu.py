"""The adjoint's per-bin sums at the edges of their kernels (GPU, against the FP64 oracle's gradients
binned by the GPU's energies): molecule counts around the 4,096 keys that a bin's CTA lists at
a time, more parameters than it has threads, and an energy coordinate of so many bins that the
molecules are sorted instead."""
import numpy as np
import pytest

from ermod_gb300 import setconf, synth
from tests.test_adjoint_gpu import _bins, _check, _run_gpu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nwater,nsite,box,lattice,cavity,hist", [
    (4095, 6, 52.0, 17, 5.2, {}), (4097, 7, 52.0, 17, 6.0, {}), (2000, 90, 50.0, 17, 18.2, dict(ecdmin=-200.0)),
    (3900, 6, 48.0, 16, 5.2, dict(eclbin=4.6e-3))])
def test_bins_against_oracle(gpu_lib, oracle, nwater, nsite, box, lattice, cavity, hist):
    sol = synth.random_solute(np.random.default_rng(31), nsite)
    w = synth.Workload("adj_bins", "soln", box, nwater, sol, synth._params(1, 40, corrcal=0, wgtslf=0), 17, 3, 1,
                       lattice, cavity=cavity)
    w.params.update(estype=1, lwljcut=8.0, upljcut=10.0, elecut=10.0)
    topo = setconf.setparam_topology(w.species(), slttype=1)
    bins = setconf.enginit_bins(topo["numslv"], dict(setconf.HIST_DEFAULT, **hist))
    g, wt, us = _run_gpu(w, topo, bins, [0])
    orc = oracle.Oracle(w.params, topo, bins)
    pos, cell = w.frame(0)
    orc.frame(pos, cell)
    du = orc.adjoint(topo["nummol"])
    edges = bins["uvcrd"]
    b = _bins(us[0][:-1], edges)  # the solute itself is the last
    ref, mag, cnt = np.zeros((3 * nsite, len(edges))), np.zeros((3 * nsite, len(edges))), np.zeros(len(edges))
    np.add.at(ref.T, b, du[:-1])
    np.add.at(mag.T, b, np.abs(du[:-1]))
    np.add.at(cnt, b, 1.0)
    np.testing.assert_array_equal(wt, cnt)
    _check(g, ref, mag)
