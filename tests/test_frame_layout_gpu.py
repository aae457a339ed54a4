"""The frame's spatial layout (GPU, against the oracle): molecules sorted by counting in one CTA,
in a cluster, and by radix sort; sites listed by brick inside the scan and grid-wide; the cells
of a dilute box (coarser codes); batches of one, two and three placements in solution mode
(accumulated in one launch or three), whose molecules fill a 64-molecule tile exactly, by one
more, and not."""
import numpy as np
import pytest

from ermod_gb300 import setconf, synth
from tests import helpers

pytestmark = pytest.mark.gpu


def _workload(nwater, box, K, lattice, mode="refs"):
    return synth.Workload("layout", mode, box, nwater, synth.methanol_like(),
                          synth._params(1 if mode == "soln" else 2, K, corrcal=0, wgtslf=0), 7, 1, 2, lattice, cavity=4.5)


def _wide_hist():
    """A coordinate whose soft region holds every energy of these inputs."""
    return dict(setconf.HIST_DEFAULT, ecdmin=-400.0, eccore=400.0, eclbin=0.5)


def _engines(oracle, w, topo, bins, precision):
    from ermod_gb300.engproc import EnergyRepresentation
    return EnergyRepresentation(w.params, topo, bins, precision=precision), oracle.Oracle(w.params, topo, bins)


# one CTA; its last size and the next (cluster); sites listed grid-wide; radix sort; dilute
@pytest.mark.parametrize("nwater,box,K,lattice", [(50, 26.0, 32, 9), (3072, 46.0, 45, 15), (3073, 46.0, 45, 15),
                                                  (9000, 66.0, 64, 21), (98305, 144.0, 72, 47), (200, 190.0, 64, 9)])
@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_layout_against_oracle(gpu_lib, oracle, precision, nwater, box, K, lattice):
    w = _workload(nwater, box, K, lattice)
    topo, bins = helpers.build_inputs(w)
    gpu, orc = _engines(oracle, w, topo, bins, precision)
    pos, cell = w.frame(0)
    pos = pos + np.array([0.3 * box, -0.7 * box, 1.4 * box])  # sites outside the cell
    gpu.frame(pos, cell)
    orc.frame(pos, cell)
    pl = w.placements(0, 2)
    tag = np.full(2, topo["nummol"], np.int32)
    rg = gpu.placements(tag, pl, want_uvengy=True)
    ro = orc.placements(tag, pl)
    helpers.check_energies(rg["uvengy"][:, 1:], ro["uvengy"][:, 1:], precision, f"{nwater} waters")
    a = gpu.accum()
    np.testing.assert_allclose(a["edens"].sum(), a["engnorm"] * nwater, rtol=1e-12)
    gpu.close()


@pytest.mark.parametrize("nwater", [60, 61, 130])
@pytest.mark.parametrize("nsol", [1, 2, 3])
@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_small_solution_batches(gpu_lib, oracle, precision, nwater, nsol):
    """nsol solutes: 64 physical molecules for (60, 4 - nsol), one more or fewer otherwise."""
    w = _workload(nwater + 4, 26.0, 32, 9, mode="soln")
    sol = w.solute
    species = [dict(count=nwater, sluvid=0, charge=synth.WATER_CHARGE, eps=synth.WATER_EPS, len=synth.WATER_SIG),
               dict(count=nsol, sluvid=1, charge=sol["charge"], eps=sol["eps"], len=sol["sig"])]
    topo = setconf.setparam_topology(species, slttype=1)
    bins = setconf.enginit_bins(topo["numslv"], _wide_hist())
    w.params["selfcal"] = 1
    gpu, orc = _engines(oracle, w, topo, bins, precision)
    pos, cell = w.frame(0)
    sxyz = pos[-len(sol["charge"]):]
    shifts = [np.zeros(3), np.array([11.0, 4.0, -8.0]), np.array([-9.0, 10.0, 6.0])]
    pos = np.concatenate([pos[:3 * nwater]] + [sxyz + s for s in shifts[:nsol]])
    tag = np.arange(nwater + 1, nwater + 1 + nsol, dtype=np.int32)
    gpu.frame(pos, cell)
    orc.frame(pos, cell)
    ro = orc.placements(tag)
    rg = gpu.placements(tag, want_uvengy=True, want_flceng=True)
    helpers.check_energies(rg["uvengy"][:, 1:], ro["uvengy"][:, 1:], precision, f"{nsol} solutes")
    # sums over fewer than 200 molecules, each within the energy tolerance
    tol = 200 * helpers.ENERGY_TOL[precision][0]
    np.testing.assert_allclose(rg["flceng"], ro["flceng"], rtol=1e-11, atol=tol)
    ag, ao = gpu.accum(), orc.accum()
    for k in ("engnorm", "engsmpl", "avslf"):
        np.testing.assert_allclose(ag[k], ao[k], rtol=1e-12)
    for k in ("minuv", "maxuv", "slnuv"):
        np.testing.assert_allclose(ag[k], ao[k], rtol=1e-11, atol=tol * max(1.0, ao["engnorm"]))
    assert ag["eself"].sum() == pytest.approx(ao["eself"].sum(), rel=1e-12)
    helpers.check_histograms(rg["uvengy"][:, 1:], ro["uvengy"][:, 1:], bins["uvcrd"][:bins["uvmax"][0]], precision)
    gpu.close()
