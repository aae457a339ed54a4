"""Solution mode's molecules per finish block at their edges (GPU, mixed path, against the oracle):
one block of 16 exactly full, one more and one fewer, and the largest system that takes 16 and
the first that takes 64."""
import numpy as np
import pytest

from ermod_gb300 import synth
from tests import helpers

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("molecules", [15, 16, 17, 16 * 152, 16 * 152 + 1])
def test_against_oracle(gpu_lib, oracle, molecules):
    from ermod_gb300.engproc import EnergyRepresentation
    nwater = molecules - 1  # the solute is a molecule of the frame
    box, lattice = (26.0, 9) if nwater < 300 else (43.0, 14)
    w = synth.Workload("tiles", "soln", box, nwater, synth.methanol_like(), synth._params(1, 40, corrcal=0, wgtslf=0), 5,
                       1, 1, lattice, cavity=4.5)
    topo, bins = helpers.build_inputs(w)
    gpu = EnergyRepresentation(w.params, topo, bins, precision="mixed")
    orc = oracle.Oracle(w.params, topo, bins)
    pos, cell = w.frame(0)
    gpu.frame(pos, cell)
    orc.frame(pos, cell)
    rg = gpu.placements([topo["nummol"]], want_uvengy=True, want_flceng=True)
    ro = orc.placements([topo["nummol"]])
    label = f"{molecules} molecules"
    helpers.check_energies(rg["uvengy"][:, 1:], ro["uvengy"][:, 1:], "mixed", label)
    helpers.check_histograms(rg["uvengy"][:, 1:-1], ro["uvengy"][:, 1:-1], bins["uvcrd"], "mixed", label)
    # flceng is the sum of the molecules' energies, each within the band
    np.testing.assert_allclose(rg["flceng"], ro["flceng"], rtol=0, atol=helpers.MIXED_BAND * molecules)
    gpu.close()
