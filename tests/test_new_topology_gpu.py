"""A context that takes another topology (GPU): a rigid solute's self energy is the new solute's."""
import numpy as np
import pytest

from ermod_gb300 import synth
from tests import helpers

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_self_energy_of_the_new_solute(gpu_lib, precision):
    from ermod_gb300.engproc import EnergyRepresentation
    first = synth.methanol_like()
    second = dict(first, charge=2.0 * first["charge"][::-1])
    hist = dict(helpers.setconf.HIST_DEFAULT, ecdmin=-400.0)
    ws = [helpers.small_refs(corrcal=0, wgtslf=0, solute=s) for s in (first, second)]
    (topo, bins), (topo2, _) = (helpers.build_inputs(w, hist) for w in ws)
    pos, cell = ws[0].frame(0)
    pl = ws[0].placements(0, 5)
    tag = np.full(5, topo["nummol"], np.int32)
    gpu = EnergyRepresentation(ws[0].params, topo, bins, precision=precision)
    gpu.frame(pos, cell)
    gpu.placements(tag, pl)
    gpu.set_topology(topo2)
    gpu.frame(pos, cell)
    got = gpu.placements(tag, pl, want_uvengy=True)["uvengy"]
    gpu.close()
    ref = EnergyRepresentation(ws[1].params, topo2, bins, precision=precision)
    ref.frame(pos, cell)
    want = ref.placements(tag, pl, want_uvengy=True)["uvengy"]
    ref.close()
    np.testing.assert_array_equal(got, want)
