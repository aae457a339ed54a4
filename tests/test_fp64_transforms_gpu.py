"""The FP64 path's own inverse transforms (GPU, against the oracle): lengths of one, two, three and
four passes, odd ones (whose last row has no partner in its complex transform, also across
placements), the largest radices, and a grid with a length that cuFFT still takes."""
import numpy as np
import pytest

from tests import helpers

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid,order,nplace", [((96, 96, 96), 4, 2), ((45, 27, 25), 4, 3), ((25, 25, 25), 6, 1),
                                               ((16, 12, 10), 4, 5), ((128, 20, 36), 8, 2), ((15, 250, 9), 4, 3),
                                               ((125, 18, 54), 4, 1), ((9, 15, 375), 4, 1), ((240, 8, 81), 6, 2),
                                               ((32, 32, 34), 4, 2)])
def test_against_oracle(gpu_lib, oracle, grid, order, nplace):
    from ermod_gb300.engproc import EnergyRepresentation
    w = helpers.small_refs(nwater=301, box=21.0, corrcal=0, wgtslf=0, lattice=7)
    w.params.update(splodr=order, ms1max=grid[0], ms2max=grid[1], ms3max=grid[2], estype=1)
    topo, bins = helpers.build_inputs(w)
    gpu = EnergyRepresentation(w.params, topo, bins, precision="fp64")
    orc = oracle.Oracle(w.params, topo, bins)
    pos, cell = w.frame(0)
    gpu.frame(pos, cell)
    orc.frame(pos, cell)
    pl = w.placements(0, nplace)
    tag = np.full(nplace, topo["nummol"], np.int32)
    rg, ro = gpu.placements(tag, pl, want_uvengy=True), orc.placements(tag, pl)
    helpers.check_energies(rg["uvengy"], ro["uvengy"], "fp64", f"{grid} order {order}")
    np.testing.assert_array_equal(gpu.accum()["edens"], orc.accum()["edens"])
    gpu.close()
