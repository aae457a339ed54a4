"""Grid shapes and the PME kernels they take (GPU, mixed path, against the oracle): cubic grids of
every kind of compile-time plan (multiples of four, even, odd, three radices), square planes
with another third length (the compile-time plane kernel with the general slab kernel), and
grids with three lengths of their own."""
import numpy as np
import pytest

from tests import helpers

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid,order", [((36, 36, 36), 4), ((54, 54, 54), 6), ((75, 75, 75), 4), ((81, 81, 81), 4),
                                        ((135, 135, 135), 4), ((54, 54, 80), 6), ((45, 45, 36), 4),
                                        ((64, 64, 25), 8), ((36, 36, 128), 4), ((40, 48, 48), 4), ((27, 30, 50), 6)])
def test_against_oracle(gpu_lib, oracle, grid, order):
    from ermod_gb300.engproc import EnergyRepresentation
    w = helpers.small_refs(corrcal=0, wgtslf=0)
    w.params.update(splodr=order, ms1max=grid[0], ms2max=grid[1], ms3max=grid[2])
    topo, bins = helpers.build_inputs(w)
    gpu = EnergyRepresentation(w.params, topo, bins, precision="mixed")
    orc = oracle.Oracle(w.params, topo, bins)
    pos, cell = w.frame(0)
    pl = w.placements(0, 7)  # the last interleaved group of four holds three
    tag = np.full(len(pl), topo["nummol"], np.int32)
    orc.frame(pos, cell)
    ro = orc.placements(tag, pl)
    gpu.frame(pos, cell)
    rg = gpu.placements(tag, pl, want_uvengy=True)
    label = f"{grid} order {order}"
    helpers.check_energies(rg["uvengy"][:, 1:], ro["uvengy"][:, 1:], "mixed", label)
    helpers.check_histograms(rg["uvengy"][:, 1:], ro["uvengy"][:, 1:], bins["uvcrd"], "mixed", label)
    np.testing.assert_allclose(rg["uvengy"][:, 0], ro["uvengy"][:, 0], rtol=0, atol=helpers.self_tol("mixed", w.solute))
    gpu.close()
