"""FP64 path in batches (GPU, against the oracle): calls of one placement, of a power of two,
of one more and one less (the inverse transforms split into powers of two, the last batch
ragged); orders 4, 6 and 8 (stencils wider than a molecule's four threads) on grids whose
spectrum rows end inside a CTA; solution mode's wider split of a molecule; a failing
placement in the middle of a batch, before which every placement is accumulated."""
import numpy as np
import pytest

from tests import helpers

pytestmark = pytest.mark.gpu


def _engines(oracle, w, **kw):
    from ermod_gb300.engproc import EnergyRepresentation
    topo, bins = helpers.build_inputs(w)
    return EnergyRepresentation(w.params, topo, bins, precision="fp64"), oracle.Oracle(w.params, topo, bins), topo, bins


@pytest.mark.parametrize("nplace,order,grid", [(1, 4, (32, 32, 32)), (63, 4, (32, 32, 32)), (64, 4, (32, 32, 32)),
                                               (67, 4, (31, 34, 37)), (3, 6, (27, 33, 30)), (5, 8, (64, 28, 26))])
def test_batches_against_oracle(gpu_lib, oracle, nplace, order, grid):
    w = helpers.small_refs(nwater=301, box=21.0, corrcal=1, wgtslf=0, lattice=7)
    w.params.update(splodr=order, ms1max=grid[0], ms2max=grid[1], ms3max=grid[2], estype=1)
    gpu, orc, topo, bins = _engines(oracle, w)
    pos, cell = w.frame(0)
    gpu.frame(pos, cell)
    orc.frame(pos, cell)
    pl = w.placements(0, nplace)
    tag = np.full(nplace, topo["nummol"], np.int32)
    rg, ro = gpu.placements(tag, pl, want_uvengy=True), orc.placements(tag, pl)
    helpers.check_energies(rg["uvengy"], ro["uvengy"], "fp64", f"{nplace} placements")
    ag, ao = gpu.accum(), orc.accum()
    np.testing.assert_array_equal(ag["edens"], ao["edens"])
    np.testing.assert_array_equal(ag["ecorr"], ao["ecorr"])
    gpu.close()


@pytest.mark.parametrize("nwater", [37, 250])
def test_solution_mode_split(gpu_lib, oracle, nwater):
    from ermod_gb300 import synth
    w = synth.Workload("soln_test", "soln", 26.0, nwater, synth.methanol_like(),
                       synth._params(1, 30, corrcal=0, wgtslf=0), 5, 1, 1, 9, cavity=4.5)
    gpu, orc, topo, bins = _engines(oracle, w)
    pos, cell = w.frame(0)
    gpu.frame(pos, cell)
    orc.frame(pos, cell)
    rg = gpu.placements([topo["nummol"]], want_uvengy=True, want_flceng=True)
    ro = orc.placements([topo["nummol"]])
    helpers.check_energies(rg["uvengy"], ro["uvengy"], "fp64", "solution mode")
    np.testing.assert_allclose(rg["flceng"], ro["flceng"], rtol=1e-10, atol=1e-9)
    ag, ao = gpu.accum(), orc.accum()
    np.testing.assert_array_equal(ag["edens"], ao["edens"])
    gpu.close()


@pytest.mark.parametrize("bad", [0, 5, 40])
def test_failing_placement_inside_a_batch(gpu_lib, oracle, bad):
    """The charged site without LJ of placement `bad` lands next to a water hydrogen: eng_min."""
    from ermod_gb300 import engproc
    sol = dict(xyz=np.array([[0.0, 0.0, 0.0], [2.0, 0.0, 0.0]]), charge=np.array([0.02, -0.02]), sig=np.array([3.0, 0.0]),
               eps=np.array([0.1, 0.0]), mass=np.array([12.0, 1.0]))
    w = helpers.small_refs(nwater=301, box=21.0, corrcal=1, wgtslf=1, lattice=7, solute=sol)
    gpu, _, topo, bins = _engines(oracle, w)
    ref, _, _, _ = _engines(oracle, w)
    pos, cell = w.frame(0)
    n = 48
    pl = w.placements(0, n)
    pl[bad, 1] = pos[10] + np.array([0.01, 0.0, 0.0])
    pl[bad, 0] = pl[bad, 1] + np.array([0.0, 0.0, 2.0])
    tag = np.full(n, topo["nummol"], np.int32)
    gpu.frame(pos, cell)
    with pytest.raises(engproc.ErmodError) as err:
        gpu.placements(tag, pl)
    assert err.value.name == "eng_min" and gpu.error_info()[0] == bad
    ref.frame(pos, cell)
    ref.placements(tag[:bad], pl[:bad])
    a, b = gpu.accum(), ref.accum()
    assert a["engsmpl"] == bad
    for k in ("edens", "ecorr", "minuv", "maxuv", "engnorm"):
        np.testing.assert_allclose(a[k], b[k], rtol=1e-10, err_msg=k)
    gpu.close()
    ref.close()
