"""The host API's frames (GPU): a call that returns before its copy has run leaves the caller free to
overwrite the array, below, at and above the largest frame that is staged; and a graph launched
right after such a call, on another stream, is not disturbed by it."""
import numpy as np
import pytest

from ermod_gb300 import setconf, synth
from tests import helpers

pytestmark = pytest.mark.gpu

STAGED = (256 << 10) // 24  # sites whose coordinates fill the staging


def _engine(w, topo, bins, **kw):
    from ermod_gb300.engproc import EnergyRepresentation
    return EnergyRepresentation(w.params, topo, bins, **kw)


# a solute of as many sites as make numatm the wanted number
@pytest.mark.parametrize("numatm", [600, STAGED - 1, STAGED, STAGED + 1])
def test_caller_overwrites_the_frame(gpu_lib, numatm):
    nwater = (numatm - 6) // 3
    nsite = numatm - 3 * nwater
    box = 1.05 * (nwater / 0.0334) ** (1.0 / 3.0)
    sol = synth.random_solute(np.random.default_rng(5), nsite)
    w = synth.Workload("frames", "refs", box, nwater, sol, synth._params(2, 48, corrcal=0, wgtslf=0), 3, 6, 4,
                       int(np.ceil(nwater ** (1.0 / 3.0))) + 1)
    topo, bins = helpers.build_inputs(w, dict(setconf.HIST_DEFAULT, ecdmin=-400.0))
    assert int(topo["numatm"]) == numatm
    tag = np.full(4, topo["nummol"], np.int32)
    a, b = _engine(w, topo, bins), _engine(w, topo, bins)
    buf = np.empty((numatm, 3))
    for f in range(6):
        pos, cell = w.frame(f)
        pl = w.placements(f)
        a.frame(pos, cell)
        a.sync()
        want = a.placements(tag, pl, want_uvengy=True)["uvengy"]
        buf[:] = pos
        b.frame(buf, cell)
        buf[:] = 1.0e3  # the caller's array is its own again
        np.testing.assert_array_equal(b.placements(tag, pl, want_uvengy=True)["uvengy"], want)
    for f in range(6):  # frames in quick succession: the last one counts
        buf[:] = w.frame(f)[0]
        b.frame(buf, cell)
    buf[:] = 1.0e3
    np.testing.assert_array_equal(b.placements(tag, pl, want_uvengy=True)["uvengy"], want)
    a.close()
    b.close()


def test_graph_right_after_a_frame(gpu_lib):
    from ermod_gb300.multisystem import SystemGraph
    w = helpers.small_refs(nwater=3000, box=46.0, K=48, corrcal=0, wgtslf=0, lattice=15)
    topo, bins = helpers.build_inputs(w, dict(setconf.HIST_DEFAULT, ecdmin=-400.0))
    n = 40
    tag = np.full(n, topo["nummol"], np.int32)
    pos, cell = w.frame(0)
    other = np.random.default_rng(2).uniform(0.0, 46.0, pos.shape)
    pl = w.placements(0, n)
    ref = _engine(w, topo, bins)
    ref.frame(pos, cell)
    ref.placements(tag, pl)
    want = ref.accum()["edens"]
    gpu = _engine(w, topo, bins)
    gpu.frame(pos, cell)
    gpu.placements(tag, pl)
    g = SystemGraph([gpu], [(pos, cell)], [pl], [topo["nummol"]])
    for _ in range(20):
        gpu.engclear()
        gpu.frame(other, cell)  # replaced by the graph's own frame
        g.launch()
        g.sync()
        np.testing.assert_array_equal(gpu.accum()["edens"], want)
    g.close()
    gpu.close()
    ref.close()
