"""Energy coordinates of tens of thousands of bins (GPU, mixed path): at and beyond the most that the
finish kernel's scratch for four and for eight placements leaves room for, up to 52,120, and with a
solute of many sites.  Energies do not depend on the coordinate, and edens counts them."""
import numpy as np
import pytest

from ermod_gb300 import setconf, synth
from tests import helpers

pytestmark = pytest.mark.gpu


def _bins(ermax):
    edges = np.concatenate([np.linspace(-400.0, 400.0, ermax - 1), [1.0e11]])
    return dict(uvcrd=edges, uvmax=np.array([ermax], np.int32), uvsoft=np.array([ermax - 1], np.int32),
                escrd=np.array([-1.0e11, 1.0e11]), esmax=2)


@pytest.mark.parametrize("ermax,nsite,group", [(48276, 16, 0), (48277, 16, 0), (48788, 6, 0), (48789, 6, 0),
                                               (50040, 6, 8), (52120, 6, 0), (52120, 20, 0)])
def test_counts(gpu_lib, ermax, nsite, group):
    from ermod_gb300.engproc import EnergyRepresentation
    sol = synth.methanol_like() if nsite == 6 else synth.random_solute(np.random.default_rng(nsite), nsite)
    # enough blocks for the whole group of placements
    w = helpers.small_refs(nwater=2600, box=44.0, K=45, corrcal=0, wgtslf=0, lattice=14, solute=sol)
    w.params["estype"] = 1
    topo = setconf.setparam_topology(w.species(), slttype=2)
    pos, cell = w.frame(0)
    n = 200
    pl = w.placements(0, n)
    tag = np.full(n, topo["nummol"], np.int32)
    uv = []
    for bins in (_bins(1000), _bins(ermax)):
        gpu = EnergyRepresentation(w.params, topo, bins, precision="mixed", finish_group=group)
        gpu.frame(pos, cell)
        uv.append(gpu.placements(tag, pl, want_uvengy=True)["uvengy"][:, 1:])
        count = np.bincount((np.searchsorted(bins["uvcrd"], uv[-1], side="left") - 1).reshape(-1),
                            minlength=len(bins["uvcrd"]))
        np.testing.assert_array_equal(gpu.accum()["edens"], count)
        gpu.close()
    np.testing.assert_array_equal(uv[0], uv[1])
