"""Many batches without pair correlations (GPU): each batch's histogram is accumulated before its
place is used again, so edens is the count of every placement's energies, whatever the batch."""
import numpy as np
import pytest

from ermod_gb300 import setconf
from tests import helpers

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,batch,nplace", [("mixed", 16, 160), ("mixed", 64, 400), ("mixed", 0, 900),
                                                    ("fp64", 0, 330)])
def test_edens_of_many_batches(gpu_lib, precision, batch, nplace):
    from ermod_gb300.engproc import EnergyRepresentation
    w = helpers.small_refs(corrcal=0, wgtslf=0)
    w.params["estype"] = 1  # unit weights: edens holds counts
    topo = setconf.setparam_topology(w.species(), slttype=2)
    bins = setconf.enginit_bins(topo["numslv"], dict(setconf.HIST_DEFAULT, ecdmin=-200.0))
    gpu = EnergyRepresentation(w.params, topo, bins, precision=precision, batch=batch)
    pos, cell = w.frame(0)
    gpu.frame(pos, cell)
    pl = w.placements(0, nplace)
    tag = np.full(nplace, topo["nummol"], np.int32)
    u = gpu.placements(tag, pl, want_uvengy=True)["uvengy"][:, 1:]
    count = np.bincount((np.searchsorted(bins["uvcrd"], u, side="left") - 1).reshape(-1), minlength=len(bins["uvcrd"]))
    for _ in range(3):
        np.testing.assert_array_equal(gpu.accum()["edens"], count)
        gpu.engclear()
        gpu.placements(tag, pl)
    gpu.close()
