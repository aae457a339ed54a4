"""The ecorr flush beside the batches that follow it (GPU): short batches of few molecules, two to a half
of the ring, on an energy coordinate whose flush takes longer than they do.  With unit weights ecorr
holds exact counts, so one call of many batches equals calls of a single batch each."""
import numpy as np
import pytest

from ermod_gb300 import setconf
from tests import helpers

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch,nplace", [(256, 256 * 14), (0, 256 * 9 + 100), (512, 512 * 7)])
def test_many_batches(gpu_lib, batch, nplace):
    from ermod_gb300.engproc import EnergyRepresentation
    w = helpers.small_refs(nwater=150, box=17.0, K=24, corrcal=1, wgtslf=0, lattice=6)
    w.params["estype"] = 1
    topo = setconf.setparam_topology(w.species(), slttype=2)
    edges = np.concatenate([np.arange(-400.0, -1.0, 0.5), np.linspace(-1.0, 1.0, 3000), np.arange(1.5, 400.0, 0.5), [1.0e11]])
    bins = dict(uvcrd=edges, uvmax=np.array([len(edges)], np.int32), uvsoft=np.array([len(edges) - 1], np.int32),
                escrd=np.array([-1.0e11, 1.0e11]), esmax=2)
    pos, cell = w.frame(0)
    rng = np.random.default_rng(3)
    pl = w.placements(0, 64)[rng.integers(0, 64, nplace)] + rng.uniform(0.0, 17.0, (nplace, 1, 3))
    tag = np.full(nplace, topo["nummol"], np.int32)
    one = batch or 256
    gpu, ref = (EnergyRepresentation(w.params, topo, bins, precision="mixed", batch=b) for b in (batch, one))
    ref.frame(pos, cell)
    for p0 in range(0, nplace, one):
        ref.placements(tag[p0:p0 + one], pl[p0:p0 + one])
    want = ref.accum()["ecorr"]
    gpu.frame(pos, cell)
    for _ in range(2):
        gpu.engclear()
        gpu.placements(tag, pl)
        np.testing.assert_array_equal(gpu.accum()["ecorr"], want)
    gpu.close()
    ref.close()
