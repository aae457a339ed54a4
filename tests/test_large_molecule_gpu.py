"""A solvent molecule of more than 8,192 sites beside small ones (GPU, against the oracle): the
finish kernel's queued pairs name a site within a window of 8,192, so sites on both sides of the
windows' edges interact here, among them overlapping ones (the FP64 list), at equal offsets in
two windows."""
import numpy as np
import pytest

from ermod_gb300 import setconf, synth
from tests import helpers

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_sites_beyond_one_window(gpu_lib, oracle, precision):
    from ermod_gb300.engproc import EnergyRepresentation
    rng = np.random.default_rng(8)
    n, box = 8500, 60.0
    g = (np.arange(21) + 0.5) * box / 21
    pts = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    rng.shuffle(pts)
    big = pts[:n] + rng.uniform(-0.2, 0.2, (n, 3))
    big[8192 + 37] = big[37] + [0.4, 0.0, 0.0]  # the same offset in both windows
    q = np.zeros(n)
    q[[0, 1000, 4000, 8191, 8192, 8300]] = [0.4, -0.4, 0.3, -0.3, 0.5, -0.5]
    eps = np.where(np.arange(n) % 37 == 0, 0.1, 0.0)
    eps[[8191, 8192, 8192 + 37]] = 0.1
    sol = synth.methanol_like()
    nw = 40
    wq = np.array([-0.8, 0.4, 0.4])
    wat = pts[n:n + nw][:, None] + rng.uniform(-0.7, 0.7, (nw, 3, 3))
    species = [dict(count=1, sluvid=0, charge=q, eps=eps, len=np.full(n, 2.5)),
               dict(count=nw, sluvid=0, charge=wq, eps=[0.15, 0.0, 0.0], len=[3.1, 0.0, 0.0]),
               dict(count=1, sluvid=2, charge=sol["charge"], eps=sol["eps"], len=sol["sig"])]
    topo = setconf.setparam_topology(species, slttype=2)
    bins = setconf.enginit_bins(topo["numslv"], dict(setconf.HIST_DEFAULT, ecdmin=-1.0e5, eclbin=50.0, eccore=200.0))
    params = synth._params(2, 60, corrcal=0, wgtslf=0)
    s0 = sol["xyz"] - sol["xyz"].mean(0)
    pos = np.concatenate([big, wat.reshape(-1, 3), s0 + box / 2])
    cell = np.diag([box] * 3)
    at = [big[37], big[8192 + 37], big[8191], big[8192], big[8300], big[4000]]
    pl = np.stack([s0 + x + rng.uniform(0.3, 1.2, 3) for x in at])
    tag = np.full(len(pl), topo["nummol"], np.int32)
    orc = oracle.Oracle(params, topo, bins)
    orc.frame(pos, cell)
    uo = orc.placements(tag, pl)["uvengy"][:, 1:]
    gpu = EnergyRepresentation(params, topo, bins, precision=precision)
    gpu.frame(pos, cell)
    ug = gpu.placements(tag, pl, want_uvengy=True)["uvengy"][:, 1:]
    gpu.close()
    # twice the charged sites of a water molecule
    helpers.check_energies(ug, uo, precision, "8,500 sites", band=2 * helpers.MIXED_BAND if precision == "mixed" else None)
