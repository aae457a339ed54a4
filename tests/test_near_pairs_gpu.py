"""The finish kernel's real-space pass at its edges (GPU, against the oracle): more FP64 pairs in a
block than its list holds (a 200-site solute compressed into water), solvent molecules of more
than three sites, solutes of one site, and energies that do not depend on the batch, the
finish group or the tile."""
import numpy as np
import pytest

from ermod_gb300 import setconf, synth
from tests import helpers

pytestmark = pytest.mark.gpu

HIST = dict(setconf.HIST_DEFAULT, ecdmin=-1.0e5, eclbin=50.0, eccore=200.0)


def _solute(n, spread, seed):
    rng = np.random.default_rng(seed)
    q = rng.normal(0.0, 0.3, n)
    return dict(xyz=rng.uniform(-spread, spread, (n, 3)), charge=q - q.mean(), sig=rng.uniform(2.5, 3.5, n),
                eps=rng.uniform(0.05, 0.2, n), mass=np.full(n, 12.0))


def _chain(n, count, box, seed):
    """count solvent molecules of n sites on a lattice, n x 1.3 A long at most."""
    rng = np.random.default_rng(seed)
    m = int(np.ceil(count ** (1 / 3)))
    g = (np.arange(m) + 0.5) * box / m
    c = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)[:count]
    return (c[:, None] + rng.uniform(-1.0, 1.0, (count, n, 3))).reshape(-1, 3)


@pytest.mark.parametrize("nsolute,spread,nsolv,ncount", [(200, 3.0, 3, 600), (1, 0.0, 3, 300), (17, 2.5, 7, 150),
                                                         (40, 4.0, 1, 700)])
def test_pairs_against_oracle(gpu_lib, oracle, nsolute, spread, nsolv, ncount):
    from ermod_gb300.engproc import EnergyRepresentation
    rng = np.random.default_rng(nsolute)
    sol = _solute(nsolute, spread, nsolute)
    box = 26.0
    sq = rng.normal(0.0, 0.2, nsolv)
    species = [dict(count=ncount, sluvid=0, charge=sq - sq.mean(), eps=np.full(nsolv, 0.1), len=np.full(nsolv, 3.0)),
               dict(count=1, sluvid=2, charge=sol["charge"], eps=sol["eps"], len=sol["sig"])]
    topo = setconf.setparam_topology(species, slttype=2)
    bins = setconf.enginit_bins(topo["numslv"], HIST)
    params = synth._params(2, 32, corrcal=0, wgtslf=0)
    pos = np.concatenate([_chain(nsolv, ncount, box, 3), sol["xyz"] + box / 2])
    cell = np.diag([box] * 3)
    n = 9
    pl = sol["xyz"] + rng.uniform(0.0, box, (n, 1, 3))
    tag = np.full(n, topo["nummol"], np.int32)
    orc = oracle.Oracle(params, topo, bins)
    orc.frame(pos, cell)
    uo = orc.placements(tag, pl)["uvengy"][:, 1:]
    first = None
    for kw in (dict(), dict(batch=4), dict(batch=8, finish_group=8), dict(finish_group=4)):
        gpu = EnergyRepresentation(params, topo, bins, precision="mixed", **kw)
        gpu.frame(pos, cell)
        ug = gpu.placements(tag, pl, want_uvengy=True)["uvengy"][:, 1:]
        helpers.check_energies(ug, uo, "mixed", str(kw), band=_band(sol, sq, nsolv))
        if first is None:
            first = ug
        np.testing.assert_array_equal(ug, first)
        gpu.close()


def _band(sol, sq, nsolv):
    """helpers.mixed_band, grown with the square root of the pair terms a molecule sums in FP32
    against a 12-site solute's 36, each rounded by itself."""
    return helpers.mixed_band(sol) * max(1.0, np.sqrt(len(sol["charge"]) * nsolv / 36.0))
