"""The finish kernel's sums of FP32 pair terms (GPU, mixed path, against the oracle): terms far below
a kcal/mol keep their bits, in molecules whose pairs are few and in those whose pairs are many, and
many terms just below the largest that is summed in FP32 do not overflow."""
import numpy as np
import pytest

from ermod_gb300 import setconf, synth
from tests import helpers

pytestmark = pytest.mark.gpu

SCALE = 1.0e-5  # of every charge: energies of 1e-10 of their size


@pytest.mark.parametrize("big", [0, 300])
def test_small_terms(gpu_lib, oracle, big):
    """Charges alone.  Bound: the mixed band (twice it: close pairs run in FP32 here too, 4e-7 of some
    70 kcal/mol), grown as the square root of a molecule's sites beyond three, at this scale; and a
    unit of 2^-51 (2^-58 for many pairs) for each pair."""
    from ermod_gb300.engproc import EnergyRepresentation
    rng = np.random.default_rng(12)
    box, sol = 26.0, synth.methanol_like()
    w = synth.Workload("small", "soln", box, 400, sol, synth._params(1, 32, corrcal=0, wgtslf=0), 5, 1, 1, 9, cavity=4.5)
    pos, cell = w.frame(0)
    species = [dict(count=400, sluvid=0, charge=SCALE * np.array(synth.WATER_CHARGE), eps=np.zeros(3), len=np.full(3, 3.0))]
    if big:  # one molecule of the cavity's surroundings
        x = rng.uniform(0.0, box, (4 * big, 3))
        x = x[np.linalg.norm(x - box / 2, axis=1) > 5.5][:big]
        assert len(x) == big
        pos = np.concatenate([x, pos])
        species.insert(0, dict(count=1, sluvid=0, charge=SCALE * rng.choice([-0.5, 0.5], big), eps=np.zeros(big),
                               len=np.full(big, 3.0)))
    ns = len(sol["charge"])
    species.append(dict(count=1, sluvid=1, charge=SCALE * np.asarray(sol["charge"]), eps=np.zeros(ns), len=np.full(ns, 3.0)))
    topo = setconf.setparam_topology(species, slttype=1)
    bins = setconf.enginit_bins(topo["numslv"], setconf.HIST_DEFAULT)
    gpu = EnergyRepresentation(w.params, topo, bins, precision="mixed")
    orc = oracle.Oracle(w.params, topo, bins)
    gpu.frame(pos, cell)
    orc.frame(pos, cell)
    ug = gpu.placements([topo["nummol"]], want_uvengy=True)["uvengy"][0, 1:]
    uo = orc.placements([topo["nummol"]])["uvengy"][0, 1:]
    gpu.close()
    sites = np.array([big] * (1 if big else 0) + [3] * 400 + [ns])
    unit = 2.0 ** -58 if big else 2.0 ** -51
    tol = 2 * helpers.MIXED_BAND * SCALE ** 2 * np.sqrt(sites / 3.0) + sites * ns * unit / 2
    assert np.abs(uo).max() > 5.0e-11
    err = np.abs(ug - uo)
    assert np.all(err <= tol), (err / tol).max()


def test_large_sums(gpu_lib, oracle):
    """128 x 256 pairs of 14 to 16 (Coulomb) and 1 to 8 kcal/mol (LJ): 6e5 together, above 2^19.
    Bound: 1e-6, some ten times the FP32 rounding of a term."""
    from ermod_gb300.engproc import EnergyRepresentation
    rng = np.random.default_rng(3)

    def ball(n, centre):
        v = rng.normal(size=(n, 3))
        return centre + 0.28 * v / np.linalg.norm(v, axis=1)[:, None] * rng.uniform(0.0, 1.0, (n, 1))

    q = np.sqrt(14.8 * 10.0) / 18.22261721  # the charge unit of the topology
    solv, solu = ball(128, np.array([10.0, 0.0, 0.0])), ball(256, np.zeros(3))
    d = np.linalg.norm(solv[:, None] - solu[None], axis=2)
    co, lj = 148.0 / d, 4 * 0.1475 * ((12.0 / d) ** 12 - (12.0 / d) ** 6)
    assert co.max() < 16.0 and lj.max() < 8.0 and (co + lj).sum() > 2.0 ** 19
    species = [dict(count=1, sluvid=0, charge=np.full(128, q), eps=np.full(128, 0.1475), len=np.full(128, 12.0)),
               dict(count=1, sluvid=2, charge=np.full(256, q), eps=np.full(256, 0.1475), len=np.full(256, 12.0))]
    topo = setconf.setparam_topology(species, slttype=2)
    bins = setconf.enginit_bins(topo["numslv"], dict(setconf.HIST_DEFAULT, ecdmin=-2.0e6, eccore=2.0e6, eclbin=1000.0))
    params = dict(synth.droplet().params, slttype=2, lwljcut=14.0, upljcut=16.0)
    pos = np.concatenate([solv, solu])
    gpu = EnergyRepresentation(params, topo, bins, precision="mixed")
    orc = oracle.Oracle(params, topo, bins)
    cell = np.zeros((3, 3))
    gpu.frame(pos, cell)
    orc.frame(pos, cell)
    ug = gpu.placements([topo["nummol"]], solu[None], want_uvengy=True)["uvengy"][0, 1]
    uo = orc.placements([topo["nummol"]], solu[None])["uvengy"][0, 1]
    gpu.close()
    assert uo > 2.0 ** 19
    assert ug == pytest.approx(uo, rel=1e-6)


@pytest.mark.parametrize("nsolute,nsolv,ncount", [(6, 240, 20), (17, 200, 20)])
def test_many_pairs_in_groups(gpu_lib, oracle, nsolute, nsolv, ncount):
    """Molecules of so many sites that the sums take three words, in blocks of one to eight placements."""
    from tests import test_near_pairs_gpu
    test_near_pairs_gpu.test_pairs_against_oracle(gpu_lib, oracle, nsolute, 2.5, nsolv, ncount)
