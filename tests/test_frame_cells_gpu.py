"""The frame's spatial sort where the molecules fill few of the box's cells, or cells that are many along
one axis (GPU, against the oracle): a cluster of molecules with one far away, sorted by counting with
most of them in one code, and by radix sort; boxes much longer along one axis, with a layer of
liquid or full of it."""
import numpy as np
import pytest

from ermod_gb300 import setconf, synth
from tests import helpers

pytestmark = pytest.mark.gpu


def _check(oracle, params, cell, waters, precision):
    """waters: the frames of one run, each (n, 3)."""
    from ermod_gb300.engproc import EnergyRepresentation
    sol = synth.methanol_like()
    n = len(waters[0])
    perm = np.random.default_rng(1).permutation(n)
    frames = [np.concatenate([(x[perm, None] + synth.water_body()).reshape(-1, 3), sol["xyz"] + cell.diagonal() / 2])
              for x in waters]
    species = [dict(count=n, sluvid=0, charge=synth.WATER_CHARGE, eps=synth.WATER_EPS, len=synth.WATER_SIG),
               dict(count=1, sluvid=1, charge=sol["charge"], eps=sol["eps"], len=sol["sig"])]
    topo = setconf.setparam_topology(species, slttype=1)
    bins = setconf.enginit_bins(topo["numslv"], dict(setconf.HIST_DEFAULT, ecdmin=-1.0e4, eccore=1.0e4, eclbin=50.0))
    gpu = EnergyRepresentation(params, topo, bins, precision=precision)
    orc = oracle.Oracle(params, topo, bins)
    for pos in frames:
        orc.frame(pos, cell)
        uo = orc.placements([topo["nummol"]])["uvengy"][0, 1:]
        gpu.frame(pos, cell)
        ug = gpu.placements([topo["nummol"]], want_uvengy=True)["uvengy"][0, 1:]
        helpers.check_energies(ug, uo, precision, f"{n} waters")
    a = gpu.accum()
    np.testing.assert_allclose(a["edens"].sum(), a["engnorm"] * n, rtol=1e-12)
    gpu.close()


def _ball(n):
    m = int(np.ceil((2.2 * n) ** (1 / 3))) + 2
    g = (np.arange(m) - m / 2) * 3.107
    pts = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    r = np.linalg.norm(pts, axis=1)
    return pts[np.argsort(r, kind="stable")][r[np.argsort(r, kind="stable")] > 5.0][:n]


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("n,far", [(300, 40.0), (2500, 1000.0), (3500, 1000.0), (9500, 1000.0)])
def test_cluster_and_one_far_molecule(gpu_lib, oracle, precision, n, far):
    near = _ball(n)
    water = near.copy()
    water[n // 2] = [far, 0.0, 0.0]
    # the molecule comes and goes: a frame's way of sorting is its own
    _check(oracle, dict(synth.droplet().params), np.zeros((3, 3)), [near, water, water, near], precision)


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("box,grid,layers", [((30.0, 30.0, 300.0), (32, 32, 150), 20), ((300.0, 30.0, 30.0), (150, 32, 32), 9),
                                             ((30.0, 30.0, 600.0), (27, 27, 250), 185)])
def test_long_boxes(gpu_lib, oracle, precision, box, grid, layers):
    nx, ny = (96, 9) if box[0] > 100 else (9, 9)
    g = np.stack(np.meshgrid((np.arange(nx) + 0.5) * box[0] / nx, (np.arange(ny) + 0.5) * box[1] / ny,
                             (np.arange(layers) + 0.5) * 3.2, indexing="ij"), -1).reshape(-1, 3)
    water = g[np.linalg.norm(g - np.array(box) / 2, axis=1) > 5.0]
    params = dict(synth._params(1, 32, corrcal=0, wgtslf=0), ms1max=grid[0], ms2max=grid[1], ms3max=grid[2])
    _check(oracle, params, np.diag(box), [water, water], precision)
