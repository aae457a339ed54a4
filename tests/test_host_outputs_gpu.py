"""What a host call returns (GPU): energies and flceng of calls whose outputs just fit the pinned staging and
the kept workspace, and of one placement more and one fewer, in any order; and solution mode's
energies, which do not depend on the molecules per finish block, at the system sizes where that
number changes."""
import numpy as np
import pytest

from ermod_gb300 import setconf, synth
from tests import helpers

pytestmark = pytest.mark.gpu


def test_output_sizes(gpu_lib):
    from ermod_gb300.engproc import EnergyRepresentation
    # 2,046 waters: a placement returns its self energy, 2,046 energies and one flceng
    w = helpers.small_refs(nwater=2046, box=40.0, K=40, corrcal=0, wgtslf=0, lattice=13)
    topo, bins = helpers.build_inputs(w, dict(setconf.HIST_DEFAULT, ecdmin=-400.0))
    staged, kept = (256 << 10) // 8 // 2048, (8 << 20) // 2048
    n = kept + 1
    rng = np.random.default_rng(6)
    pl = w.placements(0, 64)[rng.integers(0, 64, n)] + rng.uniform(0.0, 40.0, (n, 1, 3))
    tag = np.full(n, topo["nummol"], np.int32)
    gpu = EnergyRepresentation(w.params, topo, bins, precision="mixed")
    gpu.frame(*w.frame(0))
    want, sums = np.empty((n, 2047)), np.empty((n, 1))
    for p0 in range(0, n, 100):
        r = gpu.placements(tag[p0:p0 + 100], pl[p0:p0 + 100], want_uvengy=True, want_flceng=True)
        want[p0:p0 + 100], sums[p0:p0 + 100] = r["uvengy"], r["flceng"]
    # flceng: float-float totals, summed in FP64
    np.testing.assert_allclose(sums[:, 0], want[:, 1:].sum(1), rtol=1e-12, atol=1e-9 * np.abs(want[:, 1:]).max())
    for m in (staged, kept, staged + 1, kept + 1, staged - 1, kept - 1):
        r = gpu.placements(tag[:m], pl[:m], want_uvengy=True, want_flceng=True)
        np.testing.assert_array_equal(r["uvengy"], want[:m])
        np.testing.assert_array_equal(r["flceng"], sums[:m])
        r = gpu.placements(tag[:m], pl[:m], want_flceng=True)
        assert r["uvengy"] is None
        np.testing.assert_array_equal(r["flceng"], sums[:m])
    gpu.close()


@pytest.mark.parametrize("per_sm,more", [(16, -1), (16, 0), (16, 1), (192, -1), (192, 0)])
def test_solution_tiles(gpu_lib, oracle, per_sm, more):
    """16 molecules a block up to 16 per SM, 64 below 192 per SM, then 256."""
    import torch
    from ermod_gb300.engproc import EnergyRepresentation
    molecules = per_sm * torch.cuda.get_device_properties(0).multi_processor_count + more
    nwater = molecules - 1  # the solute is a molecule of the frame
    lattice = int(np.ceil((1.04 * nwater + 40) ** (1.0 / 3.0)))
    box = 3.107 * lattice
    w = synth.Workload("tiles", "soln", box, nwater, synth.methanol_like(),
                       synth._params(1, synth.fft_friendly(int(box)), corrcal=0, wgtslf=0), 5, 1, 1, lattice, cavity=4.5)
    topo, bins = helpers.build_inputs(w, dict(setconf.HIST_DEFAULT, ecdmin=-400.0, eccore=400.0, eclbin=0.5))
    pos, cell = w.frame(0)
    orc = oracle.Oracle(w.params, topo, bins)
    orc.frame(pos, cell)
    uo = orc.placements([topo["nummol"]])["uvengy"][:, 1:]
    uv = []
    for group in (0, 4):
        gpu = EnergyRepresentation(w.params, topo, bins, precision="mixed", finish_group=group)
        gpu.frame(pos, cell)
        uv.append(gpu.placements([topo["nummol"]], want_uvengy=True)["uvengy"])
        np.testing.assert_array_equal(
            gpu.accum()["edens"] > 0, np.bincount(helpers.bin_index(uv[-1][0, 1:-1], bins["uvcrd"]), minlength=gpu.ermax) > 0)
        gpu.close()
        helpers.check_energies(uv[-1][:, 1:], uo, "mixed", f"{molecules} molecules, group {group}")
    np.testing.assert_array_equal(uv[0], uv[1])
