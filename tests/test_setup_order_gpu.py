"""Set-up memory is ready before the kernels that use it, whatever else the process has queued on
the legacy default stream (torch's default stream): the batch buffers made by a context's first
call, the counts and accumulators made by set-up calls in either order."""
import numpy as np
import pytest

from tests import helpers

pytestmark = pytest.mark.gpu


def _backlog(torch, ms):
    """About ms milliseconds of work on the legacy default stream, without waiting for it."""
    a = torch.randn(4096, 4096, device="cuda")
    b = torch.empty_like(a)
    t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    for timed in (False, True):
        t0.record()
        torch.matmul(a, a, out=b)
        t1.record()
        t1.synchronize()
    for _ in range(max(1, int(ms / t0.elapsed_time(t1)))):
        torch.matmul(a, a, out=b)


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("order", ["bins last", "topology last"])
def test_first_calls_beside_a_busy_default_stream(gpu_lib, precision, order):
    import torch
    from ermod_gb300 import _lib
    from ermod_gb300.engproc import EnergyRepresentation
    w = helpers.small_refs(nwater=700, corrcal=1, wgtslf=1)
    topo, bins = helpers.build_inputs(w, dict(helpers.setconf.HIST_DEFAULT, ecdmin=-200.0))
    pos, cell = w.frame(0)
    pl = w.placements(0, 300)
    tag = np.full(len(pl), topo["nummol"], np.int32)
    ref = EnergyRepresentation(w.params, topo, bins, precision=precision)
    ref.frame(pos, cell)
    want = ref.placements(tag, pl, want_uvengy=True)["uvengy"]
    torch.cuda.synchronize()
    _backlog(torch, 20.0)
    gpu = EnergyRepresentation(w.params, topo, bins, precision=precision)
    if order == "topology last":
        gpu.set_topology(topo)
    _backlog(torch, 60.0)  # behind the set-up calls, before the first frame and call
    gpu.frame(pos, cell)
    calls = 0
    busy = torch.cuda.Event()
    busy.record()
    while calls < 3 or (not busy.query() and calls < 400):
        np.testing.assert_array_equal(gpu.placements(tag, pl, want_uvengy=True)["uvengy"], want)
        calls += 1
    for _ in range(calls - 1):
        ref.placements(tag, pl)
    a, b = gpu.accum(), ref.accum()
    for k in ("edens", "ecorr", "slnuv", "minuv", "maxuv"):
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)
    assert a["engnorm"] == b["engnorm"] and a["engsmpl"] == b["engsmpl"]
    ref.close()
    gpu.close()
