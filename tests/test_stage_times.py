"""dpg_last_timings: the stage times of the last call that succeeded, also when a
call that failed came after it."""
import ctypes as C

import numpy as np
import pytest

from dynoplan_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("failing", ["capacity", "pairs"])
def test_times_survive_a_failed_call(dpg_lib, failing):
    torch = pytest.importorskip("torch")
    from dynoplan_gb300 import _lib
    from dynoplan_gb300 import gpu as G
    wl = W.make_workload(3, seed=5, N=4000, P=800)
    with G.Context(wl.robot) as ctx:
        ctx.upload_primitives(wl.prims)
        ctx.upload_env(wl.env)
        xd = torch.from_numpy(wl.nodes).cuda()
        cap = ctx.expand(wl.nodes, wl.radius, ball_only=True, capacity=4000 * 800)["n_pairs"]
        dev = {k: torch.empty(cap, dtype=t, device="cuda") for k, t in
               (("node", torch.int32), ("prim", torch.int32), ("verdict", torch.uint8))}
        ptr = {k: t.data_ptr() for k, t in dev.items()}
        for _ in range(3):
            ctx.expand_device(xd.data_ptr(), len(wl.nodes), wl.radius, ptr, cap)
        want = ctx.timings()
        assert want[0] > 0 and want[1] > 0 and want[3] >= 0
        ctx.expand_device(xd.data_ptr(), len(wl.nodes), wl.radius, ptr, cap)  # (its times are read after the failure)
        with pytest.raises(_lib.DpgError) as e:
            if failing == "capacity":
                ctx.expand_device(xd.data_ptr(), 40, wl.radius, ptr, 1)
            else:  # device lists, an index past the nodes
                bad = torch.tensor([0, 5000], dtype=torch.int32, device="cuda")
                opts = _lib.ExpandOpts(x_on_device=1, out_on_device=1, contact_band=1e-4)
                out = _lib.ExpandOut(capacity=2)
                out.verdict = C.c_void_p(ptr["verdict"])
                _lib.check(dpg_lib.dpg_check_pairs(ctx.h, C.byref(opts), 40, C.c_void_p(xd.data_ptr()), 2,
                                                   C.c_void_p(bad.data_ptr()), C.c_void_p(bad.data_ptr()), C.byref(out)), ctx.h)
        assert e.value.code == (_lib.DPG_ERR_CAPACITY if failing == "capacity" else _lib.DPG_ERR_ARG)
        got = ctx.timings()
        # the same call's times again: stages of some hundred microseconds against the failed call's few
        assert np.all(np.array(got) >= 0) and 0.5 * want[1] < got[1] < 2 * want[1] and got[0] > 0.5 * want[0], (got, want)
