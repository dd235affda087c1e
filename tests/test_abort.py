"""dpg_set_abort during a call: the check kernel's warps poll the flag while
they draw work items, so a call whose flag is raised from another host thread
ends early with DPG_ERR_ABORTED, and the context works as before afterwards."""
import threading
import time

import numpy as np
import pytest

from dynoplan_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant", [0, 1])  # lockstep, slots
def test_abort_raised_during_a_call(dpg_lib, variant):
    from dynoplan_gb300 import _lib
    from dynoplan_gb300 import gpu as G
    wl = W.make_workload(3, seed=77, N=4000, P=1500)
    cap = int(0.25 * 4000 * 1500)
    with G.Context(wl.robot) as ctx:
        ctx.upload_primitives(wl.prims)
        ctx.upload_env(wl.env)
        ctx.set_tuning(check_variant=variant, host_output=0, pipe_launches=1)
        out = dict(node=np.empty(cap, np.uint32), prim=np.empty(cap, np.uint32), verdict=np.empty(cap, np.uint8))
        before = ctx.expand(wl.nodes, wl.radius, outputs=out, capacity=cap)["verdict"].copy()
        t0 = time.perf_counter()
        ctx.expand(wl.nodes, wl.radius, outputs=out, capacity=cap)
        call = time.perf_counter() - t0
        seen = ""
        for i in range(200):  # raised at times spread over the call
            timer = threading.Thread(target=lambda d=call * (i % 20) / 20: (time.sleep(d), ctx.set_abort(True)))
            timer.start()
            try:
                ctx.expand(wl.nodes, wl.radius, outputs=out, capacity=cap)
            except _lib.DpgError as e:
                assert e.code == _lib.DPG_ERR_ABORTED
                seen = str(e)
            timer.join()
            ctx.set_abort(False)
            if seen.endswith("expand: aborted"):  # (not the check of the flag on entry)
                break
        assert seen.endswith("expand: aborted"), seen
        after = ctx.expand(wl.nodes, wl.radius, outputs=out, capacity=cap)["verdict"]
        np.testing.assert_array_equal(before, after)
