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


@pytest.mark.parametrize("host_output,launches", [(2, 8), (0, 8)])  # copy ranges flagged by the check; launches on two streams
def test_abort_with_results_copied_in_ranges(dpg_lib, host_output, launches):
    from dynoplan_gb300 import _lib
    from dynoplan_gb300 import gpu as G
    wl = W.make_workload(3, seed=78, N=6000, P=2000)
    with G.Context(wl.robot) as ctx:
        ctx.upload_primitives(wl.prims)
        ctx.upload_env(wl.env)
        ctx.set_tuning(host_output=host_output, pipe_launches=launches)
        cap = ctx.expand(wl.nodes, wl.radius, ball_only=True, capacity=6000 * 2000)["n_pairs"]
        out = dict(node=np.empty(cap, np.uint32), prim=np.empty(cap, np.uint32), verdict=np.empty(cap, np.uint8),
                   end_state=np.empty((cap, ctx.nx), np.float32))
        _abort_in_call(_lib, ctx, lambda: ctx.expand(wl.nodes, wl.radius, outputs=out, capacity=cap), "verdict")


@pytest.mark.parametrize("precision", [0, 2])  # slots, lockstep walk
def test_abort_is_seen_by_the_last_items(dpg_lib, precision):
    """About 1.5 work items a warp, milliseconds each: every warp's second item
    is drawn when the launch begins, so a flag read only with the draw would
    never be seen.  Robots that stand still on a grid, obstacles on the cells'
    corners (none is touched, all lie between the nodes of an item)."""
    from dynoplan_gb300 import _lib
    from dynoplan_gb300 import gpu as G
    torch = pytest.importorskip("torch")
    m = W.robot_model(W.UNICYCLE1)
    warps = 8 * torch.cuda.get_device_properties(0).multi_processor_count  # a block of eight warps an SM
    N, L = 960, (30000 if precision == 0 else 100)
    P = int(1.5 * warps) // (N // 32)
    prims = W.Primitives(np.full(P, L, np.int32), np.zeros((P * L, 3)), np.zeros((P * (L - 1), 2)))
    at = np.stack(np.meshgrid(np.arange(22.0), np.arange(23.0), indexing="ij"), -1).reshape(-1, 2) * 4
    env = W.Env(np.array([-1e3, -1e3]), np.array([1e3, 1e3]), at + 1.9, at + 2.1)
    x = np.zeros((N, 3))
    x[:, :2] = at[np.random.default_rng(4).integers(0, len(at), N)]
    with G.Context(m) as ctx:
        ctx.upload_primitives(prims)
        ctx.upload_env(env)
        ctx.set_tuning(check_blocks_per_sm=1)
        out = dict(node=np.empty(N * P, np.uint32), prim=np.empty(N * P, np.uint32), verdict=np.empty(N * P, np.uint8))
        _abort_in_call(_lib, ctx, lambda: ctx.expand(x, 1e3, outputs=out, capacity=N * P, precision=precision), "verdict",
                       span=(0.15, 0.5))


def _abort_in_call(_lib, ctx, call, field, span=(0.0, 1.0)):
    """Raises the flag at times spread over `span` of a call until one ends early;
    then the context works as before."""
    before = call()[field].copy()
    t0 = time.perf_counter()
    call()
    took = time.perf_counter() - t0
    seen = ""
    for i in range(60):
        delay = took * (span[0] + (span[1] - span[0]) * (i % 20) / 20)
        timer = threading.Thread(target=lambda: (time.sleep(delay), ctx.set_abort(True)))
        timer.start()
        try:
            call()
        except _lib.DpgError as e:
            assert e.code == _lib.DPG_ERR_ABORTED
            seen = str(e)
        timer.join()
        ctx.set_abort(False)
        if seen.endswith("expand: aborted"):
            break
    assert seen.endswith("expand: aborted"), (seen, took)
    np.testing.assert_array_equal(before, call()[field])
