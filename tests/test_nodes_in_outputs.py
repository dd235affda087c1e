"""Device nodes that lie in an output array of the call (a planner that expands rows
of the last call's end states into the same buffer), and nodes that are not
8-byte aligned: results equal those from an array of their own."""
import numpy as np
import pytest

from dynoplan_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def _outs(torch, cap, nx, prec):
    es = torch.zeros(cap * nx, dtype=torch.float64 if prec else torch.float32, device="cuda")
    return {"node": torch.zeros(cap, dtype=torch.int32, device="cuda"), "prim": torch.zeros(cap, dtype=torch.int32, device="cuda"),
            "verdict": torch.zeros(cap, dtype=torch.uint8, device="cuda"), "end_state": es}


@pytest.mark.parametrize("cfg", [1, 2, 5])
@pytest.mark.parametrize("N", [64, 1000, 2500])  # two ball kernels; node tiles; spatial order
@pytest.mark.parametrize("prec", [0, 1, 2])
def test_nodes_in_the_end_states(dpg_lib, cfg, N, prec):
    torch = pytest.importorskip("torch")
    from dynoplan_gb300 import gpu as G
    wl = W.make_workload(cfg, seed=60 + cfg, N=N, P=300)
    with G.Context(wl.robot) as ctx:
        ctx.upload_primitives(wl.prims)
        ctx.upload_env(wl.env)
        cap = 300 * N
        ref = _outs(torch, cap, ctx.nx, prec)
        x = torch.from_numpy(wl.nodes).cuda()
        r = ctx.expand_device(x.data_ptr(), N, 0.6, {k: t.data_ptr() for k, t in ref.items()}, cap, precision=prec)
        assert r["n_pairs"] > 2 * N
        got = _outs(torch, cap, ctx.nx, prec)
        inside = got["end_state"].view(torch.float64)[:N * ctx.nx]
        inside.copy_(x.reshape(-1))
        torch.cuda.synchronize()
        q = ctx.expand_device(inside.data_ptr(), N, 0.6, {k: t.data_ptr() for k, t in got.items()}, cap, precision=prec)
        assert q == r
        n = r["n_pairs"]
        for k in ref:
            m = n * (ctx.nx if k == "end_state" else 1)
            assert torch.equal(ref[k][:m], got[k][:m]), k


@pytest.mark.parametrize("N", [64, 1000, 2500])
def test_nodes_not_aligned(dpg_lib, N):
    torch = pytest.importorskip("torch")
    from dynoplan_gb300 import gpu as G
    wl = W.make_workload(2, seed=71, N=N, P=300)
    with G.Context(wl.robot) as ctx:
        ctx.upload_primitives(wl.prims)
        ctx.upload_env(wl.env)
        cap = 300 * N
        raw = torch.from_numpy(np.concatenate([np.zeros(4, np.uint8), wl.nodes.reshape(-1).view(np.uint8)])).cuda()
        x = torch.from_numpy(wl.nodes).cuda()
        a, b = _outs(torch, cap, ctx.nx, 0), _outs(torch, cap, ctx.nx, 0)
        torch.cuda.synchronize()
        ra = ctx.expand_device(x.data_ptr(), N, 0.6, {k: t.data_ptr() for k, t in a.items()}, cap)
        rb = ctx.expand_device(raw.data_ptr() + 4, N, 0.6, {k: t.data_ptr() for k, t in b.items()}, cap)
        assert ra == rb and ra["n_pairs"] > N
        for k in a:
            m = ra["n_pairs"] * (ctx.nx if k == "end_state" else 1)
            assert torch.equal(a[k][:m], b[k][:m]), k
