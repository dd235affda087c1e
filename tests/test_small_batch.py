"""Small batches (dpg_expand's two-kernel ball stage and its mapped inputs and
results) against dpg_expand_noalloc, which tests every (node, primitive) pair
in node tiles: the same pairs in the same order and the same results, bit for
bit, at the edges of the kernels' words (32 nodes), blocks (128 and 256
primitives) and of the batch limit (128 nodes)."""
import ctypes as C

import numpy as np
import pytest

from dynoplan_gb300 import workloads as W

pytestmark = pytest.mark.gpu

FIELDS = ["node", "prim", "verdict", "first_invalid", "end_state", "min_gap", "flags"]
EXTENT = {W.UNICYCLE1: (6.0, 6.0), W.CAR1: (10.0, 10.0), W.QUAD2D: (8.0, 4.0), W.QUAD3D: (6.0, 6.0, 3.0)}


def _noalloc(torch, ctx, x, radius, prec, cap, mode=0):
    from dynoplan_gb300 import _lib
    dt = {"node": torch.int32, "prim": torch.int32, "verdict": torch.uint8, "first_invalid": torch.int16,
          "min_gap": torch.float32, "flags": torch.uint8}
    dev = {k: torch.zeros(cap, dtype=t, device="cuda") for k, t in dt.items()}
    dev["end_state"] = torch.zeros((cap, ctx.nx), dtype=torch.float64 if prec else torch.float32, device="cuda")
    xd = torch.from_numpy(x).cuda()
    opts = _lib.ExpandOpts(radius=radius, precision=prec, x_on_device=1, out_on_device=1, mode=mode, contact_band=1e-4,
                           ball_band=1e-5)
    out = _lib.ExpandOut(capacity=cap)
    for k, t in dev.items():
        setattr(out, k, C.c_void_p(t.data_ptr()))
    _lib.check(_lib.load().dpg_expand_noalloc(ctx.h, C.byref(opts), len(x), C.c_void_p(xd.data_ptr()), C.byref(out)), ctx.h)
    n = int(out.n_pairs)
    return xd, n, {k: t[:n].cpu().numpy() for k, t in dev.items()}, int(out.n_ball_recheck)


def _same(ref, n, got, fields=FIELDS):
    assert got["n_pairs"] == n
    for k in fields:
        np.testing.assert_array_equal(ref[k].view(got[k].dtype) if ref[k].dtype != got[k].dtype else ref[k], got[k], err_msg=k)


@pytest.mark.parametrize("kind,radius", [(W.UNICYCLE1, 0.4), (W.CAR1, 0.5), (W.QUAD2D, 0.8), (W.QUAD3D, 0.5)])
@pytest.mark.parametrize("N,P", [(1, 1), (1, 300), (31, 127), (32, 128), (33, 129), (64, 256), (127, 257), (128, 700), (129, 300)])
def test_small_batch(dpg_lib, kind, radius, N, P):
    torch = pytest.importorskip("torch")
    from dynoplan_gb300 import gpu as G
    m = W.robot_model(kind)
    prims = W.make_primitives(m, P, 3, 40, seed=N + P)
    env = W.make_env(EXTENT[kind], 25, 0.2, 1.0, seed=N + P + 1)
    x = W.make_nodes(m, env, N, seed=N + P + 2)
    prec = (N + P) % 2
    with G.Context(m) as ctx:
        ctx.upload_primitives(prims)
        ctx.upload_env(env)
        xd, n, ref, rechecks = _noalloc(torch, ctx, x, radius, prec, N * P + 1)
        got = ctx.expand(x, radius, precision=prec, capacity=N * P + 1)  # results through mapped memory when they fit
        _same(ref, n, got)
        assert got["n_ball_recheck"] == rechecks
        got = ctx.expand(x, radius, precision=prec, capacity=max(n, 1))  # the capacity just right
        _same(ref, n, got)
        # some outputs left out; results on the device; the ball alone
        part = dict(node=np.empty(N * P + 1, np.uint32), prim=np.empty(N * P + 1, np.uint32), verdict=np.empty(N * P + 1, np.uint8))
        _same(ref, n, ctx.expand(x, radius, precision=prec, capacity=N * P + 1, outputs=part), ["node", "prim", "verdict"])
        dev = {k: torch.zeros(N * P + 1, dtype=t, device="cuda") for k, t in
               (("node", torch.int32), ("prim", torch.int32), ("verdict", torch.uint8), ("flags", torch.uint8))}
        r = ctx.expand_device(xd.data_ptr(), N, radius, {k: t.data_ptr() for k, t in dev.items()}, N * P + 1, precision=prec)
        _same(ref, n, {"n_pairs": r["n_pairs"], **{k: t[:n].cpu().numpy() for k, t in dev.items()}}, list(dev))
        got = ctx.expand(x, radius, ball_only=True, capacity=N * P + 1)
        _same(ref, n, got, ["node", "prim"])
        if n > 1:
            from dynoplan_gb300 import _lib
            with pytest.raises(_lib.DpgError) as e:
                ctx.expand(x, radius, capacity=n - 1, outputs=part)
            assert e.value.code == _lib.DPG_ERR_CAPACITY


def test_small_batch_equals_its_part_of_a_large_one(dpg_lib):
    """Results past the mapped buffer's size, and copied in ranges."""
    from dynoplan_gb300 import gpu as G
    m = W.robot_model(W.QUAD2D)
    prims = W.make_primitives_hover(m, 9000, 20, 60, seed=4)
    env = W.make_env((8.0, 4.0), 40, 0.2, 1.0, seed=5)
    x = W.make_nodes(m, env, 1500, seed=6, vel_sigma=0.2)
    x[:, 2] *= 0.1
    with G.Context(m) as ctx:
        ctx.upload_primitives(prims)
        ctx.upload_env(env)
        a = ctx.expand(x, 0.25, capacity=1500 * 9000)  # node tiles, copied in ranges
        for n in (40, 128):
            b = ctx.expand(x[:n], 0.25, capacity=n * 9000)
            k = a["node"] < n
            assert b["n_pairs"] == k.sum() > 100000
            for f in FIELDS:
                np.testing.assert_array_equal(a[f][k], b[f], err_msg=f)
