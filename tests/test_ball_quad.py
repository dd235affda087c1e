"""The quadrotor's ball scan decides most pairs from an approximate distance: the
same pairs and the same number of FP64 decisions as batches of at most 128
nodes, which take the exact FP32 distance throughout, and the oracle's pairs.
Primitive counts around groups of 4 and 32 and the tile of 256, node counts
around a warp and a block, quaternions of other norms, a primitive's own start,
NaN and infinite components (exact: no tolerance)."""
import numpy as np
import pytest

import oracle_bind as ob
from dynoplan_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def pairs(r, shift=0):
    return (r["node"].astype(np.int64) + shift) * (1 << 20) + r["prim"]


@pytest.mark.parametrize("N,P", [(129, 1), (255, 3), (257, 33), (300, 255), (161, 258), (2100, 517)])
@pytest.mark.parametrize("radius", [0.3, 1.0])
def test_ball_quadrotor(dpg_lib, N, P, radius):
    from dynoplan_gb300 import gpu as G
    wl = W.make_workload(3, seed=900 + P, N=N, P=P)
    rng = np.random.default_rng(N)
    x = wl.nodes.copy()
    x[1::7, 3:7] *= rng.uniform(0.3, 2.0, (len(x[1::7]), 1))
    x[2::7, 3:13] = wl.prims.states[0, 3:13]
    odd = x.copy()
    odd[5, 4], odd[40, 11], odd[41, 3], odd[100, 12] = np.nan, np.nan, np.inf, -np.inf
    with G.Context(wl.robot) as ctx:
        ctx.upload_primitives(wl.prims)
        ctx.upload_env(wl.env)
        for nodes in (x, odd):
            whole = ctx.expand(nodes, radius, ball_only=True)
            parts = [ctx.expand(nodes[s:s + 128], radius, ball_only=True) for s in range(0, N, 128)]
            want = np.concatenate([pairs(r, 128 * k) for k, r in enumerate(parts)])
            np.testing.assert_array_equal(np.sort(pairs(whole)), np.sort(want))
            assert whole["n_ball_recheck"] == sum(r["n_ball_recheck"] for r in parts)
            if nodes is x:
                ora = ob.expand(wl.robot, wl.prims, wl.env, nodes, radius, fast=True, threads=ob.lib().orc_max_threads())
                np.testing.assert_array_equal(np.sort(pairs(whole)), np.sort(pairs(ora)))


@pytest.mark.parametrize("w", [(-2e4, 0.5, 1.0, 2e4), (1.0, 0.5, -2e4, 2e4), (1.0, -0.5, 1.0, 1.0), (1.0, 0.5, 1.0, -1.0)])
def test_ball_quadrotor_negative_weights(dpg_lib, w):
    """With a negative weight the terms of the distance may cancel near the radius
    (nodes placed there by the rounding of terms of 1e4): exact distances."""
    import dataclasses

    from dynoplan_gb300 import gpu as G
    N, P, radius = 1000, 64, 1.0
    wl = W.make_workload(3, seed=31, N=N, P=P)
    m = dataclasses.replace(wl.robot, w=w)
    prims = wl.prims
    start = np.concatenate([[0], np.cumsum(prims.length)[:-1]])
    rng = np.random.default_rng(8)
    s = prims.states[start]
    s[:, :3], s[:, 7:10] = rng.uniform(0.3, 1.0, (2, P, 3))  # starts that differ in position and velocity
    prims.states[start] = s
    p = np.arange(N) % P
    x = wl.nodes.copy()
    x[:, 3:13] = s[p, 3:13]  # the orientation is the primitive's: acos 0
    kc = w[0] * np.linalg.norm(s[p, :3], axis=1) + w[2] * np.linalg.norm(s[p, 7:10], axis=1)
    gap = np.maximum((radius + rng.uniform(-4e-3, 4e-3, N) - kc) / w[3], 0.0)
    x[:, 10] += gap
    with G.Context(m) as ctx:
        ctx.upload_primitives(prims)
        ctx.upload_env(wl.env)
        whole = ctx.expand(x, radius, ball_only=True, capacity=N * P)
        parts = [ctx.expand(x[i:i + 128], radius, ball_only=True, capacity=N * P) for i in range(0, N, 128)]
        want = np.concatenate([pairs(r, 128 * k) for k, r in enumerate(parts)])
        np.testing.assert_array_equal(np.sort(pairs(whole)), np.sort(want))
        assert whole["n_ball_recheck"] == sum(r["n_ball_recheck"] for r in parts)
