"""The slot-parallel exact check against the lockstep walk: the same outputs,
bit for bit (both run the same FP32 tests with FP64 decisions), at the edges
of its lists and windows -- obstacle counts around the 32 of a ballot and the
512 slots of a window (more slots than that are checked in several passes,
more obstacles than that by the lockstep walk), motions of one state up to
several windows, every kind of output."""
import numpy as np
import pytest

from dynoplan_gb300 import workloads as W

pytestmark = pytest.mark.gpu

EXTENT = {W.UNICYCLE1: (3.0, 3.0), W.CAR1: (3.5, 3.5), W.QUAD2D: (4.0, 3.0), W.QUAD3D: (3.0, 3.0, 2.0)}


def _world(kind, n_obs, N, steps, seed):
    m = W.robot_model(kind)
    prims = W.make_primitives(m, 24, steps[0], steps[1], seed=seed)
    # small boxes all over a small environment: many candidates a lane
    env = W.make_env(EXTENT[kind], n_obs, 0.01, 0.05 if n_obs > 40 else 0.5, seed=seed + 1)
    rng = W.Rng(seed + 2)
    x = W.make_nodes(m, W.Env(env.lo, env.hi, env.obs_lo[:0], env.obs_hi[:0]), N, seed=seed + 3)
    x[0] = np.nan  # in no ball; a neighbour of real nodes in a warp of check_pairs
    return m, prims, env, x, rng


@pytest.mark.parametrize("kind", [W.UNICYCLE1, W.CAR1, W.QUAD2D, W.QUAD3D])
@pytest.mark.parametrize("n_obs", [0, 1, 31, 33, 128, 129, 400, 512, 513])
def test_slots_equal_lockstep(dpg_lib, kind, n_obs):
    from dynoplan_gb300 import gpu as G
    m, prims, env, x, _ = _world(kind, n_obs, 150, (0, 150) if kind in (W.QUAD2D, W.QUAD3D) else (0, 90), 31 + n_obs)
    res = {}
    with G.Context(m) as ctx:
        ctx.upload_primitives(prims)
        ctx.upload_env(env)
        for variant in (0, 1):
            ctx.set_tuning(check_variant=variant)
            for prec in (0, 1):
                res[variant, prec] = ctx.expand(x, 1.5, precision=prec)
            # a list in another order: rows of their own
            r = res[variant, 0]
            k = np.argsort(r["node"], kind="stable")
            res[variant, "pairs"] = ctx.check_pairs(x, r["node"][k], r["prim"][k], precision=1)
    for key in (0, 1, "pairs"):
        a, b = res[0, key], res[1, key]
        assert a["n_pairs"] == b["n_pairs"] > 500
        assert a["n_contact_recheck"] == b["n_contact_recheck"]
        for f in ("node", "prim", "verdict", "first_invalid", "min_gap", "flags", "end_state"):
            np.testing.assert_array_equal(a[f], b[f], err_msg=f"{key} {f}")


def test_nan_node_in_a_list(dpg_lib):
    """A NaN state makes no test fail: its pairs are valid, those beside it unchanged."""
    from dynoplan_gb300 import gpu as G
    m, prims, env, x, _ = _world(W.CAR1, 33, 64, (5, 60), 5)
    node, prim = np.repeat(np.arange(64), 4).astype(np.uint32), np.tile(np.arange(4), 64).astype(np.uint32)
    out = []
    with G.Context(m) as ctx:
        ctx.upload_primitives(prims)
        ctx.upload_env(env)
        for variant in (0, 1):
            ctx.set_tuning(check_variant=variant)
            out.append(ctx.check_pairs(x, node, prim))
    for f in ("verdict", "first_invalid", "min_gap", "flags", "end_state"):
        np.testing.assert_array_equal(out[0][f], out[1][f], err_msg=f)
    assert (out[1]["verdict"][:4] == 0).all()
