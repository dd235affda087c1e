"""The check's work queue: a warp with a long item leaves the launch's last items to
the others.  32 or 64 motions over 37 words of nodes, one or two items a warp,
a quarter of them long (robots that stand still between obstacles), the others
over at once (nodes in collision).  Items that wait for their warp's long one
would double the time; taken up by free warps they add little."""
import numpy as np
import pytest

from dynoplan_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant,L", [(1, 30000), (0, 20000)])  # slots, lockstep
def test_long_items_start_on_free_warps(dpg_lib, variant, L):
    from dynoplan_gb300 import gpu as G
    torch = pytest.importorskip("torch")
    m = W.robot_model(W.UNICYCLE1)
    warps = 8 * torch.cuda.get_device_properties(0).multi_processor_count  # a block of eight warps an SM
    words = 37
    P = warps // words
    at = np.stack(np.meshgrid(np.arange(10.0), np.arange(12.0), indexing="ij"), -1).reshape(-1, 2) * 4
    obs_lo, obs_hi = np.concatenate([[[-100, -100]], at + 1.9]), np.concatenate([[[-50, 100]], at + 2.1])
    env = W.Env(np.array([-1e3, -1e3]), np.array([1e3, 1e3]), obs_lo, obs_hi)
    rng = np.random.default_rng(1)
    x = np.zeros((32 * words, 3))
    x[:, :2] = at[rng.integers(0, len(at), len(x))]
    x.reshape(words, 32, 3)[rng.permutation(words)[words // 4:], :, 0] = -75.0  # in the first obstacle
    times = []
    for p in (P, 2 * P):
        prims = W.Primitives(np.full(p, L, np.int32), np.zeros((p * L, 3)), np.zeros((p * (L - 1), 2)))
        cap = len(x) * p
        dev = {k: torch.empty(cap, dtype=t, device="cuda") for k, t in
               (("node", torch.int32), ("prim", torch.int32), ("verdict", torch.uint8))}
        xd = torch.from_numpy(x).cuda()
        torch.cuda.synchronize()
        with G.Context(m) as ctx:
            ctx.upload_primitives(prims)
            ctx.upload_env(env)
            ctx.set_tuning(check_blocks_per_sm=1, check_variant=variant)
            t = []
            for _ in range(7):
                r = ctx.expand_device(xd.data_ptr(), len(x), 1e3, {k: v.data_ptr() for k, v in dev.items()}, cap)
                t.append(ctx.timings()[1])
            assert r["n_pairs"] == cap
            times.append(float(np.median(t)))
    assert times[1] < 1.6 * times[0], times


@pytest.mark.parametrize("n_obs", [20, 100, 128, 400])
@pytest.mark.parametrize("kind,P,steps,radius", [(W.QUAD2D, 1500, (20, 150), 0.3), (W.CAR1, 1000, (5, 100), 0.25)])
def test_slots_among_many_obstacles(dpg_lib, kind, P, steps, radius, n_obs):
    """The windows' slots must not cost more than a lane walking its own tests: no
    slower than the lockstep walk (1.7 times as slow for quad2d with windows
    whose slots did not fit)."""
    from dynoplan_gb300 import gpu as G
    m = W.robot_model(kind)
    prims = W.make_primitives(m, P, *steps, seed=3)
    env = W.make_env((8.0, 4.0), n_obs, 0.05, 0.25, seed=4)
    x = W.make_nodes(m, W.Env(env.lo, env.hi, env.obs_lo[:0], env.obs_hi[:0]), 1200, seed=6)
    x = np.ascontiguousarray(x[np.sort(np.argsort(-W.state_gap(m, env, x))[:300])])  # the freest
    with G.Context(m) as ctx:
        ctx.upload_primitives(prims)
        ctx.upload_env(env)
        t = {0: [], 1: []}
        for i in range(14):
            for v in t:
                ctx.set_tuning(check_variant=v)
                r = ctx.expand(x, radius, capacity=300 * P)
                if i >= 3:
                    t[v].append(ctx.timings()[1])
                elif v == 0:
                    ref = r
                elif i == 0:  # (the same results, bit for bit)
                    for k in ("node", "prim", "verdict", "first_invalid", "end_state", "min_gap", "flags"):
                        np.testing.assert_array_equal(r[k], ref[k], err_msg=k)
        assert np.median(t[1]) <= 1.1 * np.median(t[0]), (np.median(t[1]), np.median(t[0]))
