"""dpg_mlp_node_features against numpy: the occupancy patch exactly (the same
FP32 comparisons), the state part to bf16 rounding; node and obstacle counts
around the kernel's 32 nodes a block and 8 lanes a node, a goal or none, and a
destination that is not 16-byte aligned."""
import math

import numpy as np
import pytest

from dynoplan_gb300 import workloads as W

pytestmark = pytest.mark.gpu

EXTENT = {W.UNICYCLE1: (6.0, 6.0), W.CAR1: (10.0, 10.0), W.QUAD2D: (8.0, 4.0), W.QUAD3D: (6.0, 6.0, 3.0)}


def reference(m, env, x, goal):
    d, f = env.dim, np.zeros((len(x), 80))
    ext = env.hi - env.lo
    f[:, :d] = 2 * (x[:, :d] - env.lo) / ext - 1
    for i in range(d, m.nx):
        if m.kind != W.QUAD3D and (i == 2 or (m.kind == W.CAR1 and i == 3)):
            f[:, i] = ((x[:, i] + math.pi) % (2 * math.pi) - math.pi) / math.pi
        else:
            f[:, i] = x[:, i] if m.kind == W.QUAD3D and i < 7 else x[:, i] / 4
    if goal is not None:
        f[:, 13:13 + d] = 2 * (goal[:d] - x[:, :d]) / ext
    f32 = np.float32
    cen = (0.5 * (env.obs_lo + env.obs_hi)).astype(f32)
    half = (0.5 * (env.obs_hi - env.obs_lo)).astype(f32)
    p, h = x[:, :d].astype(f32), f32(0.375)
    for c in range(64):
        q = [p[:, 0] + f32((c % 8 - 3.5) * 0.75), p[:, 1] + f32((c // 8 - 3.5) * 0.75)] + ([p[:, 2]] if d == 3 else [])
        if len(cen):
            near = [np.abs(q[i][:, None] - cen[:, i]) <= h + half[:, i] for i in range(d)]
            f[:, 16 + c] = np.logical_and.reduce(near).any(1)
    return f


@pytest.mark.parametrize("kind", [W.UNICYCLE1, W.CAR1, W.QUAD2D, W.QUAD3D])
@pytest.mark.parametrize("N,n_obs,shift", [(1, 1, 0), (31, 0, 0), (33, 7, 1), (64, 9, 0), (1000, 80, 3)])
def test_features(dpg_lib, kind, N, n_obs, shift):
    import ctypes as C

    import torch

    from dynoplan_gb300 import _lib
    from dynoplan_gb300 import gpu as G
    m = W.robot_model(kind)
    env = W.make_env(EXTENT[kind], n_obs, 0.1, 1.0, seed=N + n_obs)
    x = W.make_nodes(m, env, N, seed=N + 5)
    if kind != W.QUAD3D:
        x[0, 2] += 6 * math.pi  # an angle to wrap
    goal = x[-1].copy() if N % 2 else None
    buf = torch.full((N * 80 + 8,), 7.0, dtype=torch.bfloat16, device="cuda")
    x_dev = torch.from_numpy(x).cuda()
    with G.Context(m) as ctx:
        ctx.upload_env(env)
        _lib.check(_lib.load().dpg_mlp_node_features(ctx.h, C.c_void_p(x_dev.data_ptr()), N,
                                                     goal.ctypes.data if goal is not None else None,
                                                     C.c_void_p(buf.data_ptr() + 2 * shift)), ctx.h)
    out = buf.float().cpu().numpy()
    assert (out[:shift] == 7).all() and (out[shift + N * 80:] == 7).all()
    got, ref = out[shift:shift + N * 80].reshape(N, 80), reference(m, env, x, goal)
    np.testing.assert_array_equal(got[:, 16:], ref[:, 16:])
    np.testing.assert_allclose(got[:, :16], ref[:, :16], rtol=2.0 ** -8, atol=1e-6)


@pytest.mark.parametrize("kind", [W.CAR1, W.QUAD3D])
def test_positions_are_divided_by_the_extent(dpg_lib, kind):
    """The middle of the environment is exactly 0, its upper bound exactly 1, and
    every position 2 (x - lo) / extent - 1 as FP64 gives it (infinite ones too), for
    extents whose reciprocal is not exact."""
    import torch

    from dynoplan_gb300 import gpu as G
    from dynoplan_gb300.surrogate import node_features
    m = W.robot_model(kind)
    d = 3 if kind == W.QUAD3D else 2

    def bf16(a):
        with np.errstate(over="ignore"):  # (-1e300 becomes -inf)
            return torch.from_numpy(a.astype(np.float32)).to(torch.bfloat16)

    with G.Context(m) as ctx:
        for e in range(3, 120):
            ext = np.array([e, e + 0.1, e / 7.0])[:d]
            ctx.upload_env(W.Env(np.zeros(d), ext, np.zeros((0, d)), np.zeros((0, d))))
            x = np.zeros((64, m.nx))
            x[:, :d] = ext * np.linspace(0, 1, 64)[:, None]
            x[0, :d], x[1, :d], x[2, :d] = 0.5 * ext, ext, 0.25 * ext
            x[3, :d], x[4, :d] = np.inf, -1e300
            goal = x[5].copy()
            f = node_features(ctx, torch.from_numpy(x).cuda(), goal).cpu()
            assert torch.equal(f[:, :d], bf16(2.0 * x[:, :d] / ext - 1.0)), e
            assert torch.equal(f[:, 13:13 + d], bf16(2.0 * (goal[:d] - x[:, :d]) / ext)), e
