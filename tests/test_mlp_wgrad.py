"""Weight, bias and embedding gradients at batch sizes around the tiles of the
weight-gradient kernel (64-row chunks split over the CTAs, 128-row padding),
against the FP64 restatement with bf16 rounding (tests/mlp_ref.py).

Tolerance: relative L2 error <= 2e-2 per parameter, as test_mlp.py (the bf16
operands are the same; rare rounding flips of pre-activation gradients)."""
import numpy as np
import pytest

from test_mlp import _random_params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B", [1, 63, 64, 128, 129, 700, 9729, 20000])
def test_gradients(dpg_lib, B):
    torch = pytest.importorskip("torch")
    import mlp_ref
    from dynoplan_gb300.surrogate import Surrogate
    rng = np.random.default_rng(B + 1)
    P, N = 40, 100
    params = _random_params(rng, P)
    feat = rng.normal(0, 1, (N, 80)).astype(np.float32)
    node, prim = rng.integers(0, N, B), rng.integers(0, P, B)
    target = np.stack([(rng.random(B) < 0.4).astype(np.float32), rng.random(B).astype(np.float32)], 1)
    s = Surrogate(P, max_rows=20000, seed=1)
    for k, v in params.items():
        s.set(k, v)
    dev = lambda a: torch.from_numpy(a).cuda()
    feat_d = dev(feat).to(torch.bfloat16)
    loss = s.train_step(feat_d, dev(node.astype(np.int32)), dev(prim.astype(np.int32)), dev(target), lr=0.0)
    _, ref_loss, ref = mlp_ref.forward_backward(params, feat_d.float().cpu().numpy(), node, prim, target, 1.0)
    assert loss == pytest.approx(ref_loss, rel=1e-3)
    for k in ref:
        g = s.get(k, grad=True).astype(np.float64)
        r = ref[k]
        assert not np.any(g[2:]) if k in ("W4", "b4") else True
        if k in ("W4", "b4"):
            g, r = g[:2], r[:2]
        assert np.linalg.norm(g - r) <= 2e-2 * max(np.linalg.norm(r), 1e-12), k


def test_bias_gradient_keeps_small_terms(dpg_lib):
    """db3 = sum_b dZ3[b] with one row of 1 and 65,535 of 2^-26 (weights zero, so
    that dZ3 = dY / 2 exactly).  Tolerance: a sum of 32 rows, of a CTA's parts
    (under 64) and of the CTAs (under 64), each addition within half an ulp:
    (31 + 64 + 64) 2^-24 = 9.5e-6; one running sum over a CTA's rows loses
    1,400 x 2^-26 = 2.1e-5."""
    torch = pytest.importorskip("torch")
    from dynoplan_gb300.surrogate import SHAPES, Surrogate
    B, P = 65536, 4
    s = Surrogate(P, max_rows=B, seed=1)
    for k, shape in SHAPES.items():
        s.set(k, np.zeros(shape, np.float32))
    w4 = np.zeros((16, 256), np.float32)
    w4[1] = 1.0
    s.set("W4", w4)
    dz = np.full(B, 2.0 ** -26)
    dz[0] = 1.0
    target = np.stack([np.full(B, np.nan), -2.0 * dz * B], 1).astype(np.float32)  # dY = -target / B
    feat = torch.zeros((1, 80), dtype=torch.bfloat16, device="cuda")
    zero = torch.zeros(B, dtype=torch.int32, device="cuda")
    s.train_step(feat, zero, zero, torch.from_numpy(target).cuda(), lr=0.0)
    g = s.get("b3", grad=True).astype(np.float64)
    assert np.abs(g / dz.sum() - 1).max() <= (31 + 64 + 64) * 2.0 ** -24
    s.close()


def test_weight_gradient_of_one_sign(dpg_lib):
    """dW3 = sum_b dZ3[b] H2[b] at 65,536 rows of one sign, H2 = b2 (gelu of 8 to 16
    in bf16) and dZ3 = dY / 2 exactly.  Tolerance (rms, relative): an accumulator
    takes at most 14 x 64 rows, 56 steps that each cut half a unit in the last place
    on average off a partial sum that is half the total on average, 56 x 2^-23 / 4 =
    1.7e-6, and 2 x 45 roundings of the CTAs' sums, sqrt(90) 2^-25 = 0.3e-6
    (2.3e-6 with 92 steps)."""
    torch = pytest.importorskip("torch")
    from dynoplan_gb300.surrogate import SHAPES, Surrogate
    B = 65536
    s = Surrogate(4, max_rows=B, seed=1)
    for k, shape in SHAPES.items():
        s.set(k, np.zeros(shape, np.float32))
    w4, b2 = np.zeros((16, 256), np.float32), (8 + (2 * (np.arange(256) % 64) + 1) / 16).astype(np.float32)
    w4[1] = 1.0
    s.set("W4", w4)
    s.set("b2", b2)
    dy = torch.from_numpy(np.random.default_rng(3).random(B) / B).to(torch.bfloat16).double().numpy()
    target = np.stack([np.full(B, np.nan), -dy * B], 1).astype(np.float32)
    feat = torch.zeros((1, 80), dtype=torch.bfloat16, device="cuda")
    zero = torch.zeros(B, dtype=torch.int32, device="cuda")
    s.train_step(feat, zero, zero, torch.from_numpy(target).cuda(), lr=0.0)
    g = s.get("W3", grad=True).astype(np.float64)
    e = g / (0.5 * dy.sum() * b2[None, :].astype(np.float64)) - 1
    assert np.sqrt((e ** 2).mean()) <= 56 * 2.0 ** -25 + 90 ** 0.5 * 2.0 ** -25
    s.close()


_SHIM = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stdlib.h>
#include <string.h>
/* with SHIM_NO_MAPS the driver has no cuTensorMapEncodeTiled; the rest goes to the runtime */
int cudaGetDriverEntryPointByVersion(const char *s, void **p, unsigned v, unsigned long long f, int *q) {
  if (getenv("SHIM_NO_MAPS") && !strcmp(s, "cuTensorMapEncodeTiled")) { *p = 0; if (q) *q = 1; return 0; }
  int (*real)(const char *, void **, unsigned, unsigned long long, int *) =
      dlsym(dlopen("libcudart.so.13", RTLD_LAZY), "cudaGetDriverEntryPointByVersion");
  return real(s, p, v, f, q);
}
/* no launch while SHIM_FAIL is set */
int cudaGraphLaunch(void *g, void *st) {
  if (getenv("SHIM_FAIL")) return 999;
  int (*real)(void *, void *) = dlsym(dlopen("libcudart.so.13", RTLD_LAZY), "cudaGraphLaunch");
  return real(g, st);
}
"""

_TRAIN = r"""
import sys
sys.path[:0] = sys.argv[1:3]
import numpy as np, torch
from test_mlp import _random_params
from dynoplan_gb300.surrogate import Surrogate
B, P, N = int(sys.argv[3]), 40, 100
rng = np.random.default_rng(B)
params = _random_params(rng, P)
feat = torch.from_numpy(rng.normal(0, 1, (N, 80)).astype(np.float32)).cuda().to(torch.bfloat16)
dev = lambda a: torch.from_numpy(a).cuda()
node, prim = dev(rng.integers(0, N, B).astype(np.int32)), dev(rng.integers(0, P, B).astype(np.int32))
target = dev(np.stack([(rng.random(B) < 0.4), rng.random(B)], 1).astype(np.float32))
s = Surrogate(P, max_rows=max(B, 128), seed=1)
for k, v in params.items():
    s.set(k, v)
loss = [s.train_step(feat, node, prim, target, lr=1e-3)]
if sys.argv[5] == "fail":
    import os
    from dynoplan_gb300 import _lib
    ms = s.timing()[0]
    s.train_step(feat, node, prim, target, lr=0.0)
    os.environ["SHIM_FAIL"] = "1"
    try:
        s.train_step(feat, node, prim, target, lr=1e-3)
        raise SystemExit("no error")
    except _lib.DpgError as e:
        assert e.code == _lib.DPG_ERR_CUDA
    del os.environ["SHIM_FAIL"]
    assert 0.2 * ms < s.timing()[0] < 5 * ms, (ms, s.timing())  # the last step that ran
elif sys.argv[5] == "two":
    s.train_step(feat, node, prim, target, lr=0.0)
loss.append(s.train_step(feat, node, prim, target, lr=1e-3))
out = {"g_" + k: s.get(k, grad=True) for k in params}
out.update({"w_" + k: s.get(k) for k in params})
np.savez(sys.argv[4], loss=np.array(loss), out=s.forward(feat, node, prim).cpu().numpy(), **out)
"""


def _train_in_children(tmp_path, B, runs):
    """_TRAIN in a process a run (name: environment, mode), with the stand-in preloaded"""
    import os
    import subprocess
    import sys
    here = os.path.dirname(os.path.abspath(__file__))
    (tmp_path / "shim.c").write_text(_SHIM)
    (tmp_path / "train.py").write_text(_TRAIN)
    shim = str(tmp_path / "shim.so")
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", shim, str(tmp_path / "shim.c"), "-ldl"], check=True)
    got = []
    for k, (env, mode) in enumerate(runs):
        path = str(tmp_path / f"{k}.npz")
        r = subprocess.run([sys.executable, str(tmp_path / "train.py"), os.path.dirname(here), here, str(B), path, mode],
                           env={**os.environ, "LD_PRELOAD": shim, **env}, capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stderr[-2000:]
        got.append(dict(np.load(path)))
    return got


@pytest.mark.parametrize("B", [1, 700, 9729])
def test_training_without_tensor_maps(dpg_lib, tmp_path, B):
    """Two steps and a forward in a process where the driver gives no
    cuTensorMapEncodeTiled (a preloaded stand-in says so), against the same with
    it: both compute the same bf16 products (tolerance as above; the weights
    after two steps of 1e-3 within 1e-4)."""
    a, b = _train_in_children(tmp_path, B, [({}, ""), ({"SHIM_NO_MAPS": "1"}, "")])
    np.testing.assert_allclose(a["loss"], b["loss"], rtol=1e-3)
    for k in a:
        if k.startswith("g_"):
            assert np.linalg.norm(a[k] - b[k]) <= 2e-2 * max(np.linalg.norm(a[k]), 1e-12), k
        elif k.startswith("w_"):
            assert np.abs(a[k] - b[k]).mean() <= 1e-4, k
    assert np.abs(a["out"] - b["out"]).max() <= 2e-2 * (1 + np.abs(a["out"]).max())


def test_failed_step_does_not_count(dpg_lib, tmp_path):
    """A step whose launch fails (a preloaded stand-in refuses it): the weights, the
    next step's bias corrections (a fourth step's instead of a third's would change
    its update by a tenth) and the stage times are as if it had not been called."""
    a, b = _train_in_children(tmp_path, 700, [({}, "two"), ({}, "fail")])
    for k in a:
        if k.startswith("w_"):
            assert np.abs(a[k] - b[k]).mean() <= 1e-5, k
