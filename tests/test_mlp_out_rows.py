"""dpg_mlp_forward writes n rows of its output and no more, with every forward
kernel (the tensor-core tiles hold 128 rows)."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fused", [0, 1, 2])
@pytest.mark.parametrize("n", [1, 127, 128, 130, 300])
def test_forward_writes_n_rows(dpg_lib, fused, n):
    torch = pytest.importorskip("torch")
    from dynoplan_gb300 import _lib
    from dynoplan_gb300.surrogate import Surrogate
    g = torch.Generator(device="cuda").manual_seed(n)
    feat = torch.randn((50, 80), generator=g, device="cuda").to(torch.bfloat16)
    node = torch.randint(50, (n,), generator=g, device="cuda", dtype=torch.int32)
    prim = torch.randint(9, (n,), generator=g, device="cuda", dtype=torch.int32)
    buf = torch.full((n + 512, 2), 3.0, device="cuda")  # room for whole tiles behind the n rows
    s = Surrogate(9, max_rows=128, seed=1)  # (n = 130 and 300: several chunks of rows for the layer-by-layer form)
    s.set_fused(fused)
    _lib.check(_lib.load().dpg_mlp_forward(s.h, C.c_void_p(feat.data_ptr()), C.c_void_p(node.data_ptr()),
                                           C.c_void_p(prim.data_ptr()), n, C.c_void_p(buf.data_ptr())))
    out = buf.cpu().numpy()
    assert (out[n:] == 3.0).all()
    assert np.isfinite(out[:n]).all() and (out[:n] != 3.0).any()
