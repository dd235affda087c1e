"""dpg_mlp_last_timing's FLOPs: the products the kernels compute, rows padded to 128."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 128, 300])
def test_flops(dpg_lib, n):
    torch = pytest.importorskip("torch")
    from dynoplan_gb300.surrogate import Surrogate
    s = Surrogate(4, max_rows=512)
    feat = torch.zeros((1, 80), dtype=torch.bfloat16, device="cuda")
    zero = torch.zeros(n, dtype=torch.int32, device="cuda")
    layer = lambda k, m: 2.0 * ((n + 127) // 128 * 128) * k * m
    hidden = 2 * layer(256, 256)
    for kernel, want in ((2, layer(96, 256) + hidden + layer(256, 2)), (1, layer(128, 256) + hidden + layer(256, 16)),
                         (0, layer(128, 256) + hidden + layer(256, 16))):
        s.set_fused(kernel)
        s.forward(feat, zero, zero)
        assert s.timing()[1] == want, kernel
    s.train_step(feat, zero, zero, torch.zeros((n, 2), device="cuda"))
    forward = layer(128, 256) + hidden + layer(256, 16)
    backward = layer(64, 256) + hidden + layer(256, 16)        # dH3, dH2, dH1, the embedding's columns of dX
    weights = layer(96, 256) + hidden + layer(256, 16)
    assert s.timing()[1] == forward + backward + weights
    s.close()
