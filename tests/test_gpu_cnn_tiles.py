"""The network's tensor-core tiles at their edges: one pixel, one row, a strip
of 128 pixels and one more, planes whose width is no multiple of 16, and
planes large enough for tiles of 4 and 8 rows.  Against the CPU oracle with
the tolerances of test_gpu_cnn.py (a layer on BF16-exact inputs 1e-5 of the
largest value, the network's output 3e-3 and its gradient 2e-2 relative L2)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,W", [(1, 1), (3, 128), (2, 129), (37, 257), (200, 300), (400, 300)])
def test_layer(H, W):
    import torch
    import cnn_oracle as co
    from pvof.cnn import _ptr
    from pvof.runtime import check, load
    rng = np.random.default_rng(H * 1000 + W)
    x = co.to_bf16(rng.standard_normal((32, H, W)).astype(np.float32))
    w = co.to_bf16((rng.standard_normal((32, 32, 3, 3)) * 0.1).astype(np.float32))
    b = rng.standard_normal(32).astype(np.float32)
    wb = torch.tensor((w.view(np.uint32) >> 16).astype(np.int16).ravel(), device="cuda")
    xt, bt = torch.tensor(x.ravel(), device="cuda"), torch.tensor(b, device="cuda")
    yt = torch.empty(32 * H * W, dtype=torch.float32, device="cuda")
    check(load().pvof_cnn_conv32(_ptr(xt), _ptr(wb), _ptr(bt), _ptr(yt), H, W, 1, None), "conv32")
    check(load().pvof_cnn_status(None), "status")
    ref = np.maximum(co.conv(x.astype(np.float64), w.astype(np.float64), b), 0.0)
    assert np.abs(yt.cpu().numpy().reshape(32, H, W) - ref).max() <= 1e-5 * np.abs(ref).max()


@pytest.mark.parametrize("H,W", [(1, 5), (4, 128), (11, 150), (70, 129)])
def test_gradient(H, W):
    import torch
    import cnn_oracle as co
    from pvof import cnn
    rng = np.random.default_rng(H + W)
    p = co.init_params(5, last_scale=1.0)
    x = rng.standard_normal((3, H, W)).astype(np.float32)
    dy = rng.standard_normal((H, W)).astype(np.float32)
    net = cnn.Network(H, W, params=p)
    xt = torch.tensor(x.ravel(), device="cuda")
    y_ref, _ = co.forward(p, x)
    y = net.forward(xt).cpu().numpy().reshape(H, W)
    assert np.linalg.norm(y - y_ref) <= 3e-3 * np.linalg.norm(y_ref)
    g = net.gradient(xt, torch.tensor(dy.ravel(), device="cuda")).cpu().numpy()
    net.status()
    g_ref = co.backward(p, x, dy)
    assert np.linalg.norm(g - g_ref) <= 2e-2 * np.linalg.norm(g_ref)
    at = 0
    for n, cin in ((32, 3), (32, 32), (32, 32), (32, 32), (32, 32), (1, 32)):   # every layer's weights and biases
        for size in (n * cin * 9, n):
            a, b = g[at:at + size], g_ref[at:at + size]
            assert np.linalg.norm(a - b) <= 4e-2 * np.linalg.norm(b) + 1e-6 * np.linalg.norm(g_ref), (n, cin, size)
            at += size
