"""The network on planes where every block takes several tiles: a weight-gradient
CTA two or three (more than 296 tiles, the accumulation over tiles and the
mbarrier's phase), the narrow layers' blocks many trips, the convolutions and
input gradients in tiles of 4 and of 8 rows, the last layer 4 pixels a thread;
heights and widths with remainders.  The reference is the CPU oracle's arithmetic
(BF16 operands of the hidden layers, everything else in 64 bits) in plain
PyTorch, checked against the oracle itself on a small plane; tolerances as in
test_gpu_cnn.py (output 3e-3, gradient 2e-2, one layer's part of it 4e-2 relative
L2: operands near a BF16 boundary round either way)."""
import numpy as np
import pytest


def _bf16(t):
    import torch
    return t.float().to(torch.bfloat16).double()


def _taps(a):
    """The nine shifted copies of the planes (zero outside), in tap order."""
    import torch
    p = torch.nn.functional.pad(a, (1, 1, 1, 1))
    H, W = a.shape[1:]
    return [p[:, u:u + H, v:v + W].reshape(a.shape[0], -1) for u in range(3) for v in range(3)]


def _reference(params, x, dy):
    """(y, gradient) of oracle/cnn_oracle.py's forward and backward."""
    import torch
    import cnn_oracle as co
    layers, at = [], 0
    for cout, cin in co.shapes():
        n = cout * cin * 9
        layers.append((_bf16(params[at:at + n]).view(cout, cin, 9), params[at + n:at + n + cout].double()))
        at += n + cout
    H, W = x.shape[1:]
    acts, a = [x.double()], x.double()
    for l, (w, b) in enumerate(layers):
        t = _taps(_bf16(a) if l in co.TC_LAYERS else a)
        a = (sum(w[:, :, k] @ t[k] for k in range(9)) + b[:, None]).view(-1, H, W)
        if l < co.LAYERS - 1:
            a = a.clamp(min=0.0)
        acts.append(a)
    y, g, out = a[0], dy.double()[None], []
    for l in range(co.LAYERS - 1, -1, -1):
        w = layers[l][0]
        if l < co.LAYERS - 1:
            g = g * (acts[l + 1] > 0.0)
        tc = l in co.TC_LAYERS
        t, gg = _taps(_bf16(acts[l]) if tc else acts[l]), (_bf16(g) if tc else g)
        gw = torch.stack([gg.reshape(gg.shape[0], -1) @ t[k].T for k in range(9)], dim=2)
        out.append(torch.cat([gw.reshape(-1), g.sum(dim=(1, 2))]))
        if l > 0:
            t = _taps(gg)
            g = sum(w[:, :, 8 - k].T @ t[k] for k in range(9)).view(-1, H, W)
    return y, torch.cat(out[::-1])


def _inputs(H, W, device):
    import torch
    import cnn_oracle as co
    rng = np.random.default_rng(H + W)
    p = co.init_params(5, last_scale=1.0)
    x = rng.standard_normal((3, H, W)).astype(np.float32)
    dy = rng.standard_normal((H, W)).astype(np.float32)
    return p, x, dy, [torch.tensor(a, device=device) for a in (p, x, dy)]


def test_reference_is_the_oracle():
    import cnn_oracle as co
    p, x, dy, t = _inputs(13, 18, "cpu")
    y, g = (a.numpy() for a in _reference(*t))
    yo, go = co.forward(p, x)[0], co.backward(p, x, dy)
    assert np.abs(y - yo).max() <= 1e-12 * np.abs(yo).max()
    assert np.abs(g - go).max() <= 1e-12 * np.abs(go).max()


@pytest.mark.gpu
@pytest.mark.parametrize("H,W", [(400, 1000), (403, 256), (1001, 130)])
def test_large_planes(H, W):
    import cnn_oracle as co
    from pvof import cnn
    p, x, dy, (pt, xt, dyt) = _inputs(H, W, "cuda")
    yr, gr = (a.cpu().numpy() for a in _reference(pt, xt, dyt))
    net = cnn.Network(H, W, params=p)
    xf = xt.reshape(-1)
    y = net.forward(xf).cpu().numpy().reshape(H, W)
    g = net.gradient(xf, dyt.reshape(-1)).cpu().numpy()
    net.status()
    rel = lambda a, b: float(np.linalg.norm(a - b) / np.linalg.norm(b))
    ey, eg, at, el = rel(y, yr), rel(g, gr), 0, []
    for cout, cin in co.shapes():
        for n in (cout * cin * 9, cout):
            a, b = g[at:at + n], gr[at:at + n]
            el.append(float(np.linalg.norm(a - b) / (np.linalg.norm(b) + 2.5e-5 * np.linalg.norm(gr))))
            at += n
    print(H, W, ey, eg, el)
    assert ey <= 3e-3 and eg <= 2e-2 and max(el) <= 4e-2, (ey, eg, el)
