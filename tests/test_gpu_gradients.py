"""Gradient reductions of the network against float64 (GPU): the tile widths of
the weight gradient, and the vector and scalar paths of the bias gradient."""
import ctypes as C
import sys
from pathlib import Path

import numpy as np
import pytest

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "oracle"))
import cnn_oracle as O  # noqa: E402

from artefact_b200 import _native as N  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,W,cin,cout", [
    (2, 17, 30, 32, 64), (1, 9, 33, 32, 32), (1, 40, 64, 96, 8), (1, 5, 65, 16, 128), (2, 9, 32, 224, 96),
    (3, 64, 128, 16, 32), (1, 1, 1, 48, 24)])
def test_weight_gradient_tiles(gpu, B, H, W, cin, cout):
    import torch
    rng = np.random.default_rng(7 * W + cout)
    x, g = O.bf16(rng.standard_normal((B, H, W, cin))), O.bf16(rng.standard_normal((B, H, W, cout)))
    xt, gt = (torch.from_numpy(np.ascontiguousarray(a)).to("cuda", torch.bfloat16) for a in (x, g))
    dw = torch.full((cout * 9 * cin,), 0.5, dtype=torch.float32, device="cuda")
    ws = torch.empty(64 << 20, dtype=torch.uint8, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    d = N.ArtCnnWgrad()
    d.B, d.H, d.W, d.cout, d.cin = B, H, W, cout, cin
    d.dy, d.x, d.dw, d.accumulate = gt.data_ptr(), xt.data_ptr(), dw.data_ptr(), 1
    d.workspace, d.workspace_bytes, d.err = ws.data_ptr(), ws.numel(), err.data_ptr()
    N.check(N.lib().art_cnn_wgrad3x3(C.byref(d), None))
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    ref = O.conv_wgrad(x, g) + 0.5
    got = dw.cpu().numpy().astype(np.float64).reshape(cout, 9, cin)
    np.testing.assert_allclose(got, ref, rtol=0, atol=2e-5 * float(np.abs(ref).max()) + 1e-5)


@pytest.mark.parametrize("npix", [1, 7, 300, 4001])
@pytest.mark.parametrize("channels", [1, 8, 24, 32, 100, 200, 256])
@pytest.mark.parametrize("shift", [0, 1])
def test_bias_gradient(gpu, npix, channels, shift):
    """fp32 sums of at most 1024 terms in a row: an error of 1024 units of 2^-24
    of the sum of magnitudes bounds any order."""
    import torch
    g = torch.randn(npix * channels + shift, device="cuda", generator=torch.Generator("cuda").manual_seed(npix))
    g = g.to(torch.bfloat16)[shift:]  # shift 1: not aligned for 16-byte reads
    ws = torch.empty(1 << 20, dtype=torch.uint8, device="cuda")
    out = torch.full((channels,), 2.0, device="cuda")
    N.check(N.lib().art_cnn_bias_grad(g.data_ptr(), npix, channels, ws.data_ptr(), ws.numel(),
                                      out.data_ptr(), 1, None))
    torch.cuda.synchronize()
    g64 = g.double().reshape(npix, channels)
    bound = 1024 * 2.0**-24 * (g64.abs().sum(0) + 2)
    assert bool(((out.double() - g64.sum(0) - 2).abs() <= bound).all())
