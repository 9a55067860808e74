"""Last passes of the network's reductions over few and many partials (GPU)."""
import ctypes as C
import sys
from pathlib import Path

import numpy as np
import pytest

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "oracle"))
import cnn_oracle as O  # noqa: E402

from artefact_b200 import _native as N  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bands", [1, 2, 7, 8, 9, 20])
@pytest.mark.parametrize("cin,cout", [(16, 8), (48, 24)])
@pytest.mark.parametrize("accumulate", [0, 1])
def test_weight_gradient_bands(gpu, bands, cin, cout, accumulate):
    """A tile of 2 rows a band; outputs are no multiple of a block, and what lies
    behind them stays."""
    import torch
    B, H, W = 1, 2 * bands, 128
    rng = np.random.default_rng(bands + cin)
    x, g = O.bf16(rng.standard_normal((B, H, W, cin))), O.bf16(rng.standard_normal((B, H, W, cout)))
    xt, gt = (torch.from_numpy(np.ascontiguousarray(a)).to("cuda", torch.bfloat16) for a in (x, g))
    total = cout * 9 * cin
    dw = torch.full((total + 256,), 0.5, dtype=torch.float32, device="cuda")
    ws = torch.empty(total * 4 * bands, dtype=torch.uint8, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    d = N.ArtCnnWgrad()
    d.B, d.H, d.W, d.cout, d.cin = B, H, W, cout, cin
    d.dy, d.x, d.dw, d.accumulate = gt.data_ptr(), xt.data_ptr(), dw.data_ptr(), accumulate
    d.workspace, d.workspace_bytes, d.err = ws.data_ptr(), ws.numel(), err.data_ptr()
    N.check(N.lib().art_cnn_wgrad3x3(C.byref(d), None))
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    got = dw.cpu().numpy().astype(np.float64)
    ref = O.conv_wgrad(x, g) + 0.5 * accumulate
    np.testing.assert_allclose(got[:total].reshape(cout, 9, cin), ref, rtol=0, atol=2e-5 * float(np.abs(ref).max()) + 1e-5)
    assert (got[total:] == 0.5).all()


@pytest.mark.parametrize("blocks", [1, 4, 5, 17, 257])
@pytest.mark.parametrize("channels", [1, 2, 16, 33, 256])
def test_bias_gradient_partials(gpu, blocks, channels):
    """The workspace sets the number of partials. fp32 sums of at most 4001 terms
    in a row: an error of 4096 units of 2^-24 of the sum of magnitudes bounds any
    order."""
    import torch
    npix = 4001
    g = torch.randn(npix * channels, device="cuda", generator=torch.Generator("cuda").manual_seed(blocks)).to(torch.bfloat16)
    ws = torch.empty(blocks * channels * 4, dtype=torch.uint8, device="cuda")
    out = torch.full((channels,), 2.0, device="cuda")
    N.check(N.lib().art_cnn_bias_grad(g.data_ptr(), npix, channels, ws.data_ptr(), ws.numel(), out.data_ptr(), 1, None))
    torch.cuda.synchronize()
    g64 = g.double().reshape(npix, channels)
    bound = 4096 * 2.0**-24 * (g64.abs().sum(0) + 2)
    assert bool(((out.double() - g64.sum(0) - 2).abs() <= bound).all())
