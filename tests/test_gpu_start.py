"""Device coefficients at any alignment (GPU).

art_context_compute_device takes the caller's coefficient pointers as they
are; the start kernel reads 16 bytes at a time where they allow it. Planes
must equal those of the host entry point, whose staging is aligned.
"""
import ctypes as C

import numpy as np
import pytest

from artefact_b200 import _native as N
from artefact_b200 import synth
from artefact_b200.api import Context, Jpeg, JpegSource

pytestmark = pytest.mark.gpu


def _device(ctx, j, dtype, shift, iterations, bad=None):
    import torch

    W, H, _ = j.max_rounded()
    ch, keep = (N.ArtChannel * j.nchannel)(), []
    for a, co in zip(ch, j.coefs):
        v = torch.from_numpy(co.dct_coefs.astype(dtype))
        if bad is not None:
            v[-1] = bad
        buf = torch.zeros(v.numel() + 16, dtype=v.dtype, device="cuda")
        buf[shift:shift + v.numel()] = v.cuda()
        q = np.ascontiguousarray(co.quant_table, np.float32)
        keep += [buf, q]
        a.rounded_px_w, a.rounded_px_h, a.block_w, a.block_h = co.rounded_px_w, co.rounded_px_h, co.block_w, co.block_h
        a.samp_h, a.samp_v = co.horizontal_samp_factor, co.vertical_samp_factor
        a.coef_type = N.ART_COEF_I16 if dtype == np.int16 else N.ART_COEF_F32
        a.dct_coefs = buf.data_ptr() + shift * buf.element_size()
        a.quant_table = q.ctypes.data_as(C.POINTER(C.c_float))
    outs = [torch.empty(H, W, device="cuda") for _ in range(j.nchannel)]
    ptrs = (C.c_void_p * j.nchannel)(*[o.data_ptr() for o in outs])
    N.check(N.lib().art_context_compute_device(ctx.handle, j.nchannel, ch, 0.3, (C.c_float * 3)(*[0.001] * 3),
                                               iterations, W, H, ptrs, W, None, None))
    torch.cuda.synchronize()
    return N.lib().art_context_synchronize(ctx.handle), [o.cpu().numpy().ravel() for o in outs]


@pytest.mark.parametrize("sub", ["4:4:4", "4:2:2", "4:2:0"])
@pytest.mark.parametrize("dtype,shift", [(np.int16, 0), (np.int16, 1), (np.int16, 4), (np.float32, 0), (np.float32, 1)])
def test_coefficient_alignment(gpu, sub, dtype, shift):
    j = Jpeg.from_source(JpegSource.Buffer(synth.make_jpeg(136, 40, 60, sub, False, seed=4)))
    W, H, _ = j.max_rounded()
    with Context(0) as ctx:
        for iterations in (0, 3):
            want = ctx.compute(j.nchannel, j.coefs, 0.3, [0.001] * 3, iterations, W, H)
            rc, got = _device(ctx, j, dtype, shift, iterations)
            assert rc == 0 and all(np.array_equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("bad", [0.5, float("nan"), float("inf"), 32768.0, -32769.0])
def test_bad_coefficients_rejected(gpu, bad, shift):
    j = Jpeg.from_source(JpegSource.Buffer(synth.make_jpeg(40, 24, 60, "4:4:4", False, seed=4)))
    with Context(0) as ctx:
        assert _device(ctx, j, np.float32, shift, 1, bad)[0] == N.ART_ERR_INVALID_DATA
        assert _device(ctx, j, np.float32, shift, 1)[0] == 0
