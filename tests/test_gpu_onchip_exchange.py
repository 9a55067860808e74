"""What the blocks of an on-chip solve exchange through global memory (GPU).

Tagged words decide when a block goes on, so no word may carry a tag that its
solve still waits for.
"""
import ctypes as C

import numpy as np
import pytest

from artefact_b200 import _native as N
from artefact_b200 import synth
from artefact_b200.api import Context, Jpeg, JpegSource

pytestmark = pytest.mark.gpu


def _jpeg(w, h, sub, seed=3):
    gray = sub == "gray"
    return Jpeg.from_source(JpegSource.Buffer(synth.make_jpeg(w, h, 50, "4:4:4" if gray else sub, gray, seed=seed)))


def _solve(ctx, j, iterations=7):
    W, H, _ = j.max_rounded()
    return ctx.compute(j.nchannel, j.coefs, 0.3, [0.001] * 3, iterations, W, H)


def _equal(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a, b))


def _leave_tagged_words():
    """Frees device memory full of words {NaN, small tag}."""
    import torch

    tags = torch.arange(1, 65, dtype=torch.int64, device="cuda") << 32 | 0x7FC00000
    held = tags.repeat((256 << 20) // tags.nbytes)
    torch.cuda.synchronize()
    del held, tags
    torch.cuda.empty_cache()


def test_grown_exchange_memory_starts_at_zero(gpu, monkeypatch):
    """The exchange buffer grows while the others do not, into memory that
    holds words an earlier program may have left."""
    jpegs = [_jpeg(96, 64, "4:2:0"), _jpeg(518, 389, "gray"), _jpeg(600, 450, "gray"), _jpeg(640, 470, "4:2:0")]
    monkeypatch.setenv("ART_RESIDENT", "0")
    with Context(0) as ctx:
        want = [_solve(ctx, j) for j in jpegs]
    monkeypatch.delenv("ART_RESIDENT")
    with Context(0) as ctx:
        for j, w in zip(jpegs, want):
            _leave_tagged_words()
            assert _equal(_solve(ctx, j), w), (j.real_px_w, j.real_px_h)


@pytest.mark.parametrize("size,sub", [((96, 64), "4:2:0"), ((518, 389), "gray")])
def test_callers_capture_is_refused(gpu, size, sub):
    """A solve cannot be captured into the caller's graph, on chip no more than
    as launch pairs: the graph would carry this call's tags."""
    import torch

    j = _jpeg(*size, sub)
    W, H, _ = j.max_rounded()
    ch, keep = (N.ArtChannel * j.nchannel)(), []
    for a, co in zip(ch, j.coefs):
        buf, q = torch.from_numpy(co.dct_coefs.astype(np.int16)).cuda(), np.ascontiguousarray(co.quant_table, np.float32)
        keep += [buf, q]
        a.rounded_px_w, a.rounded_px_h, a.block_w, a.block_h = co.rounded_px_w, co.rounded_px_h, co.block_w, co.block_h
        a.samp_h, a.samp_v = co.horizontal_samp_factor, co.vertical_samp_factor
        a.coef_type, a.dct_coefs = N.ART_COEF_I16, buf.data_ptr()
        a.quant_table = q.ctypes.data_as(C.POINTER(C.c_float))
    outs = [torch.empty(H, W, device="cuda") for _ in range(j.nchannel)]
    ptrs = (C.c_void_p * j.nchannel)(*[o.data_ptr() for o in outs])
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()

    def call(ctx):
        return N.lib().art_context_compute_device(ctx.handle, j.nchannel, ch, 0.3, (C.c_float * 3)(*[0.001] * 3), 7,
                                                  W, H, ptrs, W, None, C.c_void_p(stream.cuda_stream))

    rcs = []
    with Context(0) as ctx:
        want = _solve(ctx, j)
        for _ in range(2):  # with everything allocated, nothing else stands in the way
            N.check(call(ctx))
        torch.cuda.synchronize()
        with pytest.raises(RuntimeError):  # the refused launch invalidates the capture
            with torch.cuda.graph(torch.cuda.CUDAGraph(), stream=stream, capture_error_mode="thread_local"):
                rcs.append(call(ctx))
    assert rcs == [N.ART_ERR_CUDA]
    with Context(0) as ctx:
        call(ctx)  # reports the refused launch once more
        N.check(call(ctx))
        torch.cuda.synchronize()
    assert all(np.array_equal(o.cpu().numpy().ravel(), w) for o, w in zip(outs, want))


def test_waits_give_up(gpu, monkeypatch):
    """A block that never posts: those that wait for it leave after the limit,
    nobody is given a step formed without it, and the context solves on."""
    import time

    monkeypatch.delenv("ART_RESIDENT", raising=False)
    gave_up = C.c_int32(-1)
    jpegs = [_jpeg(518, 389, "gray"), _jpeg(200, 136, "4:2:0")]
    with Context(0) as ctx:
        want = [_solve(ctx, j) for j in jpegs]
        for j, w in zip(jpegs, want):
            t0 = time.perf_counter()
            N.check(N.lib().art_context_wait_selftest(ctx.handle, 20_000_000, C.byref(gave_up)))
            assert time.perf_counter() - t0 < 10.0
            assert gave_up.value == 1
            N.check(N.lib().art_context_synchronize(ctx.handle))
            assert _equal(_solve(ctx, j), w)
        for limit in (0, -1, 8_000_000_001):
            assert N.lib().art_context_wait_selftest(ctx.handle, limit, C.byref(gave_up)) == N.ART_ERR_INVALID_ARGUMENT


@pytest.mark.parametrize("size,sub,words", [((96, 64), "4:2:0", 0), ((518, 389), "gray", 2)])
def test_no_buffers_of_its_own(gpu, monkeypatch, size, sub, words):
    """A first solve allocates what the launch pair's does, and room in the same
    buffers for the exchange words (MiB)."""
    import torch

    j = _jpeg(*size, sub)
    taken = {}
    for mode in ("0", "2"):
        monkeypatch.setenv("ART_RESIDENT", mode)
        taken[mode] = []
        for _ in range(4):  # the first solve of a process also sets CUDA up
            with Context(0) as ctx:
                before = torch.cuda.mem_get_info()[0]
                _solve(ctx, j)
                taken[mode].append((before - torch.cuda.mem_get_info()[0]) >> 20)
    assert min(taken["2"]) <= min(taken["0"]) + words, taken


def test_planes_over_exchange_words(gpu, monkeypatch):
    """Planes of a larger solve cover the place of earlier exchange words."""
    small, large = _jpeg(518, 389, "gray"), _jpeg(720, 600, "gray")
    monkeypatch.setenv("ART_RESIDENT", "0")
    with Context(0) as ctx:
        want = [_solve(ctx, small), _solve(ctx, large)]
    with Context(0) as ctx:
        for _ in range(2):
            monkeypatch.setenv("ART_RESIDENT", "2")
            assert _equal(_solve(ctx, small), want[0])
            monkeypatch.setenv("ART_RESIDENT", "0")
            assert _equal(_solve(ctx, large), want[1])
            monkeypatch.setenv("ART_RESIDENT", "2")
            assert _equal(_solve(ctx, large), want[1])
