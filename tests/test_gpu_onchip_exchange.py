"""What the blocks of an on-chip solve exchange through global memory (GPU).

Tagged words decide when a block goes on, so no word may carry a tag that its
solve still waits for.
"""
import numpy as np
import pytest

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
