"""The autotuner and the on-chip solver (GPU).

The tuner chooses the launch pair's shape for a bucket of sizes, some of which
go on chip and some of which do not.
"""
import ctypes as C

import numpy as np
import pytest

from artefact_b200 import _native as N
from artefact_b200 import synth
from artefact_b200.api import Context, Jpeg, JpegSource

pytestmark = pytest.mark.gpu


def _jpeg(w, h, sub):
    return Jpeg.from_source(JpegSource.Buffer(synth.make_jpeg(w, h, 50, sub, False, seed=3)))


def _solve(ctx, j):
    W, H, _ = j.max_rounded()
    return ctx.compute(j.nchannel, j.coefs, 0.3, [0.001] * 3, 9, W, H)


def _tiles(ctx):
    tiles, cluster = C.c_int32(), C.c_int32()
    N.check(N.lib().art_context_last_onchip(ctx.handle, C.byref(tiles), C.byref(cluster)))
    return tiles.value


def test_tuner_times_launch_pairs(gpu):
    """Also where the tuned geometry goes on chip: each candidate's time is that
    of the launches it names."""
    with Context(0) as ctx:
        ctx.autotune(3, [1, 2, 2], [1, 2, 2], 208, 144, iterations=4)
        assert _tiles(ctx) == 0


@pytest.mark.parametrize("choice", ["0 16 8", "0 64 4", "0 128 4", "1 32 4", "2 16 2"])
def test_tuned_bucket_leaves_small_images_on_chip(gpu, tmp_path, monkeypatch, choice):
    """A choice tuned at the bucket's large end (1024x512 4:4:4 does not fit on
    chip) is not taken for the small images of the bucket that do."""
    small, large = _jpeg(520, 264, "4:4:4"), _jpeg(1024, 512, "4:4:4")
    path = tmp_path / "tune.txt"
    path.write_text(f"n3-s111111-w1024-h512 {choice}\n")
    with Context(0) as ctx:
        want = _solve(ctx, small)
        assert _tiles(ctx) > 0
        ctx.load_tune_cache(path)
        got = _solve(ctx, small)
        assert _tiles(ctx) > 0
        tuned = _solve(ctx, large)
        assert _tiles(ctx) == 0
    assert all(np.array_equal(a, b) for a, b in zip(got, want))
    kind, rows, warps = choice.split()
    monkeypatch.setenv("ART_SWEEP_KIND", kind)
    monkeypatch.setenv("ART_STRIP_ROWS", rows)
    monkeypatch.setenv("ART_PROJ_WARPS", warps)
    with Context(0) as ctx:
        assert all(np.array_equal(a, b) for a, b in zip(tuned, _solve(ctx, large)))
