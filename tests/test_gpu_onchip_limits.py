"""Where the GPU does not hold an on-chip solve, the launch pair runs (GPU).

The limits that a context asks CUDA for are set by hand: smaller than what
the GPU holds, as on a part of one, and larger, so that CUDA refuses the launch.
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


def _solve(ctx, j):
    W, H, _ = j.max_rounded()
    return ctx.compute(j.nchannel, j.coefs, 0.3, [0.001] * 3, 5, W, H)


def _route(ctx):
    tiles, cluster = C.c_int32(), C.c_int32()
    N.check(N.lib().art_context_last_onchip(ctx.handle, C.byref(tiles), C.byref(cluster)))
    return tiles.value, cluster.value


# Limits {blocks, cluster} and the route {tiles, cluster} they leave. 96x64: four tiles of 16 rows; 518x389: five
# columns of 25, 13, 9 and 7 tiles of 16, 32, 48 and 64 rows; 1300x1300 gray: 984 tiles of 16 rows.
ROUTES = [
    ((96, 64), "4:2:0", None, (4, 1)), ((96, 64), "4:2:0", (148, 4), (4, 1)), ((96, 64), "4:2:0", (148, 2), (4, 0)),
    ((96, 64), "4:2:0", (0, 4), (4, 1)), ((96, 64), "4:2:0", (3, 2), (2, 1)), ((96, 64), "4:2:0", (0, 0), (0, 0)),
    ((518, 389), "gray", None, (125, 0)), ((518, 389), "gray", (124, 16), (65, 0)),
    ((518, 389), "gray", (36, 16), (35, 0)), ((518, 389), "gray", (20, 8), (0, 0)),
    ((1300, 1300), "gray", None, (0, 0)), ((1300, 1300), "gray", (5000, 16), (0, 0)),
]


@pytest.mark.parametrize("size,sub,limits,route", ROUTES)
def test_solves_within_limits(gpu, monkeypatch, size, sub, limits, route):
    j = _jpeg(*size, sub)
    monkeypatch.setenv("ART_RESIDENT", "0")
    monkeypatch.setenv("ART_STRIP_ROWS", "16")
    with Context(0) as ctx:
        want = _solve(ctx, j)
        assert _route(ctx) == (0, 0)
        monkeypatch.delenv("ART_RESIDENT")
        if limits:
            N.check(N.lib().art_context_set_onchip_limits(ctx.handle, *limits))
        got = _solve(ctx, j)
        assert _route(ctx) == route
        again = _solve(ctx, j)
        assert N.lib().art_context_set_onchip_limits(ctx.handle, 1, -1) == N.ART_ERR_INVALID_ARGUMENT
        N.check(N.lib().art_context_set_onchip_limits(ctx.handle, -1, 0))
        asked = _solve(ctx, _jpeg(96, 64, "4:2:0"))
        assert _route(ctx) == (4, 1) and all(np.isfinite(p).all() for p in asked)
    for planes in (got, again):
        assert all(np.array_equal(a, b) for a, b in zip(planes, want))
