"""The on-chip solver against the launch pair per iteration (GPU).

A solve whose tiles are all resident at once runs its whole iteration loop as
one launch (k_resident): one cluster for up to 16 tiles, a cooperative grid
above. Its arithmetic and its order of summation are those of k_grad_sweep_n
and k_project, so the planes must be equal bit for bit. ART_RESIDENT=0 turns
it off, 1 keeps it from forming clusters.
"""
import numpy as np
import pytest

from artefact_b200 import synth
from artefact_b200.api import Context, Jpeg, JpegSource

pytestmark = pytest.mark.gpu

SIZES = [(8, 8), (112, 16), (113, 17), (224, 32), (120, 130), (200, 136), (520, 264), (632, 472)]


def _jpeg(w, h, sub, seed=3):
    gray = sub == "gray"
    return Jpeg.from_source(JpegSource.Buffer(synth.make_jpeg(w, h, 50, "4:4:4" if gray else sub, gray, seed=seed)))


def _solve(monkeypatch, mode, j, iterations, ctx=None, **kw):
    monkeypatch.setenv("ART_RESIDENT", mode)
    W, H, _ = j.max_rounded()
    own = ctx or Context(0)
    try:
        return own.compute(j.nchannel, j.coefs, 0.3, kw.pop("pweight", [0.001] * 3), iterations, W, H, **kw)
    finally:
        if ctx is None:
            own.close()


def _equal(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a, b))


@pytest.mark.parametrize("sub", ["gray", "4:4:4", "4:2:2", "4:2:0"])
@pytest.mark.parametrize("size", SIZES)
def test_onchip_equals_launch_pair(gpu, monkeypatch, size, sub):
    j = _jpeg(*size, sub)
    want = _solve(monkeypatch, "0", j, 12)
    for mode in ("1", "2"):
        assert _equal(_solve(monkeypatch, mode, j, 12), want), (size, sub, mode)


@pytest.mark.parametrize("iterations,kw", [
    (0, {}), (1, {}), (2, {}), (9, dict(step_iterations=1, step_decay=0.9, tail_iterations=2, tail_step_iterations=100)),
    (6, dict(pweight=[0.0, 0.001, 0.0]))])
def test_onchip_schedules(gpu, monkeypatch, iterations, kw):
    j = _jpeg(200, 136, "4:2:0")
    want = _solve(monkeypatch, "0", j, iterations, **dict(kw))
    for mode in ("1", "2"):
        assert _equal(_solve(monkeypatch, mode, j, iterations, **dict(kw)), want), mode


def test_onchip_context_reused(gpu, monkeypatch):
    """Changing geometry, image and path on one context: what blocks exchange
    in one solve is never taken for the next one's."""
    order = [(200, 136, "gray", 1), (200, 136, "gray", 2), (520, 264, "4:2:0", 1), (96, 64, "4:2:0", 1),
             (520, 264, "4:2:0", 2), (200, 136, "gray", 1)]
    with Context(0) as ctx:
        for w, h, sub, seed in order:
            j = _jpeg(w, h, sub, seed)
            want = _solve(monkeypatch, "0", j, 7)
            for mode in ("2", "1", "0"):
                assert _equal(_solve(monkeypatch, mode, j, 7, ctx=ctx), want), (w, h, sub, seed, mode)
