"""Launch shapes of small images with the on-chip solver off, and on-chip
solves with every height of norm strips (GPU).

The shapes named here are the ones that run: images of these sizes go on chip
unless ART_RESIDENT=0 keeps them off.
"""
import numpy as np
import pytest

from artefact_b200 import synth
from artefact_b200.api import Context, Jpeg, JpegSource
from parity import check_parity

pytestmark = pytest.mark.gpu

SHAPES = [(72, 40, "4:2:0", False), (200, 136, "4:4:4", False), (128, 96, "4:2:2", False), (96, 64, "4:4:4", True)]


def _jpeg(w, h, sub, gray, seed):
    return Jpeg.from_source(JpegSource.Buffer(synth.make_jpeg(w, h, 80, sub, gray, seed=seed)))


def _solve(j, iterations):
    W, H, _ = j.max_rounded()
    with Context(0) as ctx:
        return ctx.compute(j.nchannel, j.coefs, 0.3, [0.001] * 3, iterations, W, H)


def _equal(a, b):
    return all(np.array_equal(x, y) for x, y in zip(a, b))


@pytest.mark.parametrize("rows", [16, 32, 64, 128])
@pytest.mark.parametrize("kind", [0, 1, 2])
@pytest.mark.parametrize("shape", SHAPES)
def test_launch_pair_shapes_agree(gpu, monkeypatch, shape, kind, rows):
    """Against the oracle; 2, 4 and 8 projection warps give identical planes."""
    j = _jpeg(*shape, seed=900 + shape[0])
    monkeypatch.setenv("ART_RESIDENT", "0")
    monkeypatch.setenv("ART_SWEEP_KIND", str(kind))
    monkeypatch.setenv("ART_STRIP_ROWS", str(rows))
    outs = []
    for warps in (2, 4, 8):
        monkeypatch.setenv("ART_PROJ_WARPS", str(warps))
        outs.append(_solve(j, 30))
    assert _equal(outs[1], outs[0]) and _equal(outs[2], outs[0])
    check_parity(j, 30, label=f"{shape} sweep {kind} rows {rows}", gpu=outs[0])


@pytest.mark.parametrize("rows", [8, 16, 20, 32, 48, 64, 96])
@pytest.mark.parametrize("sub", ["gray", "4:4:4", "4:2:2", "4:2:0"])
@pytest.mark.parametrize("size", [(72, 40), (200, 136), (520, 264)])
def test_onchip_strip_heights(gpu, monkeypatch, size, sub, rows):
    """Tiles of several norm strips, and taller tiles, equal the launch pair bit
    for bit (a height that no tile has runs as the launch pair itself)."""
    j = _jpeg(*size, "4:4:4" if sub == "gray" else sub, sub == "gray", seed=5)
    monkeypatch.setenv("ART_STRIP_ROWS", str(rows))
    monkeypatch.setenv("ART_RESIDENT", "0")
    want = _solve(j, 11)
    for mode in ("1", "2"):
        monkeypatch.setenv("ART_RESIDENT", mode)
        assert _equal(_solve(j, 11), want), mode
