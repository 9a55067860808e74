"""Iterations of dependent launches against ordinary ones (GPU).

An iteration's kernels are launched as dependents of one another, except while
a context records events between them (timing) or a batch needs several sweep
launches. The kernels are the same, so the planes must be equal bit for bit.
"""
import numpy as np
import pytest

from artefact_b200 import _native as N, synth
from artefact_b200.api import Context, Jpeg, JpegSource

pytestmark = pytest.mark.gpu

BATCHES = {
    "gray": ["gray"] * 3, "444": ["4:4:4"] * 3, "422": ["4:2:2"] * 2, "420": ["4:2:0"] * 3,
    "subsampled": ["4:2:0", "4:2:2", "4:2:0"], "all": ["4:4:4", "4:2:2", "4:2:0"],
    "mixed_channels": ["gray", "4:2:0"],
}
SIZES = [(1000, 667), (17, 9), (1920, 1080)]


def _jpeg(w, h, sub, seed):
    gray = sub == "gray"
    return Jpeg.from_source(JpegSource.Buffer(synth.make_jpeg(w, h, 50, "4:4:4" if gray else sub, gray, seed=seed)))


@pytest.mark.parametrize("name", sorted(BATCHES))
def test_dependent_launches_equal_ordinary_ones(gpu, name):
    jobs = [dict(coefs=_jpeg(*SIZES[i], sub, seed=20 + i).coefs) for i, sub in enumerate(BATCHES[name])]
    with Context(0) as ctx:
        got = [ctx.compute_batch(jobs, 12) for _ in range(3)]
        N.check(N.lib().art_context_set_timing(ctx.handle, 1))
        want = ctx.compute_batch(jobs, 12)
    for g in got:
        assert all(np.array_equal(a, b) for pa, pb in zip(g, want) for a, b in zip(pa, pb))


def test_planes_beyond_l2_equal_planes_within(gpu, monkeypatch):
    """The projection stages in another order, and without L2 hints, where the
    planes of a solve exceed 200 MiB: a batch above the line against its images
    alone, with the same norm strips."""
    monkeypatch.setenv("ART_STRIP_ROWS", "32")
    monkeypatch.setenv("ART_RESIDENT", "0")
    subs = ["4:2:0", "4:2:2", "4:4:4", "gray"]
    jobs = [dict(coefs=_jpeg(*SIZES[i % 2], sub, seed=40 + i).coefs) for i, sub in enumerate(subs)]
    jobs += [dict(coefs=_jpeg(1920, 1080, "4:4:4", seed=50).coefs)] * 3
    with Context(0) as ctx:
        got = ctx.compute_batch(jobs, 6)
        for job, g in zip(jobs[:5], got):
            alone = ctx.compute_batch([job], 6)[0]
            assert all(np.array_equal(a, b) for a, b in zip(g, alone))
