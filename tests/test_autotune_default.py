"""The autotuner times the library's own tiling (nothing configured) of every
blocksize beside the configured ones: a configured h bounds the levels of an
overlapped block, so without it a tuned solver could only be slower than an untuned
one (no GPU needed)."""
import pytest
import torch

from pysweep_b200 import autotune


@pytest.mark.parametrize("eq,n,rate,want", [
    ("heat", 1400, lambda bs, h, nseg: 10.0 if h == 0 else h / 100, {"blocksize": 8, "h": 0, "nseg": 0}),
    ("heat", 384, lambda bs, h, nseg: bs + (0.5 if h == 0 else 0.0), {"blocksize": 64, "h": 0, "nseg": 0}),
    ("half", 256, lambda bs, h, nseg: 1.0 if (bs, h, nseg) == (16, 5, 0) else 0.5,
     {"blocksize": 16, "h": 5, "nseg": 0}),
])
def test_own_tiling_is_among_the_timed_ones(monkeypatch, eq, n, rate, want):
    timed = []

    def fake(equation, nx, ny, nv, its, ops, bs, h, nseg, levels, reps, device, field):
        timed.append((bs, h, nseg))
        return rate(bs, h, nseg)

    monkeypatch.setattr(autotune, "_time_config", fake)
    monkeypatch.setattr(torch.Tensor, "cuda", lambda self, device=None: self)
    best = autotune.tune(eq, n, n, use_cache=False)
    assert {k: best[k] for k in want} == want
    sizes = {bs for bs, _, _ in autotune.candidates(eq, n, n)}
    assert {(bs, 0, 0) for bs in sizes} <= set(timed) and len(timed) == len(set(timed))
    assert set(autotune.candidates(eq, n, n)) <= set(timed)
