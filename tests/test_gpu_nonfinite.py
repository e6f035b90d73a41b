"""Samples and taps that are not finite: what the CUDA cores make of them, the tensor
cores make of them too (needs a GB300)."""
import numpy as np
import pytest

import fast_matched_filter_gb300 as fmf
from tests._cases import random_search

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("step", [1, 2, 65])
def test_sample_of_a_search_with_per_channel_lengths(monkeypatch, step, bad):
    """'short': the energies are running sums of integers, so that only the numerators
    tell of the sample."""
    rng = np.random.default_rng(1)
    tp, mo, w, d = random_search(9, 2, 3, 2, 150 * step, 9000 + 1000 * step, -30, 90, zero_weights=1)
    n = rng.integers(112 * step, 150 * step + 1, mo.shape).astype(np.int32)
    n[0, 0, 0] = 150 * step
    for i in np.ndindex(n.shape):
        tp[i][n[i]:] = 0.0
    w[:, 1, 0] = 0.1
    at = 4000
    d[1, 0, at] = bad

    def search(tile, precision):
        monkeypatch.setenv("FMF_TC32", str(tile))
        return fmf.matched_filter(tp, mo, w, d, step, n_samples_template=n, check_zeros=False, precision=precision)

    plain = search(0, "fp32")
    first = np.arange(plain.shape[1])[None, :] * step + mo[:, 1, 0][:, None]  # of the windows
    holds = np.isnan(plain) & (first <= at) & (at < first + n[:, 1, 0][:, None])
    assert holds.any(axis=1).all()
    assert np.array_equal(search(32, "fp32"), plain, equal_nan=True)  # left to the CUDA cores
    for precision in ("split_bf16", "bf16"):
        got = search(0, precision)
        assert np.isnan(got[holds]).all()
        far = (first > at + 300 * step) | (first + n[:, 1, 0][:, None] < at - 300 * step)
        assert np.isfinite(got[far]).all()


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("normalize", ["short", "full"])
@pytest.mark.parametrize("given", [True, False])
def test_template_that_is_not_finite(monkeypatch, normalize, bad, given):
    """given: with the energies of the templates as they were before."""
    torch = pytest.importorskip("torch")
    tp, mo, w, d = random_search(5, 2, 2, 1, 60, 6000, 0, 50)
    sst = np.sum(tp ** 2, axis=-1) if given else None
    tp[1, 0, 0, 7] = bad
    if not given:
        sst = np.sum(tp ** 2, axis=-1)
    monkeypatch.setenv("FMF_TC32", "0")
    dev = [torch.from_numpy(np.ascontiguousarray(x, x.dtype)).cuda() for x in (tp, sst, mo, w, d)]
    outs = []
    for precision in ("fp32", "split_bf16", "bf16"):
        out = torch.empty((2, 5941, 2, 1), device="cuda")
        fmf.matched_filter_device(*dev, 1, out, normalize, False, precision)
        outs.append(out.cpu().numpy())
    assert given <= (not np.isfinite(outs[0]).all())
    for got in outs[1:]:
        assert np.array_equal(np.isfinite(got), np.isfinite(outs[0]))
