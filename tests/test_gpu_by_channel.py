"""Outputs by channel of few and many channels, which tensor-core tiles write in place or
through an array that is turned (needs a GB300)."""
import numpy as np
import pytest

import fast_matched_filter_gb300 as fmf
from tests._cases import random_search

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("SC", [1, 2, 9, 10, 11])
@pytest.mark.parametrize("normalize", ["short", "full"])
def test_outputs_by_channel_equal_the_cuda_cores(monkeypatch, SC, normalize):
    """Both within 22 * 2^-23 of exact (half of it the CUDA cores')."""
    tp, mo, w, d = random_search(SC, 3, SC, 1, 100, 9001, -40, 300, dc=1.0, zero_weights=SC // 3)
    monkeypatch.setenv("FMF_TC32", "0")
    plain = fmf.matched_filter(tp, mo, w, d, 1, check_zeros=False, normalize=normalize, network_sum=False)
    monkeypatch.setenv("FMF_TC32", "64")
    got = fmf.matched_filter(tp, mo, w, d, 1, check_zeros=False, normalize=normalize, network_sum=False)
    assert np.array_equal(got == 0, plain == 0)
    assert np.abs(got - plain).max() <= 2 * 22 * 2.0 ** -23
    for precision, tol in (("split_bf16", 1e-5), ("bf16", 2e-2)):
        got = fmf.matched_filter(tp, mo, w, d, 1, check_zeros=False, normalize=normalize, network_sum=False,
                                 precision=precision)
        assert np.array_equal(got == 0, plain == 0)
        assert np.abs(got - plain).max() <= tol
