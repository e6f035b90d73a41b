"""Results in fresh host memory, around the sizes at which its pages are mapped ahead
of the copy and in pieces (needs a GB300): equal to those left on the device."""
import numpy as np
import pytest

import fast_matched_filter_gb300 as fmf
from fast_matched_filter_gb300 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("megabytes", [0.01, 1, 15.9, 16.1, 63.9, 64.1])
@pytest.mark.parametrize("T", [1, 9])
def test_host_output_equals_device_output(megabytes, T):
    import torch

    L = 16
    n_corr = int(megabytes * 2 ** 20 / (4 * T)) + 1
    rng = np.random.default_rng(T)
    tp = rng.standard_normal((T, 1, 1, L)).astype(np.float32)
    d = rng.standard_normal((1, 1, n_corr + L - 1)).astype(np.float32)
    mo, w = np.zeros((T, 1, 1), np.int32), np.ones((T, 1, 1), np.float32)
    got = fmf.matched_filter(tp, mo, w, d, 1, check_zeros=False)
    out = torch.empty((T, n_corr), device="cuda")
    fmf.matched_filter_device(torch.tensor(tp).cuda(), None, torch.tensor(mo).cuda(), torch.tensor(w).cuda(),
                              torch.tensor(d).cuda(), 1, out)
    torch.cuda.synchronize()
    assert np.array_equal(got, out.cpu().numpy())
    given = np.empty(T * n_corr + 1, np.float32)[1:].reshape(T, n_corr)  # not on a page
    fmf.matched_filter(tp, mo, w, d, 1, check_zeros=False, out=given)
    assert np.array_equal(given, got)


@pytest.mark.parametrize("bad", [None, np.inf, 1e30])
@pytest.mark.parametrize("network_sum", [True, False])
def test_parts_of_an_fp32_search_run_on_the_same_cores(monkeypatch, bad, network_sum):
    """A result copied in pieces behind the kernels of parts of the templates, and the same
    on the device in one: the last template decides for both."""
    import torch

    monkeypatch.setenv("FMF_TC32", "128")
    T, L, n_corr = 9, 60, int(64.1 * 2 ** 20 / (4 * 9)) + 1
    if not network_sum:
        n_corr //= 2
    rng = np.random.default_rng(3)
    tp = rng.standard_normal((T, 2, 1, L)).astype(np.float32)
    if bad is not None:
        tp[T - 1, 1, 0, 5] = bad
    d = rng.standard_normal((2, 1, n_corr + L - 1)).astype(np.float32)
    mo, w = np.zeros((T, 2, 1), np.int32), np.ones((T, 2, 1), np.float32)
    with np.errstate(all="ignore"):
        sst = np.sum(tp ** 2, axis=-1)
    lib = _lib.load()
    lib.fmf_last_tensor_cores()
    with np.errstate(all="ignore"):
        got = fmf.matched_filter(tp, mo, w, d, 1, check_zeros=False, network_sum=network_sum)
    assert lib.fmf_last_tensor_cores() == (1 if bad is None else 2)
    out = torch.empty((T, n_corr) if network_sum else (T, n_corr, 2, 1), device="cuda")
    fmf.matched_filter_device(*[torch.tensor(x).cuda() for x in (tp, sst, mo, w, d)], 1, out, "short", network_sum)
    assert lib.fmf_last_tensor_cores() == (1 if bad is None else 2)
    assert np.array_equal(got, out.cpu().numpy(), equal_nan=True)
