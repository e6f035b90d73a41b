"""FP32 searches with too little memory for the tensor cores' operands run on the CUDA
cores, whichever call they come through (needs a GB300)."""
import contextlib

import numpy as np
import pytest

import fast_matched_filter_gb300 as fmf
from fast_matched_filter_gb300 import _lib

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _search(T=500, S=20, C=3, L=600, N=20000):
    """Operands of 950 MB; 5 MB of window statistics and 40 MB of outputs."""
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    tp = torch.randn((T, S, C, L), device="cuda", generator=g)
    d = torch.randn((S, C, N), device="cuda", generator=g)
    mo = torch.zeros((T, S, C), dtype=torch.int32, device="cuda")
    w = torch.full((T, S, C), 1 / (S * C), device="cuda")
    return (tp, (tp * tp).sum(-1), mo, w, d), torch.empty((T, N - L + 1), device="cuda")


@contextlib.contextmanager
def _little_memory(megabytes):
    torch.cuda.synchronize()
    lib = _lib.load()
    _lib.check(lib.fmf_release_cache(), lib)
    hold = torch.empty(torch.cuda.mem_get_info()[0] - (megabytes << 20), dtype=torch.uint8, device="cuda")
    try:
        yield
    finally:
        del hold
        torch.cuda.empty_cache()


def test_batch(monkeypatch):
    args, out = _search()
    monkeypatch.setenv("FMF_TC32", "0")
    want = torch.empty_like(out)
    fmf.matched_filter_device(*args, 1, want)
    monkeypatch.delenv("FMF_TC32")
    b = fmf.Batch("fp32")
    b.add(*args, 1, out)
    with _little_memory(500):
        for _ in range(2):
            out.zero_()
            b.run()
            torch.cuda.synchronize()
            assert np.array_equal(out.cpu().numpy(), want.cpu().numpy())
    b.close()


@pytest.mark.parametrize("megabytes", [500, 1180])
def test_search_and_detection(megabytes):
    """1,180 MB hold the operands (945) or what detection needs (220) beside inputs, sums and
    statistics (120)."""
    args, _ = _search()
    tp, _, mo, w, d = [x.cpu().numpy() for x in args]
    del args
    torch.cuda.empty_cache()
    first = fmf.matched_filter_detect(tp, mo, w, d, 1)
    with _little_memory(megabytes):
        again = fmf.matched_filter_detect(tp, mo, w, d, 1)
    assert np.array_equal(first.count, again.count) or megabytes == 500
    assert np.abs(first.threshold - again.threshold).max() <= 1e-6


@pytest.mark.parametrize("lengths", [False, True])
@pytest.mark.parametrize("normalize", ["short", "full"])
def test_statistics_of_a_large_step(monkeypatch, normalize, lengths):
    """Tiles of 128 lag blocks have 33,000 statistics of padding round each of the 3,000 rows
    of 60 channels at step 50: 390 MB and more."""
    T, S, C, L, N, step = 4, 20, 3, 600, 100000, 50
    (tp, sst, mo, w, d), _ = _search(T, S, C, L, N)
    n = torch.full((T, S, C), L, dtype=torch.int32, device="cuda")
    lib = _lib.load()

    def run():
        out = torch.zeros((T, (N - L) // step + 1), device="cuda")
        if lengths:
            _lib.check(lib.fmf_matched_filter_variable_ex(
                *[x.data_ptr() for x in (tp, sst, mo, d, w)], step, n.data_ptr(), N, T, S, C, out.shape[1],
                out.data_ptr(), normalize == "full", _lib.FLAG_DEVICE_POINTERS,
                torch.cuda.current_stream().cuda_stream), lib)
        else:
            fmf.matched_filter_device(tp, sst, mo, w, d, step, out, normalize)
        return out.cpu().numpy()

    monkeypatch.setenv("FMF_TC32", "0")
    want = run()
    monkeypatch.setenv("FMF_TC32", "128")
    with _little_memory(280):
        got = run()
    assert lib.fmf_last_tensor_cores() == 0
    assert np.array_equal(got, want)
