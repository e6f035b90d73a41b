"""The FP32 form on the tensor cores, at the sizes where its tiles, K steps and
chains end (needs a GB300).

Tolerance, per channel of weight 1 (|cc| <= 1): a chain of at most 16 K steps
loses up to 2^-23 of its partial sum at each (the tensor core truncates), the
partial sums of all chains together are at most 1 (Cauchy-Schwarz), so 16 *
2^-23; an operand pair is within 2^-23 of its value and l * l is dropped, two
more; the additions of the chains, the window energy, the reciprocal root and
the network sum round to nearest, 8 * 2^-24 with room.  In all 22 * 2^-23 =
2.6e-6 for weights that sum to 1.
"""
import numpy as np
import pytest

import fast_matched_filter_gb300 as fmf
from fast_matched_filter_gb300 import _lib
from oracle import fp64
from tests._cases import random_search

pytestmark = pytest.mark.gpu
TOL = 22 * 2.0 ** -23


def _search(monkeypatch, tile, tp, mo, w, d, step=1, **kw):
    monkeypatch.setenv("FMF_TC32", str(tile))
    return fmf.matched_filter(tp, mo, w, d, step, check_zeros=False, **kw)


def _check(got, ref):
    assert np.array_equal(got == 0, ref == 0)
    err = np.abs(got.astype(np.float64) - ref)
    assert err.max() <= TOL, "max %.3g at %s" % (err.max(), np.unravel_index(err.argmax(), err.shape))


@pytest.mark.parametrize("tile", [32, 64, 128])
@pytest.mark.parametrize("extra", [-1, 0, 1, 129])
def test_output_counts_around_a_tile(monkeypatch, tile, extra):
    # n_corr one short of a tile, a tile, one more, one row and one more
    L = 33
    N = 128 * tile + extra + L - 1
    tp, mo, w, d = random_search(tile + extra, 2, 2, 1, L, N, -9, 140)
    got = _search(monkeypatch, tile, tp, mo, w, d)
    _check(got, fp64.fp64_matched_filter(tp, mo, w, d, 1, "short", True))


@pytest.mark.parametrize("L", [1, 15, 16, 17, 113, 128, 129, 143, 144, 145, 257, 1201])
@pytest.mark.parametrize("normalize", ["short", "full"])
def test_template_lengths_around_k_steps_and_chains(monkeypatch, L, normalize):
    tp, mo, w, d = random_search(L, 2, 2, 2, L, 5000 + L, -130, 260, dc=3.0, zero_weights=1)
    got = _search(monkeypatch, 32, tp, mo, w, d, normalize=normalize)
    _check(got, fp64.fp64_matched_filter(tp, mo, w, d, 1, normalize, True))


@pytest.mark.parametrize("step", [2, 3, 7, 50])
@pytest.mark.parametrize("network_sum", [True, False])
def test_phases_of_a_decimated_search(monkeypatch, step, network_sum):
    tp, mo, w, d = random_search(step, 2, 2, 2, 45, 9000 + step, -40, 300, dc=1.0, zero_weights=1)
    got = _search(monkeypatch, 32, tp, mo, w, d, step, normalize="full", network_sum=network_sum)
    ref = fp64.fp64_matched_filter(tp, mo, w, d, step, "full", network_sum)
    _check(got, ref.reshape(got.shape))


@pytest.mark.parametrize("parts", [1, 2, 5])
def test_channel_parts(monkeypatch, parts):
    monkeypatch.setenv("FMF_TC_PARTS", str(parts))
    tp, mo, w, d = random_search(50 + parts, 3, 3, 2, 90, 20000, 0, 200, zero_weights=4)
    got = _search(monkeypatch, 128, tp, mo, w, d)
    _check(got, fp64.fp64_matched_filter(tp, mo, w, d, 1, "short", True))


@pytest.mark.parametrize("normalize", ["short", "full"])
def test_per_channel_lengths(monkeypatch, normalize):
    rng = np.random.default_rng(8)
    tp, mo, w, d = random_search(9, 2, 3, 2, 150, 9000, -30, 90, dc=2.0, zero_weights=1)
    n = rng.integers(20, 151, mo.shape).astype(np.int32)
    n[0, 0, 0] = 150
    for i in np.ndindex(n.shape):
        tp[i][n[i]:] = 0.0
    got = _search(monkeypatch, 32, tp, mo, w, d, normalize=normalize, n_samples_template=n)
    ref = fp64.fp64_matched_filter_variable(tp, n, mo, w, d, 1, normalize)
    # up to |cc| = 0.9 the inverse hyperbolic tangent grows an error by 1 / (1 - 0.81) < 6
    scale = np.cumsum(w.reshape(2, -1).sum(axis=1))[:, None]
    assert (np.abs(got - ref) / scale).max() <= 6 * TOL


def _both(monkeypatch, tp, mo, w, d, **kw):
    return [_search(monkeypatch, tile, tp, mo, w, d, **kw) for tile in (0, 32)]


@pytest.mark.parametrize("normalize", ["short", "full"])
@pytest.mark.parametrize("bad", [np.nan, np.inf, 1e30])
def test_values_that_are_not_finite_or_huge(monkeypatch, normalize, bad):
    """A sample that is not finite (or whose square is not) silences the windows
    that hold it, and no others, as on the CUDA cores."""
    tp, mo, w, d = random_search(3, 2, 2, 2, 60, 6000, 0, 50)
    d[0, 0, 3000] = bad
    plain, tensor = _both(monkeypatch, tp, mo, w, d, normalize=normalize, network_sum=False)
    assert np.array_equal(np.isfinite(plain), np.isfinite(tensor))
    assert np.array_equal(plain == 0, tensor == 0)
    assert np.abs(plain - tensor).max() <= 2 * TOL


@pytest.mark.parametrize("scale", [1e-14, 1e-9, 1e9, 1e18])
def test_amplitudes_beside_one_another(monkeypatch, scale):
    """Quiet windows far below the channel's largest value, and template and data
    amplitudes far apart: what the operand pairs cannot hold runs on the CUDA
    cores."""
    tp, mo, w, d = random_search(4, 2, 2, 1, 60, 6000, 0, 50)
    tp = (tp / np.float32(scale)).astype(np.float32)
    d = (d * np.float32(scale)).astype(np.float32)
    d[1, 0, :2000] *= np.float32(1e7)
    plain, tensor = _both(monkeypatch, tp, mo, w, d)
    assert plain.any()
    assert np.array_equal(plain == 0, tensor == 0)
    assert np.abs(plain - tensor).max() <= 2 * TOL


def test_template_that_is_not_finite(monkeypatch):
    tp, mo, w, d = random_search(5, 2, 2, 1, 60, 6000, 0, 50)
    tp[1, 0, 0, 7] = np.inf
    plain, tensor = _both(monkeypatch, tp, mo, w, d)
    assert np.array_equal(plain, tensor, equal_nan=True)  # the CUDA cores ran both


def test_many_channels_written_one_by_one(monkeypatch):
    """Per-channel outputs of full tiles: the epilogue's stores, 36 channels apart,
    hold up its reads of the window statistics."""
    tp, mo, w, d = random_search(11, 3, 12, 3, 100, 60000, 0, 300)
    plain, tensor = [_search(monkeypatch, tile, tp, mo, w, d, network_sum=False) for tile in (0, 128)]
    assert np.array_equal(plain == 0, tensor == 0)
    assert np.abs(plain - tensor).max() <= 2 * TOL


@pytest.mark.parametrize("step,L", [(32, 100), (33, 100), (64, 200), (65, 200), (8, 6144), (8, 6145)])
@pytest.mark.parametrize("normalize", ["short", "full"])
def test_operands_of_large_steps_and_long_templates(monkeypatch, step, L, normalize):
    """Where a block turns two rows of every phase, one, and none (a kernel of its own);
    and where the templates' shared memory gives them a launch of their own."""
    tp, mo, w, d = random_search(step + L, 2, 2, 2, L, 150 * step + L + 4000, -200, 300, dc=1.0, zero_weights=1)
    got = _search(monkeypatch, 32, tp, mo, w, d, step, normalize=normalize)
    _check(got, fp64.fp64_matched_filter(tp, mo, w, d, step, normalize, True))


@pytest.mark.parametrize("channels", [2, 64, 65, 130])
def test_channels_written_one_by_one_around_a_tile(monkeypatch, channels):
    """Per-channel outputs are turned 64 channels at a time."""
    tp, mo, w, d = random_search(channels, 2, channels, 1, 40, 4200, -20, 60, zero_weights=1)
    plain, tensor = [_search(monkeypatch, tile, tp, mo, w, d, network_sum=False) for tile in (0, 32)]
    assert np.array_equal(plain == 0, tensor == 0)
    assert np.abs(plain - tensor).max() <= 2 * TOL


@pytest.mark.parametrize("step", [1, 3])
@pytest.mark.parametrize("normalize", ["short", "full"])
def test_per_channel_lengths_of_a_decimated_search(monkeypatch, step, normalize):
    rng = np.random.default_rng(step)
    tp, mo, w, d = random_search(21, 2, 3, 2, 150, 9000, -30, 90, dc=2.0)
    n = rng.integers(20, 151, mo.shape).astype(np.int32)
    n[0, 0, 0] = 150
    for i in np.ndindex(n.shape):
        tp[i][n[i]:] = 0.0
    got = _search(monkeypatch, 32, tp, mo, w, d, step, normalize=normalize, n_samples_template=n)
    ref = fp64.fp64_matched_filter_variable(tp, n, mo, w, d, step, normalize)
    scale = np.cumsum(w.reshape(2, -1).sum(axis=1))[:, None]
    assert (np.abs(got - ref) / scale).max() <= 6 * TOL  # as in test_per_channel_lengths


@pytest.mark.parametrize("small", [True, False])
def test_batch_of_fp32_searches(small):
    """Searches of a batch on the tensor cores and, the small ones, on the CUDA cores;
    both normalisations and output layouts."""
    import torch

    b = fmf.Batch("fp32")
    want = []
    for i in range(6):
        T, N = (1, 900) if small and i % 2 else (12, 14000)
        tp, mo, w, d = random_search(60 + i, T, 3, 2, 100, N, 0, 120, dc=1.0)
        normalize, network_sum = ("full", "short")[i % 2], i < 4
        n_corr = N - 100 + 1
        out = torch.zeros((T, n_corr) if network_sum else (T, n_corr, 3, 2), device="cuda")
        dev = [torch.tensor(x).cuda() for x in (tp, (tp * tp).sum(axis=-1), mo, w, d)]
        b.add(*dev, 1, out, normalize=normalize, network_sum=network_sum)
        want.append((out, dev, fp64.fp64_matched_filter(tp, mo, w, d, 1, normalize, network_sum)))
    b.run()
    torch.cuda.synchronize()
    for out, _, ref in want:
        _check(out.cpu().numpy(), ref.reshape(tuple(out.shape)))


@pytest.mark.parametrize("L", [56, 80, 112, 160, 257, 300, 600, 800, 1200])
@pytest.mark.parametrize("step", [1, 3])
@pytest.mark.parametrize("noise", [0.1, 0.5])
def test_error_at_matches_is_no_larger_than_on_the_cuda_cores(monkeypatch, L, step, noise):
    """RMS over 2,000 copies of a template of several amplitudes, in noise; a tenth for the
    scatter of two such figures (their relative standard deviations are 1 / sqrt(4,000))."""
    rng = np.random.default_rng(L + step)
    S, K = 8, 250
    slot = ((L + 20) // step + 1) * step
    tp = (rng.standard_normal((1, S, 1, L)) * np.hanning(L + 2)[1:-1]).astype(np.float32)
    d = rng.standard_normal((S, 1, K * slot + L)) * noise * tp.std()
    at = np.arange(K) * slot
    for a in at:
        d[:, 0, a:a + L] += rng.uniform(0.3, 3.0, (S, 1)) * tp[0, :, 0]
    d = d.astype(np.float32)
    mo, w = np.zeros((1, S, 1), np.int32), np.ones((1, S, 1), np.float32)
    t64 = tp[0, :, 0].astype(np.float64)
    win = np.stack([d[:, 0, a:a + L] for a in at]).astype(np.float64)
    ref = (win * t64).sum(-1) / np.sqrt((t64 ** 2).sum(-1) * (win ** 2).sum(-1))
    plain, tensor = [_search(monkeypatch, tile, tp, mo, w, d, step, network_sum=False)[0, at // step, :, 0] - ref
                     for tile in (0, 64)]
    assert np.sqrt((tensor ** 2).mean()) <= 1.1 * np.sqrt((plain ** 2).mean())


@pytest.mark.parametrize("normalize", ["short", "full"])
@pytest.mark.parametrize("step", [1, 2])
def test_per_channel_lengths_of_one_and_several_chains(monkeypatch, normalize, step):
    """Long channels, whose column-block pairs are several chains each, beside short ones."""
    rng = np.random.default_rng(10)
    tp, mo, w, d = random_search(12, 2, 3, 2, 1300, 9000, -30, 90, dc=2.0, zero_weights=1)
    n = rng.integers(56, 1301, mo.shape).astype(np.int32)
    n[0, 0, 0] = 1300
    for i in np.ndindex(n.shape):
        tp[i][n[i]:] = 0.0
    got = _search(monkeypatch, 32, tp, mo, w, d, step, normalize=normalize, n_samples_template=n)
    ref = fp64.fp64_matched_filter_variable(tp, n, mo, w, d, step, normalize)
    scale = np.cumsum(w.reshape(2, -1).sum(axis=1))[:, None]
    assert (np.abs(got - ref) / scale).max() <= 6 * TOL


def _ran():
    """0: the CUDA cores; 1: the tensor cores; 2: they left it to the CUDA cores."""
    return _lib.load().fmf_last_tensor_cores()


@pytest.mark.parametrize("normalize", ["short", "full"])
@pytest.mark.parametrize("network_sum", [True, False])
@pytest.mark.parametrize("tile", [0, 32, 64, 128])
@pytest.mark.parametrize("step", [1, 3])
def test_ordinary_searches_run_where_they_are_sent(monkeypatch, normalize, network_sum, tile, step):
    """Noise, levels, a gap of zeros, amplitudes a thousand apart."""
    tp, mo, w, d = random_search(21, 2, 3, 2, 100, 9000, -20, 90, dc=1.0, zero_weights=1)
    d[1] *= np.float32(1e3)
    tp[:, 2] *= np.float32(1e-3)
    d[0, :, 2000:2500] = d[0, :, 2000:2001]
    _ran()
    _search(monkeypatch, tile, tp, mo, w, d, step, normalize=normalize, network_sum=network_sum)
    assert _ran() == (tile != 0)


@pytest.mark.parametrize("normalize", ["short", "full"])
def test_ordinary_searches_with_per_channel_lengths_run_where_they_are_sent(monkeypatch, normalize):
    rng = np.random.default_rng(22)
    tp, mo, w, d = random_search(23, 2, 3, 2, 200, 9000, -20, 90, dc=1.0, zero_weights=1)
    n = rng.integers(100, 201, mo.shape).astype(np.int32)
    n[0, 0, 0] = 200
    for i in np.ndindex(n.shape):
        tp[i][n[i]:] = 0.0
    for tile in (0, 64):
        _search(monkeypatch, tile, tp, mo, w, d, normalize=normalize, n_samples_template=n)
        assert _ran() == (tile != 0)
    d[2, 0, 5000] = np.nan
    _search(monkeypatch, 64, tp, mo, w, d, normalize=normalize, n_samples_template=n)
    assert _ran() == 2


@pytest.mark.parametrize("change,ran", [("nan sample", 1), ("nan tap", 2), ("loud data", 2), ("faint template", 2),
                                        ("transient", 2)])
def test_what_operand_pairs_cannot_hold_is_left_to_the_cuda_cores(monkeypatch, change, ran):
    tp, mo, w, d = random_search(24, 2, 2, 1, 60, 6000, 0, 50)
    if change == "nan sample":
        d[0, 0, 3000] = np.nan
    elif change == "nan tap":
        tp[1, 0, 0, 7] = np.nan
    elif change == "loud data":
        d[1] *= np.float32(1e19)
    elif change == "faint template":
        tp[0, 1] *= np.float32(1e-13)
    else:
        d[1, 0, 100] = 1e8
    _ran()
    _search(monkeypatch, 32, tp, mo, w, d)
    assert _ran() == ran


@pytest.mark.parametrize("device", [False, True])
@pytest.mark.parametrize("shortest,weight,ran", [(55, 0.1, 0), (56, 0.1, 1), (10, 0.0, 1), (10, 0.1, 0)])
def test_per_channel_lengths_by_the_shortest_of_weight(monkeypatch, shortest, weight, ran, device):
    torch = pytest.importorskip("torch")
    tp, mo, w, d = random_search(25, 2, 3, 2, 150, 9000, -20, 90)
    n = np.full(mo.shape, 150, np.int32)
    n[1, 2, 0] = shortest
    w[1, 2, 0] = weight
    tp[1, 2, 0, shortest:] = 0.0
    if not device:
        _search(monkeypatch, 64, tp, mo, w, d, n_samples_template=n)
    else:
        monkeypatch.setenv("FMF_TC32", "64")
        lib = _lib.load()
        g = [torch.from_numpy(x).cuda() for x in (tp, np.sum(tp ** 2, axis=-1), mo, d, w, n)]
        out = torch.empty((2, 8851), device="cuda")
        torch.cuda.synchronize()
        _lib.check(lib.fmf_matched_filter_variable_ex(
            *[x.data_ptr() for x in g[:5]], 1, g[5].data_ptr(), 9000, 2, 3, 2, 8851, out.data_ptr(), 0,
            _lib.FLAG_DEVICE_POINTERS, None), lib)
    assert _ran() == ran


@pytest.mark.parametrize("T,SC,L,step,n_corr,ran", [(100, 9, 300, 20, 300, 0), (10, 9, 300, 20, 300, 1),
                                                    (100, 9, 300, 20, 5000, 1), (100, 9, 1600, 20, 300, 1)])
def test_many_templates_of_few_lags_stay_on_the_cuda_cores(T, SC, L, step, n_corr, ran):
    """A search on either side of the line by each of its sizes."""
    tp, mo, w, d = random_search(41, T, SC, 1, L, n_corr * step + L - 1, 0, 50, plant=False)
    fmf.matched_filter(tp, mo, w, d, step, check_zeros=False)
    assert _ran() == ran


@pytest.mark.parametrize("step,L", [(60, 59), (60, 60), (60, 61), (200, 56), (300, 1)])
@pytest.mark.parametrize("network_sum", [True, False])
def test_steps_around_and_past_the_template(monkeypatch, step, L, network_sum):
    """Phases past the last tap are left out."""
    tp, mo, w, d = random_search(step + L, 3, 2, 2, L, 40 * step + L, -200, 300, zero_weights=1)
    got = _search(monkeypatch, 32, tp, mo, w, d, step, network_sum=network_sum)
    ref = fp64.fp64_matched_filter(tp, mo, w, d, step, "short", network_sum)
    _check(got, ref.reshape(got.shape))


@pytest.mark.parametrize("precision", ["fp32", "split_bf16"])
def test_per_channel_lengths_past_the_step_and_below(monkeypatch, precision):
    rng = np.random.default_rng(31)
    tp, mo, w, d = random_search(32, 2, 3, 2, 150, 16000, -30, 90, zero_weights=1)
    n = rng.integers(56, 151, mo.shape).astype(np.int32)
    n[0, 0, 0] = 150
    for i in np.ndindex(n.shape):
        tp[i][n[i]:] = 0.0
    got = _search(monkeypatch, 32, tp, mo, w, d, 100, n_samples_template=n, precision=precision)
    ref = fp64.fp64_matched_filter_variable(tp, n, mo, w, d, 100, "short")
    scale = np.cumsum(w.reshape(2, -1).sum(axis=1))[:, None]
    assert (np.abs(got - ref) / scale).max() <= (6 * TOL if precision == "fp32" else 1e-4)


@pytest.mark.parametrize("step", [1, 5, 100])
@pytest.mark.parametrize("n", [56, 58, 62, 79, 81, 99, 100, 149])
def test_chains_of_channels_shorter_than_the_longest(monkeypatch, n, step):
    """The issuer and the epilogue count a channel's chains apart."""
    tp, mo, w, d = random_search(n, 2, 2, 1, 150, 6000 + 10 * step, -30, 90)
    lengths = np.full(mo.shape, 150, np.int32)
    lengths[:, 1] = n
    tp[:, 1, :, n:] = 0.0
    got = _search(monkeypatch, 32, tp, mo, w, d, step, n_samples_template=lengths)
    ref = fp64.fp64_matched_filter_variable(tp, lengths, mo, w, d, step, "short")
    scale = np.cumsum(w.reshape(2, -1).sum(axis=1))[:, None]
    assert (np.abs(got - ref) / scale).max() <= 6 * TOL
