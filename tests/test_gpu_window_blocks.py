"""Window statistics of large searches, whose usual blocks take fixed-point sums
(needs a GB300): the same search by all channels at once, enough blocks for
those, and channel by channel, which is too few.

Tolerance of one channel's coefficient (|cc| <= 1): an energy is within 2^-24
of its window's on both sides and 2^-26 more on one, and half of that in the
root; reciprocal root, mean and products round to nearest, 4 * 2^-24 on
either side.  In all below 2^-20.
"""
import numpy as np
import pytest

import fast_matched_filter_gb300 as fmf

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("normalize", ["short", "full"])
@pytest.mark.parametrize("L,step", [(1, 1), (15, 1), (16, 7), (600, 1), (601, 50), (2047, 3), (2048, 1), (2049, 1)])
def test_blocks_of_either_kind(monkeypatch, L, step, normalize):
    monkeypatch.setenv("FMF_TC32", "0")
    rng = np.random.default_rng(L + step)
    S, C, N = 4, 2, 79 * 4096 + 5
    d = rng.standard_normal((S, C, N)).astype(np.float32)
    d[0, 1] *= 1e-12                                   # every amplitude is its block's own
    d[1, 0, 50000:60000] = 0.0                         # a gap: windows of zeros, and ones that end in it
    d[1, 1, 70000:75000] *= 1e4                        # a transient
    d[2, 0, 90000] = np.nan
    d[2, 1, 100000] = 1e30
    d[3, 0, 120000:124000] *= np.geomspace(1, 1e-6, 4000).astype(np.float32)
    tp = rng.standard_normal((1, S, C, L)).astype(np.float32)
    tp[0, 0, 1] = d[0, 1, 5000:5000 + L]
    tp[0, 1, 1] = d[1, 1, 72000:72000 + L]
    mo = rng.integers(0, 300, (1, S, C)).astype(np.int32)
    w = np.ones((1, S, C), np.float32)

    def search(sl):
        return fmf.matched_filter(tp[:, sl[0], sl[1]], mo[:, sl[0], sl[1]], w[:, sl[0], sl[1]], d[sl], step,
                                  normalize=normalize, network_sum=False, check_zeros=False)

    together = search((slice(None), slice(None)))
    for s, c in np.ndindex(S, C):
        alone = search((slice(s, s + 1), slice(c, c + 1)))
        n = (N - L - int(mo.max())) // step + 1          # the later moveouts end the search of all
        a, b = alone[0, :n, 0, 0], together[0, :n, s, c]
        assert np.array_equal(np.isfinite(a), np.isfinite(b))
        assert np.array_equal(a == 0, b == 0)
        a, b = np.nan_to_num(a, posinf=0, neginf=0), np.nan_to_num(b, posinf=0, neginf=0)
        assert np.abs(a - b).max() <= 2.0 ** -20, (s, c)


@pytest.mark.parametrize("normalize", ["short", "full"])
@pytest.mark.parametrize("L", [7, 8, 9])
def test_windows_around_the_shortest_of_the_usual_blocks(monkeypatch, L, normalize):
    test_blocks_of_either_kind(monkeypatch, L, 1, normalize)
