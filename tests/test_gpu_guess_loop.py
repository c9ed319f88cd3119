"""Edges of the line decoder's guess loop against the restatement with the same math: steps cut by
Tmax inside a weight group and at its ends, patterns with three and more high positions, path
metrics beyond the exponential's normal range, ties, long searches, list sizes.  Exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def lines(scale, seed, n=48):
    """Random lines of the given magnitude, some of them noisy codewords."""
    import sogrand_b200 as sg

    rng = np.random.default_rng(seed)
    v = rng.normal(size=(n, 16)) * scale
    bits = sg.encode(rng.integers(0, 256, size=(1, 64), dtype=np.uint8)).reshape(-1, 16)[: n // 2]
    v[: n // 2] = (1.0 - 2.0 * bits) * np.abs(v[: n // 2]) * np.where(rng.random((n // 2, 16)) < 0.06, -1, 1)
    v[-2] = np.where(np.arange(16) % 2, scale, -scale)  # equal magnitudes
    v[-1] = np.round(v[-1] / scale * 4) / 4 * scale      # magnitudes on a grid, some tied
    return v


@pytest.fixture(scope="module", params=[0, 1])
def mode(request, sg, oracle_paths):
    from oracle_api import Oracle

    sg.set_math_mode(request.param)
    yield Oracle(oracle_paths["twin_cr" if request.param else "twin"])
    sg.set_math_mode(0)


def same(sg, oracle, v, **kw):
    ga, ge, gn, gc = sg.bitso(v, **kw)
    ta, te, tn, tc = oracle.bitso(v, **kw)
    assert np.array_equal(gn, tn) and np.array_equal(gc, tc)
    assert np.array_equal(ga.view(np.int64), ta.view(np.int64))
    assert np.array_equal(ge.view(np.int64), te.view(np.int64))


@pytest.mark.parametrize("scale", [1e-3, 0.7, 3.0, 25.0, 60.0, 400.0])
@pytest.mark.parametrize("L", [1, 3, 8])
def test_searches_of_every_length(sg, mode, scale, L):
    same(sg, mode, lines(scale, 11 + L), L=L)


@pytest.mark.parametrize("tmax", [1, 2, 5, 24, 31, 32, 33, 63, 64, 65, 96, 500, 1599, 65535, 65536])
def test_tmax_cuts(sg, mode, tmax):
    same(sg, mode, np.concatenate([lines(0.7, tmax), lines(4.0, tmax + 1)]), L=4, Tmax=tmax)


def test_small_threshold_and_none(sg, mode):
    v = lines(1.5, 3)
    for thres in (0.0, 0.5, 0.999, 1.0, 2.0, -1.0):
        same(sg, mode, v, L=5, thres=thres)
