"""Reliabilities at the ends of binary64's range, against the restatement with the same math.  Exact."""
import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=[0, 1])
def mode(request, sg, oracle_paths):
    from oracle_api import Oracle

    sg.set_math_mode(request.param)
    yield Oracle(oracle_paths["twin_cr" if request.param else "twin"])
    sg.set_math_mode(0)


@pytest.mark.parametrize("least", [672.0, 680.5, 686.2, 687.0, 687.4, 688.0, 700.0, 707.6, 708.5, 745.0])
def test_p_not_guess_below_zero(sg, mode, least):
    """Sixteen large magnitudes: the hard decision leaves P_notGuess = 0 and the next patterns move it
    to about -exp(-least), which no later pattern changes.  Every pair of wrong positions, so that the
    first codeword lies anywhere in the steps that follow."""
    mag = np.concatenate([[least], least + 10.0 + np.arange(15.0)])
    v = np.array([np.where(np.isin(np.arange(16), ij), -mag, mag) for ij in itertools.combinations(range(16), 2)])
    for L, tmax in ((3, sg.UINT64_MAX), (8, 500)):
        ga, ge, gn, gc = sg.bitso(v, L=L, Tmax=tmax)
        ta, te, tn, tc = mode.bitso(v, L=L, Tmax=tmax)
        assert np.array_equal(gn, tn) and np.array_equal(gc, tc)
        assert np.array_equal(ga.view(np.int64), ta.view(np.int64))
        assert np.array_equal(ge.view(np.int64), te.view(np.int64))
