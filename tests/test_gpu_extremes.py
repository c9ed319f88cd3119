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


@pytest.mark.parametrize("imax", [2, 3])
@pytest.mark.parametrize("form", ["default", "w16-gmem", "w8-l2-g2", "p32x3"])
def test_infinite_and_nan_lines(cuda, sg, mode, form, imax):
    """Finite LLRs near the largest number under weights of 2 and 0: extrinsic values overflow and the
    phases of weight 0 decode lines that hold NaN (0 times infinity), among ordinary ones."""
    torch = cuda
    from sogrand_b200 import autotune, batch

    _, llr = sg.gen_llr(9, 0, 3, ebn0_db=1.0)
    llr[0, [5, 777, 4000]] = [1.6e308, -1.7e308, 1.5e308]
    llr[1] *= 2e306
    llr[2, 100] = 1.7e308
    alpha = [0.7, 2.0, 2.0, 0.0, 0.5, 0.0] + [0.7] * 144
    wb, ws, wl = mode.decode(llr, Imax=imax, alpha=alpha)
    p, d = sg.params(Imax=imax, alpha=alpha), torch.from_numpy(llr).cuda()
    before = autotune.get_variant(), batch.get_variant()
    b = batch.Batch()
    try:
        if form[0] == "p":
            batch.set_variant(form)
        elif form[0] == "w":
            autotune.set_variant(form)
        bits, raw, lapp = (b.decode if form[0] == "p" else sg.decode)(d, p, want_lapp=True)
        torch.cuda.synchronize()
    finally:
        autotune.set_variant(before[0])
        batch.set_variant(before[1])
        b.close()
    st = sg.stats_from_device(raw)
    assert np.array_equal(bits.cpu().numpy(), wb)
    assert [(s["iterations"], s["ng"], s["ng_p"], s["converged"], s["phases"]) for s in st] == ws
    assert np.array_equal(lapp.cpu().numpy(), wl, equal_nan=True)
