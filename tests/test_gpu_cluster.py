"""Small batches, which the default configurations decode with a cluster of CTAs per codeword,
against the one-CTA form (w16-gmem, itself pinned to the reference by the parity tests): bits,
statistics, L_APP and checkpoints, on both sides of every change of the cluster size.  Exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(params=[0, 1])
def mode(request, sg):
    sg.set_math_mode(request.param)
    yield request.param
    sg.set_math_mode(0)


def outputs(sg, llr, p, batch=None):
    bits, raw, lapp = (batch.decode if batch else sg.decode)(llr, p, want_lapp=True)
    st = sg.stats_from_device(raw)
    ok = st["converged"] >= 0
    return bits.cpu().numpy(), st, lapp.cpu().numpy()[ok].view(np.int64)


@pytest.mark.parametrize("n", [1, 2, 8, 9, 16, 17, 18, 33, 36, 37, 74, 75, 148, 259, 260])
def test_cluster_sizes(cuda, sg, mode, n):
    from sogrand_b200 import autotune
    from sogrand_b200.batch import Batch

    torch = cuda
    _, llr = sg.gen_llr(1000 + n, 0, n, ebn0_range=(1.0, 3.0), device="cuda")
    if n > 4:
        llr[3, 77] = float("nan")
    p = sg.params(Imax=4, Tmax=1000 if n % 2 else sg.UINT64_MAX)
    got, bat = outputs(sg, llr, p), outputs(sg, llr, p, Batch())
    before = autotune.get_variant()
    try:
        autotune.set_variant("w16-gmem")
        want = outputs(sg, llr, p)
    finally:
        autotune.set_variant(before)
    torch.cuda.synchronize()
    for g in (got, bat):
        assert all(np.array_equal(a, b) for a, b in zip(g, want))


def test_cluster_checkpoints_and_last_phase(cuda, sg):
    from sogrand_b200 import autotune, diff

    for imax in (1, 3):
        _, llr = sg.gen_llr(4, 0, 5, ebn0_db=1.0, device="cuda")
        p = sg.params(Imax=imax)
        bits, raw, lapp, ckpt = diff.forward_raw(llr, p)
        before = autotune.get_variant()
        try:
            autotune.set_variant("w16-gmem")
            wbits, wraw, wlapp, wckpt = diff.forward_raw(llr, p)
        finally:
            autotune.set_variant(before)
        st = sg.stats_from_device(raw)
        assert (st == sg.stats_from_device(wraw)).all() and (bits == wbits).all()
        assert np.array_equal(lapp.cpu().numpy().view(np.int64), wlapp.cpu().numpy().view(np.int64))
        for i, ph in enumerate(st["phases"]):
            assert np.array_equal(ckpt[i, :ph].cpu().numpy().view(np.int64),
                                  wckpt[i, :ph].cpu().numpy().view(np.int64))
