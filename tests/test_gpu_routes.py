"""Dispatch lines of the line and backward kernels: results must not depend on how many lines or
codewords a call holds.  Lines: up to 256 on host buffers, one warp per line, one line per CTA below
two CTAs per SM, a persistent grid above the resident warps (4 736 on 148 SMs).  Backward: a call's
last 2 048 codewords are taken in the order of falling phase counts."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(params=[0, 1])
def mode(request, sg):
    sg.set_math_mode(request.param)
    yield request.param
    sg.set_math_mode(0)


def device_lines(torch, v, L, tmax):
    from sogrand_b200 import _lib

    n = len(v)
    d = torch.from_numpy(v).cuda()
    la, le = torch.empty_like(d), torch.empty_like(d)
    ng, nc = (torch.empty(n, dtype=torch.int32, device="cuda") for _ in range(2))
    _lib.check(_lib.load().sg_bitso_device(d.data_ptr(), n, L, C.c_uint64(tmax), C.c_double(1.0 - 1e-5),
                                           la.data_ptr(), le.data_ptr(), ng.data_ptr(), nc.data_ptr(),
                                           torch.cuda.current_stream().cuda_stream))
    return [t.cpu().numpy() for t in (la, le, ng, nc)]


def same(got, want):
    ok = got[2] >= 0  # a non-finite line: N_guess -1, NaN out
    assert np.array_equal(got[2], want[2]) and np.array_equal(got[3], want[3])
    for g, w in zip(got[:2], want[:2]):
        assert np.array_equal(g[ok].view(np.int64), w[ok].view(np.int64))
        assert np.isnan(g[~ok]).all()


def test_line_routes(cuda, sg, mode):
    """Every call against the same lines in calls of 200, and those against the restatement's by
    the tests of the guess loop."""
    torch = cuda
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n_max = 20001
    _, llr = sg.gen_llr(77, 0, n_max // 256 + 1, ebn0_range=(0.5, 3.5))
    v = np.ascontiguousarray(llr.reshape(-1, 16)[:n_max])
    v[[5, 290, 4730, 20000], [0, 3, 15, 7]] = [np.inf, np.nan, -np.inf, np.nan]
    for L, tmax in ((3, sg.UINT64_MAX), (8, 700)):
        parts = [sg.bitso(v[i : i + 200], L=L, Tmax=tmax) for i in range(0, n_max, 200)]
        want = [np.concatenate(c) for c in zip(*parts)]
        for n in (1, 15, 17, 2 * sms - 1, 2 * sms, 2 * sms + 1, 32 * sms, 32 * sms + 1, n_max):
            same(device_lines(torch, v[:n], L, tmax), [w[:n] for w in want])
        for n in (255, 256, 257):
            same(sg.bitso(v[:n], L=L, Tmax=tmax), [w[:n] for w in want])


@pytest.mark.parametrize("n,chunk,loss_mode", [(150, 50, 0), (150, 50, 1), (2047, 90, 1), (2048, 700, 0),
                                               (2049, 700, 0), (2200, 700, 0)])
def test_backward_order(cuda, sg, n, chunk, loss_mode):
    """A codeword's loss and gradients in one call against smaller calls.  The warps of a CTA add
    into a codeword's sums in an order of their own, so the bound is that of the adjoint's own tests, 1e-9 of the largest entry;
    the losses are sums of 4 096 positive terms in another grouping: 1e-12."""
    torch = cuda
    from sogrand_b200 import diff

    info, llr = sg.gen_llr(31, 0, n, ebn0_range=(1.5, 3.0), device="cuda")
    llr[3, 9] = float("nan")
    cb = diff.code_bits_for(info, "cuda")
    p = sg.params(Imax=3)
    _, st, _, ck = diff.forward_raw(llr, p)
    whole = diff.backward_raw(llr, cb, p, st, ck, want_llr=True, loss_mode=loss_mode)
    part = [torch.cat(t) for t in zip(*(diff.backward_raw(llr[a : a + chunk], cb[a : a + chunk], p, st[a : a + chunk],
                                                          ck[a : a + chunk], want_llr=True, loss_mode=loss_mode)
                                        for a in range(0, n, chunk)))]
    for w, q, tol in zip(whole, part, (1e-12, 1e-9, 1e-9)):
        w, q = w.cpu().numpy(), q.cpu().numpy()
        assert np.array_equal(np.isnan(w), np.isnan(q))
        d, ref = np.abs(w - q), np.abs(q)
        if w.ndim == 2:
            d, ref = d.max(axis=1), np.maximum(1.0, ref.max(axis=1))
        ok = ~np.isnan(d)
        assert ok.sum() >= n - 1 and (d[ok] <= tol * ref[ok]).all()


@pytest.mark.parametrize("n", [1, 8, 37, 74, 148, 259, 260, 700])
@pytest.mark.parametrize("want_bits", [False, True])
def test_summary_totals(cuda, sg, mode, n, want_bits):
    """Totals that the decode kernels keep, for every cluster size and the plain form, against those
    of the per-codeword outputs: whole numbers and multiples of 0.5, equal."""
    torch = cuda
    from sogrand_b200 import _lib

    info, llr = sg.gen_llr(500 + n, 0, n, ebn0_range=(0.5, 2.5), device="cuda")
    if n > 5:
        llr[4, 100] = float("inf")
    p = sg.params(Imax=3)
    bits, raw, _ = sg.decode(llr, p)
    st = sg.stats_from_device(raw)
    wrong = np.unpackbits((bits ^ info).cpu().numpy(), axis=1).sum(axis=1)
    want = dict(blocks=n, converged=(st["converged"] == 1).sum(), nonfinite=(st["converged"] == -1).sum(),
                total_ng=st["ng"].sum(), total_ng_p=st["ng_p"].sum(), bits_compared=512 * n, bit_errors=wrong.sum(),
                block_errors=(wrong > 0).sum(), total_iterations=st["iterations"].sum(), timeouts=0, device_error=0)
    got, b = sg.decode_summary(llr, p, ref_info=info, want_bits=want_bits)
    assert {k: got[k] for k in want} == want
    if want_bits:
        assert torch.equal(b, bits)
    summ = torch.zeros(sg.SUMMARY_DTYPE.itemsize, dtype=torch.uint8, device="cuda")
    _lib.check(_lib.load().sg_decode_summary_device_noalloc(
        llr.data_ptr(), n, C.byref(p), None, b.data_ptr() if want_bits else None, summ.data_ptr(),
        torch.cuda.current_stream().cuda_stream))
    rec = np.frombuffer(summ.cpu().numpy().tobytes(), dtype=sg.SUMMARY_DTYPE)[0]
    want.update(bits_compared=0, bit_errors=0, block_errors=0)
    assert {k: rec[k].item() for k in want} == want
