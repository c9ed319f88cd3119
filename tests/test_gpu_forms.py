"""The one-CTA and the batched kernel on small batches, which the default variants hand to clusters:
against the reference fixtures in both math modes, soft output included, and the batched kernel's
admission of codewords, fixed first ones and those of its queue.  Exact."""
import hashlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SETS = ["cfg1_2dB_100", "snr_1.0dB", "snr_1.5dB", "snr_2.5dB", "snr_3.0dB", "mixed_1to3dB", "tmax1000_2dB",
        "tmax1000_1.5dB"]


@pytest.fixture(params=["w16-gmem", "p32x3"])
def decode(request, cuda, sg):
    """decode(device LLRs, params) -> bits, stats, L_APP on the host, by the kernel of that name."""
    from sogrand_b200 import autotune, batch

    b = batch.Batch()
    plain = request.param[0] == "w"
    mod = autotune if plain else batch
    before = mod.get_variant()
    mod.set_variant(request.param)

    def run(llr, p):
        bits, raw, lapp = (sg.decode if plain else b.decode)(llr, p, want_lapp=True)
        cuda.cuda.synchronize()
        if not plain:
            b.check()
        return bits.cpu().numpy(), sg.stats_from_device(raw), lapp.cpu().numpy()

    yield run
    mod.set_variant(before)
    b.close()


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("name", SETS)
def test_fixture_sets(cuda, sg, golden, decode, name, mode):
    e = golden["sets"][name]
    snr = {"ebn0_range": tuple(e["ebn0_db"])} if isinstance(e["ebn0_db"], list) else {"ebn0_db": e["ebn0_db"]}
    _, llr = sg.gen_llr(e["seed"], 0, e["n_cw"], **snr)
    assert hashlib.sha256(llr.tobytes()).hexdigest() == e["llr_sha256"]
    want = e["ref_cr" if mode else "twin"]
    sg.set_math_mode(mode)
    try:
        bits, st, lapp = decode(cuda.from_numpy(llr).cuda(), sg.params(Tmax=e["Tmax"]))
    finally:
        sg.set_math_mode(0)
    for i in range(e["n_cw"]):
        if mode and want["undefined_lines"][i]:  # the reference reads an uninitialised list size
            continue
        assert bits[i].tobytes().hex() == want["bits"][i], i
        assert (st["iterations"][i], st["ng"][i], st["ng_p"][i], st["converged"][i]) == \
            (want["iterations"][i], want["ng"][i], want["ng_p"][i], want["converged"][i]), i
        assert hashlib.sha256(lapp[i].tobytes()).hexdigest() == want["lapp_sha256"][i], i


@pytest.mark.parametrize("n,mode", [(5, 0), (5, 1), (445, 0), (500, 1)])
def test_admission_and_nonfinite(cuda, sg, oracle_paths, decode, n, mode):
    """Non-finite codewords among the first of the slots (3 per SM) and among those the queue hands
    out, the last one included; every sixteenth other codeword against the restatement."""
    from oracle_api import Oracle

    first = 3 * cuda.cuda.get_device_properties(0).multi_processor_count
    _, llr = sg.gen_llr(5, 0, n, ebn0_range=(1.5, 3.0))
    bad = sorted({i for i in (0, 3, first // 3 + 1, first - 1, first, first + 9, n - 1) if i < n})
    llr[bad, 7] = np.nan
    sg.set_math_mode(mode)
    try:
        bits, st, lapp = decode(cuda.from_numpy(llr).cuda(), sg.params(Imax=2))
    finally:
        sg.set_math_mode(0)
    assert np.array_equal(np.flatnonzero(st["converged"] == -1), bad)
    assert not bits[bad].any() and not st["phases"][bad].any()
    pick = [i for i in range(1, n, 16) if i not in bad]
    wb, ws, wl = Oracle(oracle_paths["twin_cr" if mode else "twin"]).decode(llr[pick], Imax=2)
    assert np.array_equal(bits[pick], wb)
    assert [(s["iterations"], s["ng"], s["ng_p"], s["converged"], s["phases"]) for s in st[pick]] == ws
    assert np.array_equal(lapp[pick].view(np.int64), wl.view(np.int64))
