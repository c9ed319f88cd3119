"""The device generator against the host generator, bit for bit: odd batch sizes and ranges, per-codeword
Eb/N0, and noise deviations whose square leaves the range of the remainder-corrected quotient."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ebn0", [-1500.0, -1210.0, -1190.0, -40.0, 0.0, 2.0, 60.0, 1190.0, 1210.0, 1500.0])
def test_device_equals_host_over_deviations(cuda, sg, ebn0):
    hi, hl = sg.gen_llr(99, 5, 2, ebn0_db=ebn0)
    di, dl = sg.gen_llr(99, 5, 2, ebn0_db=ebn0, device="cuda")
    assert np.array_equal(hi, di.cpu().numpy())
    assert np.array_equal(hl.view(np.int64), dl.cpu().numpy().view(np.int64))


@pytest.mark.parametrize("n,cw0,seed", [(1, 0, 0), (7, 2**40 + 3, 2**63 + 11), (33, 1000, 5)])
def test_device_equals_host_over_ranges(cuda, sg, n, cw0, seed):
    hi, hl = sg.gen_llr(seed, cw0, n, ebn0_range=(0.5, 3.5))
    di, dl = sg.gen_llr(seed, cw0, n, ebn0_range=(0.5, 3.5), device="cuda")
    assert np.array_equal(hi, di.cpu().numpy())
    assert np.array_equal(hl.view(np.int64), dl.cpu().numpy().view(np.int64))
