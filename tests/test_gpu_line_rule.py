"""The rule that takes line calls of more than 16 lines per SM to the resident grid: results on both
sides of it, and no step down in time above it."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(params=[0, 1])
def mode(request, sg):
    sg.set_math_mode(request.param)
    yield request.param
    sg.set_math_mode(0)


def _call(torch, sg, v):
    from sogrand_b200 import _lib

    n, lib = len(v), _lib.load()
    la, le = torch.empty_like(v), torch.empty_like(v)
    ng, nc = (torch.empty(n, dtype=torch.int32, device="cuda") for _ in range(2))

    def run():
        _lib.check(lib.sg_bitso_device(v.data_ptr(), n, 3, C.c_uint64(sg.UINT64_MAX), C.c_double(1.0 - 1e-5),
                                       la.data_ptr(), le.data_ptr(), ng.data_ptr(), nc.data_ptr(),
                                       torch.cuda.current_stream().cuda_stream))

    return run, (la, le, ng, nc)


def test_results_on_both_sides(cuda, sg, mode):
    torch = cuda
    n = 16 * torch.cuda.get_device_properties(0).multi_processor_count
    _, llr = sg.gen_llr(7, 0, n // 256 + 2, ebn0_range=(0.5, 3.5), device="cuda")
    v = llr.reshape(-1, 16)
    want = [torch.cat(t) for t in zip(*[(lambda r, o: (r(), o)[1])(*_call(torch, sg, v[i : i + 128]))
                                        for i in range(0, n + 128, 128)])]
    for m in (n - 1, n, n + 1, n + 100):
        run, out = _call(torch, sg, v[:m])
        run()
        assert all(np.array_equal(o.cpu().numpy(), w[:m].cpu().numpy()) for o, w in zip(out, want))


def test_time_does_not_step_down(cuda, sg, mode):
    """Twice the rule's line, where one line per warp takes a fifth longer than the resident grid."""
    torch = cuda
    n = 32 * torch.cuda.get_device_properties(0).multi_processor_count
    _, llr = sg.gen_llr(3, 0, n // 256 + 2, ebn0_db=2.0, device="cuda")
    t = []
    for m in (n, n + 1):
        run, _ = _call(torch, sg, llr.reshape(-1, 16)[:m])
        best = 1e9
        for _ in range(5):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            for _ in range(20):
                run()
            b.record()
            torch.cuda.synchronize()
            best = min(best, a.elapsed_time(b))
        t.append(best)
    assert t[0] <= 1.08 * t[1], t
