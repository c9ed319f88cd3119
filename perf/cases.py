"""The decoder's performance cases: what a user has it do, through its public
entry points, from one call on a few lines to a batch of 30 000 codewords.

Kinds (the "kind" of a case):
  lines    SOGRAND_bitSO on channel LLR lines: host arrays (sogrand_b200.bitso)
           or device buffers (sg_bitso_device of the C ABI)
  decode   sogrand_b200.decode on device cubes (one CTA per codeword)
  batch    sogrand_b200.batch.Batch.decode (the persistent form)
  summary  sogrand_b200.decode_summary: a point of an Eb/N0 sweep
  host     sogrand_b200.decode on host buffers (copies in the call)
  train    forward and backward of sogrand_b200.diff.decode_bce
  gen      sogrand_b200.gen_llr on the device: source, encoder, channel
Eb/N0 spans 1 to 3 dB, the range of the sweep; "lo" < "hi" draws it per
codeword.  Tmax 0 means no cap.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import sogrand_b200 as sg
from sogrand_b200 import _lib, batch, diff

CUBE = 4096
# average guesses per codeword at Imax 30 against Eb/N0 (1 to 3 dB in steps of 0.5)
GUESSES = (7.60e6, 2.96e6, 1.96e6, 1.55e6, 1.31e6)
LARGEST = 30000 * GUESSES[2]


def listed():
    return [
        # one codeword's first 16 lines through the drop-in of SOGRAND_bitSO: launch and call overhead
        dict(name="lines_16_host", kind="lines", n=16, lo=2.0, hi=2.0, L=3, tmax=0, device=False),
        # a caller with its own product-code loop: a ragged number of lines resident on the device
        dict(name="lines_65537", kind="lines", n=65537, lo=2.0, hi=2.0, L=4, tmax=0, device=True),
        # one codeword: the latency of a single decode, with its soft output
        dict(name="decode_1", kind="decode", n=1, lo=2.0, hi=2.0, L=3, tmax=0, imax=30, lapp=True, math=0),
        # the reference's own 100-codeword run at 2 dB: less than one codeword per SM
        dict(name="decode_100", kind="decode", n=100, lo=2.0, hi=2.0, L=3, tmax=0, imax=30, lapp=False, math=0),
        # the top of the sweep: few iterations per codeword, many short lines
        dict(name="decode_9999_3dB", kind="decode", n=9999, lo=3.0, hi=3.0, L=3, tmax=0, imax=30, lapp=False, math=0),
        # the benchmark's workload (2 dB, persistent form) at 30 000 codewords
        dict(name="batch_30000_2dB", kind="batch", n=30000, lo=2.0, hi=2.0, L=3, tmax=0, imax=30, lapp=False, math=0),
        # a receiver whose channel varies per codeword, with soft output
        dict(name="batch_8191_mixed", kind="batch", n=8191, lo=1.0, hi=3.0, L=3, tmax=0, imax=30, lapp=True, math=0),
        # the results that equal the reference under a correctly rounded libm
        dict(name="batch_4096_exact", kind="batch", n=4096, lo=2.0, hi=2.0, L=3, tmax=0, imax=30, lapp=False, math=1),
        # the low end of the sweep under the abandonment cap: long decodes, failed lines
        dict(name="summary_2000_1dB", kind="summary", n=2000, lo=1.0, hi=1.0, L=3, tmax=1000, imax=30),
        # host buffers in, bits and statistics out: a receiver on the host
        dict(name="host_6000", kind="host", n=6000, lo=2.0, hi=2.0, L=3, tmax=0, imax=30),
        # a training step of the extrinsic weights
        dict(name="train_1024", kind="train", n=1024, lo=1.5, hi=1.5, L=3, imax=10),
        # simulated channel output for a sweep
        dict(name="gen_20000", kind="gen", n=20000, lo=2.0, hi=2.0),
    ]


def _guesses(lo, hi):
    """Expected guesses per codeword for Eb/N0 uniform in [lo, hi]."""
    tot = 0.0
    for k in range(8):
        x = min(max((lo + (hi - lo) * (k + 0.5) / 8 - 1.0) * 2.0, 0.0), 3.999)
        i = int(x)
        tot += math.exp(math.log(GUESSES[i]) * (i + 1 - x) + math.log(GUESSES[i + 1]) * (x - i))
    return tot / 8


def _loguniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["lines", "decode", "decode", "batch", "batch", "summary", "host", "train", "gen"])
    lo = round(rng.uniform(1.0, 3.0), 3)
    hi = round(rng.uniform(lo, 3.0), 3) if rng.random() < 0.3 else lo
    c = dict(kind=kind, lo=lo, hi=hi)
    if kind == "gen":
        return dict(c, n=_loguniform(rng, 1, 20000))
    if kind == "lines":
        dev = rng.random() < 0.6
        return dict(c, n=_loguniform(rng, 1, 65537 if dev else 4096), L=rng.choice([1, 2, 3, 4]),
                    tmax=rng.choice([0, 0, 100, 1000]), device=dev)
    c["L"] = rng.choice([3, 3, 2, 4])
    if kind == "train":
        return dict(c, n=_loguniform(rng, 1, 1024), L=3, imax=rng.choice([5, 10]), lo=max(lo, 1.25), hi=max(lo, 1.25))
    c.update(tmax=rng.choice([0, 0, 1000]), imax=rng.choice([10, 30, 30]))
    if kind == "host":
        return dict(c, n=_loguniform(rng, 1, 6000))
    if kind == "summary":
        return dict(c, n=_loguniform(rng, 1, min(9999, LARGEST / 4 / _guesses(lo, hi))))
    math_mode = int(rng.random() < 0.2)
    most = min(30000, LARGEST / (2 + 2 * math_mode) / _guesses(lo, hi))
    return dict(c, n=_loguniform(rng, 1, most), lapp=rng.random() < 0.4, math=math_mode)


def _cubes(case, seed, n):
    if case["lo"] == case["hi"]:
        return sg.gen_llr(seed, 0, n, ebn0_db=case["lo"], device="cuda")
    return sg.gen_llr(seed, 0, n, ebn0_range=(case["lo"], case["hi"]), device="cuda")


def _tmax(case):
    return case["tmax"] or sg.UINT64_MAX


def prepare(case, seed):
    st = dict(case=case, seed=seed)
    kind, n = case["kind"], case["n"]
    if kind == "gen":
        return st
    if kind == "lines":
        _, llr = _cubes(case, seed, (n + 255) // 256)
        lines = llr.reshape(-1, 16)[:n].contiguous()
        if case["device"]:
            st["llr"] = lines
            st["lapp"], st["le"] = torch.empty_like(lines), torch.empty_like(lines)
            st["ng"] = torch.empty(n, dtype=torch.int32, device="cuda")
            st["nc"] = torch.empty(n, dtype=torch.int32, device="cuda")
        else:
            st["llr"] = lines.cpu().numpy()
        return st
    info, llr = _cubes(case, seed, n)
    if kind == "train":
        st["cb"] = diff.code_bits_for(info, "cuda")
        st["llr"] = llr.requires_grad_(True)
        st["alpha"] = torch.full((3 * case["imax"],), 0.7, dtype=torch.float64, device="cuda", requires_grad=True)
        return st
    st["p"] = sg.params(L=case["L"], Imax=case["imax"], Tmax=_tmax(case))
    if kind == "host":
        host = torch.empty((n, CUBE), dtype=torch.float64, pin_memory=True)
        host.copy_(llr)
        st["keep"], st["llr"] = host, host.numpy()
        return st
    st["llr"], st["info"] = llr, info
    if kind == "batch":
        st["b"] = batch.Batch()
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "gen":
        info, llr = _cubes(case, st["seed"], case["n"])
        return {"info": info, "llr": llr}
    if kind == "lines":
        if not case["device"]:
            lapp, le, ng, nc = sg.bitso(st["llr"], L=case["L"], Tmax=_tmax(case))
            return {"lapp": lapp, "le": le, "ng": ng, "nc": nc}
        out = {k: st[k] for k in ("lapp", "le", "ng", "nc")}
        _lib.check(_lib.load().sg_bitso_device(
            st["llr"].data_ptr(), case["n"], case["L"], _tmax(case), ctypes.c_double(1.0 - 1e-5),
            *(out[k].data_ptr() for k in ("lapp", "le", "ng", "nc")), torch.cuda.current_stream().cuda_stream))
        return out
    if kind == "train":
        loss = diff.decode_bce(st["alpha"], st["llr"], st["cb"], imax=case["imax"], L=case["L"])
        ga, gl = torch.autograd.grad(loss, [st["alpha"], st["llr"]])
        return {"loss": loss.detach(), "grad_alpha": ga, "grad_llr": gl}
    if kind == "host":
        bits, stats, _ = sg.decode(st["llr"], st["p"])
        return {"bits": bits, "stats": stats.view(np.uint8)}
    if kind == "summary":
        s, bits = sg.decode_summary(st["llr"], st["p"], ref_info=st["info"], want_bits=True)
        return {"summary": s, "bits": bits}
    # the math mode holds for the process; a program that wants the exact one sets it around its calls
    if case["math"]:
        sg.set_math_mode(case["math"])
    try:
        if kind == "batch":
            bits, stats, lapp = st["b"].decode(st["llr"], st["p"], want_lapp=case["lapp"])
        else:
            bits, stats, lapp = sg.decode(st["llr"], st["p"], want_lapp=case["lapp"])
    finally:
        if case["math"]:
            sg.set_math_mode(0)
    out = {"bits": bits, "stats": stats}
    if lapp is not None:
        out["lapp"] = lapp
    return out


def work(case):
    """Bytes: inputs read and outputs written once.  Operations: per guess the
    path-metric addition, the exponential and the subtraction from the
    probability left, each counted as one; per generated LLR the two noise
    products, the addition and the division."""
    kind, n = case["kind"], case["n"]
    if kind == "gen":
        return {"bytes": n * (CUBE * 8.0 + 64), "flops": n * CUBE * 4.0}
    g = _guesses(case["lo"], case["hi"])
    if kind == "lines":
        return {"bytes": n * (3 * 128.0 + 8), "flops": n * 800 * 3.0}
    if kind == "train":
        frac = 0.6  # Imax 10 at low Eb/N0 cuts the longest decodes
        return {"bytes": n * (2 * CUBE * 8.0 + CUBE), "flops": n * 3 * g * frac * 3.0}
    return {"bytes": n * (CUBE * 8.0 * (2 if case.get("lapp") else 1) + 96), "flops": n * g * 3.0}


# ------------------------------------------------------------------ exact --
# The line decoder and the generator in plain numpy and torch, 64 bits.

def _code():
    """Syndrome byte of each of the 16 positions (CRC, Koopman form 0xeb)."""
    poly = [1, 1, 1, 0, 1, 0, 1, 1, 1]
    col = []
    for i in range(8):
        m = [0] * 24
        m[i] = 1
        for j in range(8):
            if m[j]:
                for k in range(9):
                    m[j + k] ^= poly[k]
        col.append(sum(m[8 + j] << j for j in range(8)))
    return col + [1 << j for j in range(8)]


def _orders(ic):
    """Patterns (bit r: sorted position r) in the order they are tested, each
    with whether it opens a logistic weight."""
    yield 0, False
    for wt in range(ic + 1, 16 * ic + 137):
        first = True
        t = 1 + 2 * (16.0 + ic)
        w = max(1, math.ceil((t - math.sqrt(t * t - 8 * wt)) / 2))
        while w <= 16 and wt - ic * w >= w * (w + 1) // 2:
            if w == 16:
                yield 0xffff, first
                break
            rest, top = wt - ic * w - w * (w + 1) // 2, 16 - w
            u = _fill([0] * w, 0, rest, top)
            while True:
                yield sum(1 << (i + x) for i, x in enumerate(u)), first
                first = False
                k = next((i for i in range(w - 1, 0, -1) if u[-1] - u[i] >= 2), 0)
                if u[-1] - u[0] < 2:
                    break
                u[k] += 1
                u = _fill(u, k, rest, top)
            w += 1


def _fill(u, k, rest, top):
    u = u[:k + 1] + [u[k]] * (len(u) - k - 1)
    more = rest - sum(u)
    q, r = divmod(more, top - u[k])
    for i in range(len(u) - q, len(u)):
        u[i] = top
    if len(u) > q:
        u[len(u) - q - 1] += r
    return u


class _Order:
    """The patterns of one IC as arrays, extended as far as they are needed."""

    def __init__(self, ic):
        self.it, self.m, self.f = _orders(ic), np.zeros(0, np.int64), np.zeros(0, bool)

    def get(self, a, b):
        while len(self.m) < b:
            got = [x for _, x in zip(range(1024), self.it)]
            if not got:
                break
            self.m = np.concatenate([self.m, np.array([x[0] for x in got], np.int64)])
            self.f = np.concatenate([self.f, np.array([x[1] for x in got], bool)])
        return self.m[a:b], self.f[a:b]


_ORDERS = {}


def _jac(x):
    return np.where(x > 50, x, np.where(x < -50, 0.0, np.log(1.0 + np.exp(np.minimum(x, 700.0)))))


def _exact_lines(v, L, tmax, thres=1.0 - 1e-5):
    """Soft output (L_APP) of each line of v [n, 16], and the guesses."""
    n = len(v)
    tmax = tmax or 1 << 60
    col = np.array(_code(), np.int64)
    hd = ~(v > 0)
    a = np.abs(v)
    perm = np.argsort(a, axis=1, kind="stable")
    asort = np.take_along_axis(a, perm, 1)
    jn = _jac(-a)
    pmhd = jn.sum(axis=1)
    delta = np.take_along_axis(_jac(a) - jn, perm, 1)
    hs = col[perm]
    s0 = np.bitwise_xor.reduce(np.where(hd, col, 0), axis=1)
    with np.errstate(all="ignore"):
        x = asort[:, 0] / ((asort[:, 7] - asort[:, 0]) / 7) - 1
    ic = np.where(np.isfinite(x), np.clip(np.sign(x) * np.floor(np.abs(x) + 0.5), 0, 64), 0).astype(int)
    bits = np.arange(16)
    P = np.ones(n)
    T = np.zeros(n, np.int64)
    found = [[] for _ in range(n)]
    pnl = np.zeros(n)
    for g in np.unique(ic):
        o = _ORDERS.setdefault(int(g), _Order(int(g)))
        live, at = np.nonzero(ic == g)[0], 0
        while len(live):
            m, f = o.get(at, at + (64 if at == 0 else 512))
            if not len(m):
                T[live] = at
                break
            cap = np.nonzero(f & (np.arange(at, at + len(m)) >= tmax) & (at + np.arange(len(m)) > 0))[0]
            last = len(cap) > 0
            if last:
                m = m[:cap[0]]
            mb = ((m[:, None] >> bits) & 1).astype(float)
            e = np.exp(-(pmhd[live][:, None] + delta[live] @ mb.T))
            left = np.subtract.accumulate(np.concatenate([P[live][:, None], e], axis=1), axis=1)[:, 1:]
            syn = np.repeat(s0[live][:, None], len(m), axis=1)
            for r in range(16):
                syn ^= hs[live, r][:, None] * (mb[:, r].astype(np.int64))[None, :]
            done = np.zeros(len(live), bool)
            for j, t in zip(*np.nonzero(syn == 0)):
                if done[j]:
                    continue
                i = live[j]
                flips = np.zeros(16, bool)
                flips[perm[i]] = mb[t] > 0
                found[i].append((e[j, t], hd[i] ^ flips))
                pnl[i] = left[j, t] * 2.0 ** -8
                pos = sum(q for q, _ in found[i])
                if (pos / (pos + pnl[i]) if pos + pnl[i] > 1e-40 else 1.0) > thres or len(found[i]) == L:
                    done[j], T[i] = True, at + t + 1
            if len(m):
                P[live] = left[:, -1]
            at += len(m)
            live = live[~done]
            if last:
                T[live] = at
                break
    out = v.copy()
    with np.errstate(over="ignore"):
        pp1 = 1.0 / (1.0 + np.exp(v))
    for i in range(n):
        if found[i]:
            e = np.array([q for q, _ in found[i]])
            c = np.array([b for _, b in found[i]], float)
            q = max(pnl[i], 1e-40)
            p1 = e @ c + q * np.clip(pp1[i], 1e-40, 1)
            p0 = e @ (1 - c) + q * np.clip(1 - pp1[i], 1e-40, 1)
            out[i] = np.log(np.maximum(p0, 1e-40)) - np.log(np.maximum(p1, 1e-40))
    return out, T


def _mix(z):
    def shr(x, k):
        return (x >> k) & ((1 << (64 - k)) - 1)

    z = (z ^ shr(z, 30)) * -0x40a7b892e31b1a47
    z = (z ^ shr(z, 27)) * -0x6b2fb644ecceee15
    return z ^ shr(z, 31)


def _rand53(seed, stream, ctr):
    """The top 53 bits of random number (seed, stream, ctr), as float64."""
    dev = ctr.device
    wrap = lambda x: (x + (1 << 63)) % (1 << 64) - (1 << 63)  # noqa: E731
    key = _mix(torch.tensor(wrap(seed + 0x9e3779b97f4a7c15 * (stream + 1)), device=dev))
    r = _mix(key ^ (ctr * wrap(0xd1b54a32d192ed03) + wrap(0x8cb92ba72f3d8dd7)))
    return ((r >> 11) & ((1 << 53) - 1)).double()


def _exact_gen(case, seed):
    n = case["n"]
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    info = sg.gen_info(seed, 0, n)  # bytes: only the noise is computed here
    code = torch.from_numpy(sg.encode(info)).to(dev).double().reshape(-1)
    ctr = torch.arange(n * CUBE, dtype=torch.int64, device=dev)
    z = torch.zeros(n * CUBE, dtype=torch.float64, device=dev)
    todo = ctr
    for a in range(64):
        u = _rand53(seed, 1 + 2 * a, todo) * 2.0 ** -52 - 1
        v = _rand53(seed, 2 + 2 * a, todo) * 2.0 ** -52 - 1
        s = u * u + v * v
        ok = (s > 0) & (s < 1)
        z[todo[ok]] = (u * torch.sqrt(-2 * torch.log(s) / s))[ok]
        todo = todo[~ok]
        if not len(todo):
            break
    if case["lo"] == case["hi"]:
        eb = torch.full((n,), case["lo"], dtype=torch.float64, device=dev)
    else:
        uu = _rand53(seed, 7, torch.arange(n, dtype=torch.int64, device=dev)) * 2.0 ** -53
        eb = case["lo"] + (case["hi"] - case["lo"]) * uu
    var = 10 ** (-(eb + 10 * math.log10(0.25)) / 10)
    var = var.repeat_interleave(CUBE)
    return 2 * ((1 - 2 * code) + torch.sqrt(var) * z) / var


def exact(case, seed):
    kind, n = case["kind"], case["n"]
    if kind == "gen":
        return {"info": None, "llr": _exact_gen(case, seed).reshape(n, CUBE)}
    if kind == "lines" and n <= 8192:
        _, llr = _cubes(case, seed, (n + 255) // 256)
        v = llr.reshape(-1, 16)[:n].cpu().numpy()
        app, _ = _exact_lines(v, case["L"], case["tmax"])
        return {"lapp": app, "le": app - v, "ng": None, "nc": None}
    # whole decodes have none: a converged line's probability left is 1 less terms that sum to 1,
    # so its soft output is the rounding of that sum; and a gradient takes thousands of line decodes
    # per codeword, minutes in numpy
    return None
