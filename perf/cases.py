"""The measured workloads: SO(3) Fourier transforms through the package's public entry points.

``listed()`` names the fixed cases, ``draw(rng)`` gives further ones of the same ranges,
``prepare`` makes what a caller holds before the call, ``run`` is one pass, ``work`` the bytes and
operations that the result needs, and ``exact`` the same result in 64 bits from torch and numpy
alone.

Kinds of case (``op``):

* ``idsoft`` / ``dsoft``: one transform of device-resident data (FourierTransforms), B from a few
  (latency, launches) through 128 (the benchmark's size) to 256; any integer bandwidth is a legal
  size, so ones with large prime factors are among them.
* ``batch_idsoft`` / ``batch_dsoft``: a BatchPlan over several bandwidths, FP64 or split precision.
* ``layers_dft2`` / ``layers_idft2``: the layer-wise 2D DFT of a grid, in place, any dimensions.
* ``host_dsoft`` / ``host_idsoft``: the drop-in call on the caller's own host arrays.
"""
import functools
import math

import numpy as np
import torch

from pfsoftlib_b200 import BatchPlan, DSOFTFourierCoefficients, FourierTransforms, grid3D


def listed():
    return [
        # one small synthesis, as in an example or an inner loop: launches and latency
        {"name": "idsoft-b8", "op": "idsoft", "B": 8},
        # the analysis of a coarse grid (the smallest size that is compared with the CPU library)
        {"name": "dsoft-b16", "op": "dsoft", "B": 16},
        # an ordinary synthesis
        {"name": "idsoft-b64", "op": "idsoft", "B": 64},
        # a round number that is no power of two: FFT length 200 = 8 * 5 * 5
        {"name": "dsoft-b100", "op": "dsoft", "B": 100},
        # the benchmark's size, each direction
        {"name": "idsoft-b128", "op": "idsoft", "B": 128},
        {"name": "dsoft-b128", "op": "dsoft", "B": 128},
        # a bandwidth with a large prime factor, as a service that takes every integer meets
        {"name": "idsoft-b137", "op": "idsoft", "B": 137},
        # the largest single transform of the benchmark
        {"name": "dsoft-b256", "op": "dsoft", "B": 256},
        # many transforms of uneven bandwidths in one call (the batched workload, FP64)
        {"name": "batch-idsoft-mixed", "op": "batch_idsoft", "bandwidths": "32x9 48x8 64x11 96x10 128x10", "split": False},
        # large transforms in one call with the split-precision option
        {"name": "batch-dsoft-split-b256", "op": "batch_dsoft", "bandwidths": "256x4", "split": True},
        # the layer-wise 2D DFT alone, on a grid that is no cube
        {"name": "layers-dft2-160x192x96", "op": "layers_dft2", "rows": 160, "cols": 192, "lays": 96},
        # the drop-in call: numpy containers in, numpy containers out
        {"name": "host-dsoft-b64", "op": "host_dsoft", "B": 64},
    ]


def _log_int(rng, lo, hi):
    return min(hi, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))


def draw(rng):
    fixed = [{k: v for k, v in c.items() if k != "name"} for c in listed()]
    case = _draw(rng)
    while case in fixed:
        case = _draw(rng)
    return case


def _draw(rng):
    kind = rng.choice(["single", "single", "single", "single", "batch", "batch", "layers", "host"])
    if kind == "single":
        # half of the larger sizes any integer, half multiples of 4 (as callers who may choose do)
        B = _log_int(rng, 6, 256)
        if B >= 24 and rng.random() < 0.5:
            B = B // 4 * 4
        return {"op": rng.choice(["idsoft", "dsoft"]), "B": B}
    if kind == "batch":
        split = rng.random() < 0.4
        groups = {}
        for _ in range(rng.randint(1, 3)):
            B = _log_int(rng, 16, 192 if split else 128)
            if rng.random() < 0.6:
                B = max(16, B // 8 * 8)
            groups[B] = rng.randint(1, 5)
        text = " ".join("%dx%d" % (B, groups[B]) for B in sorted(groups))
        return {"op": rng.choice(["batch_idsoft", "batch_dsoft"]), "bandwidths": text, "split": split}
    if kind == "layers":
        return {"op": rng.choice(["layers_dft2", "layers_idft2"]), "rows": _log_int(rng, 16, 400),
                "cols": _log_int(rng, 16, 400), "lays": _log_int(rng, 8, 256)}
    return {"op": rng.choice(["host_idsoft", "host_dsoft"]), "B": _log_int(rng, 8, 72)}


def _bandwidths(case):
    if "bandwidths" not in case:
        return [case["B"]]
    out = []
    for part in case["bandwidths"].split():
        B, n = part.split("x")
        out += [int(B)] * int(n)
    return out


def _coef_len(B):
    return B * (4 * B * B - 1) // 3


def _coeffs(B, seed):
    """A spectrum that decays with the degree, |f^l| about (1 + l)^-2."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    f = torch.randn(_coef_len(B), dtype=torch.complex128, device="cuda", generator=g)
    degree = torch.repeat_interleave(torch.arange(B, device="cuda"), (2 * torch.arange(B, device="cuda") + 1) ** 2)
    return f * (1.0 + degree.double()).pow_(-2)


def _samples(shape, seed):
    """Samples with noise in every bin (not band-limited)."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return torch.randn(shape, dtype=torch.complex128, device="cuda", generator=g)


def _inputs(case, seed):
    op = case["op"]
    if op.startswith("layers"):
        return [_samples((case["lays"], case["cols"], case["rows"]), seed)]
    out = []
    for i, B in enumerate(_bandwidths(case)):
        s = seed * 1000 + i
        out.append(_coeffs(B, s) if op.endswith("idsoft") else _samples((2 * B,) * 3, s))
    return out


def prepare(case, seed):
    op = case["op"]
    x = _inputs(case, seed)
    if op.startswith("layers"):
        return {"op": op, "grid": grid3D.wrap(x[0]), "scale": 1.0 / math.sqrt(case["rows"] * case["cols"])}
    if op.startswith("host"):
        B = case["B"]
        if op == "host_idsoft":
            return {"op": op, "grid": grid3D(2 * B), "fc": DSOFTFourierCoefficients.wrap(x[0].cpu().numpy(), B)}
        return {"op": op, "grid": grid3D.wrap(x[0].cpu().numpy()), "fc": DSOFTFourierCoefficients(B)}
    bws = _bandwidths(case)
    if op.startswith("batch"):
        plan = BatchPlan(bws, split=case["split"])
        if op == "batch_idsoft":
            y = [torch.zeros((2 * B,) * 3, dtype=torch.complex128, device="cuda") for B in bws]
        else:
            y = [torch.zeros(_coef_len(B), dtype=torch.complex128, device="cuda") for B in bws]
        return {"op": op, "plan": plan, "x": x, "y": y}
    B = bws[0]
    if op == "idsoft":
        return {"op": op, "grid": grid3D(2 * B, device="cuda"), "fc": DSOFTFourierCoefficients.wrap(x[0], B)}
    return {"op": op, "grid": grid3D.wrap(x[0]), "fc": DSOFTFourierCoefficients(B, device="cuda")}


def run(state):
    op = state["op"]
    if op in ("idsoft", "host_idsoft"):
        FourierTransforms.IDSOFT(state["fc"], state["grid"])
        return state["grid"].mem
    if op in ("dsoft", "host_dsoft"):
        FourierTransforms.DSOFT(state["grid"], state["fc"])
        return state["fc"].mem
    if op == "batch_idsoft":
        state["plan"].idsoft(state["x"], state["y"])
        return state["y"]
    if op == "batch_dsoft":
        state["plan"].dsoft(state["x"], state["y"])
        return state["y"]
    if op == "layers_dft2":
        state["grid"].layer_wise_DFT2(state["scale"])
    else:
        state["grid"].layer_wise_IDFT2(state["scale"])
    return state["grid"].mem


def work(case):
    if case["op"].startswith("layers"):
        n = case["rows"] * case["cols"] * case["lays"]
        return {"bytes": 32.0 * n, "flops": 5.0 * n * math.log2(case["rows"] * case["cols"])}
    b = f = 0.0
    for B in _bandwidths(case):
        n = (2.0 * B) ** 3
        b += 16.0 * (n + _coef_len(B))
        # two DFTs of length 2B per sample, and the sums over beta: 2 * 2 * 2B for each coefficient
        f += 10.0 * n * math.log2(2 * B) + 8.0 * B * _coef_len(B)
    return {"bytes": b, "flops": f}


# ---- the same results in 64 bits, without the package's code ---------------------------------------


@functools.lru_cache(maxsize=2)
def _delta(B):
    """p[l][n][m] for 0 <= n, m <= l: the Wigner d-functions at pi/2 with a positive seed and the factor
    ((2l+1)/2)^(1/4), from the three-term recurrence in l (extended precision), one array per degree."""
    ld = np.longdouble
    n, m = np.meshgrid(np.arange(B), np.arange(B), indexing="ij")
    J, j = np.maximum(n, m), np.minimum(n, m)
    lg = np.zeros(2 * B + 1, dtype=ld)
    lg[1:] = np.cumsum(np.log2(np.arange(1, 2 * B + 1, dtype=ld)))
    seed = np.exp2((lg[2 * J] - lg[J - j] - lg[J + j]) / 2 - J)
    prev, cur = np.zeros((B, B), ld), np.zeros((B, B), ld)
    out = []
    for l in range(B):
        cur = np.where(J == l, seed, cur)   # pairs that start at this degree
        out.append((cur[: l + 1, : l + 1] * ((2 * l + 1) / ld(2)) ** ld(0.25)).astype(np.float64))
        k = l + 1
        live = J <= l
        a1 = np.where(live, (ld(k) * k - ld(1) * n * n) * (ld(k) * k - ld(1) * m * m), 1)
        step = -(2 * l + 1) * np.asarray(n * m, ld) / ld(l) if l else np.zeros((B, B), ld)
        nxt = step * cur
        if l:
            a2 = np.where(live, (ld(l) * l - ld(1) * n * n) * (ld(l) * l - ld(1) * m * m), 0)
            nxt -= (ld(k) / l) * np.sqrt(a2) * prev
        nxt = np.where(live, nxt / np.sqrt(a1), 0)
        prev, cur = np.where(live, cur, 0), nxt
    return out


def _fourier_rows(l, p):
    """Row l of every class as a Fourier series in beta: for the orders m of the columns 0 .. 2l (m >= 0, then
    the negative ones), the factor for each n <= l; the product of two of them is the coefficient."""
    n, m = np.arange(l + 1)[:, None], np.arange(l + 1)[None, :]
    d = torch.from_numpy(p * np.where((n > m) & ((n - m) % 2 == 1), -1.0, 1.0)).cuda()
    return torch.cat([d, d[:, 1:].flip(1)], dim=1)


@functools.lru_cache(maxsize=2)
def _order_signs(B):
    """For the bins (m2, m1) of a 2B x 2B layer: orders, parity of m1 + m2, and the signs of the classes."""
    o = np.arange(2 * B)
    o = np.where(o < B, o, o - 2 * B)
    m2, m1 = o[:, None], o[None, :]
    M, Mp = np.maximum(abs(m1), abs(m2)), np.minimum(abs(m1), abs(m2))
    odd = (M - Mp) % 2 == 1
    x = np.where(abs(m1) == M, m1 < 0, m2 > 0)
    rev = (m1 < 0) != (m2 < 0)
    base = np.where(x & odd, -1.0, 1.0)
    # the series' own sign, of period 4 in M - M': that of i^(M - M') for cosines, of -i^(M - M' + 1) for sines
    base = base * np.where(((M - Mp) % 4 == 1) | ((M - Mp) % 4 == 2), -1.0, 1.0)
    return m1, m2, M, odd, rev, base


def _trig(B, s):
    """cos(n beta_k), sin(n beta_k), n < B, k < 2B, the argument reduced in integers."""
    n, k = np.arange(B)[:, None], np.arange(2 * B)[None, :]
    arg = ((n * (2 * k + 1)) % (8 * B)).astype(np.longdouble) * (np.longdouble(2) * np.arccos(np.longdouble(0)) / (4 * B))
    return (torch.from_numpy(s(arg).astype(np.float64)).cuda())


def _weights(B):
    k, q = np.arange(2 * B, dtype=np.longdouble)[:, None], np.arange(B, dtype=np.longdouble)[None, :]
    pi = np.longdouble(2) * np.arccos(np.longdouble(0))
    s = (np.sin((2 * k + 1) * (2 * q + 1) * pi / (4 * B)) / (2 * q + 1)).sum(1)
    return torch.from_numpy((2 / np.longdouble(B) * np.sin((2 * k[:, 0] + 1) * pi / (4 * B)) * s).astype(np.float64)).cuda()


def _cols(B, l):
    """Bins of the orders 0 .. l, -l .. -1 in a layer of 2B."""
    return torch.tensor(list(range(l + 1)) + list(range(2 * B - l, 2 * B)), device="cuda")


def _tables(B):
    m1, m2, M, odd, rev, base = _order_signs(B)
    n = np.arange(B)[:, None, None]
    # reversal of beta: cos(n (pi - beta)) = (-1)^n cos, sin(n (pi - beta)) = -(-1)^n sin
    turn = np.where(rev[None], np.where((n + odd[None]) % 2 == 1, -1.0, 1.0), 1.0)
    sign = torch.from_numpy(turn * base[None] * np.where(n == 0, 1.0, 2.0)).cuda()
    par = torch.from_numpy(np.where(rev & (M % 2 == 1), -1.0, 1.0)).cuda()   # (-1)^(l - M) without the l
    return sign, par, torch.from_numpy(rev).cuda(), torch.from_numpy(odd).cuda()


def _series(matrix, x):
    """A real matrix times a complex array along its first index."""
    flat = x.reshape(x.shape[0], -1)
    return torch.complex(matrix @ flat.real, matrix @ flat.imag).reshape((matrix.shape[0],) + x.shape[1:])


def _exact_dsoft(grid, B):
    spec = torch.fft.fft2(grid, dim=(1, 2)).transpose(1, 2)          # [k][row = m2][col = m1]
    sign, par, rev, odd = _tables(B)
    spec = spec * _weights(B)[:, None, None]
    t = torch.where(odd[None], _series(_trig(B, np.sin), spec), _series(_trig(B, np.cos), spec)) * sign
    del spec
    out, p = [], _delta(B)
    for l in range(B):
        a, c = _fourier_rows(l, p[l]), _cols(B, l)
        block = t[: l + 1][:, c][:, :, c] * a[:, :, None] * a[:, None, :]
        f = block.sum(0) * par[c][:, c]
        if l % 2:
            f = torch.where(rev[c][:, c], -f, f)
        out.append(f.reshape(-1) * (math.pi / (2 * B * B)))
    return torch.cat(out)


def _exact_idsoft(coef, B):
    sign, par, rev, odd = _tables(B)
    t = torch.zeros((B, 2 * B, 2 * B), dtype=torch.complex128, device="cuda")
    p = _delta(B)
    for l in range(B):
        a, c = _fourier_rows(l, p[l]), _cols(B, l)
        f = coef[l * (4 * l * l - 1) // 3:][: (2 * l + 1) ** 2].reshape(2 * l + 1, 2 * l + 1) * par[c][:, c]
        if l % 2:
            f = torch.where(rev[c][:, c], -f, f)
        part = f[None] * a[:, :, None] * a[:, None, :]
        if l + 1 < B:
            r = l + 1   # the four corners of the orders' block
            for rows, prow in ((slice(0, r), slice(0, r)), (slice(2 * B - l, 2 * B), slice(r, 2 * l + 1))):
                for cs, pc in ((slice(0, r), slice(0, r)), (slice(2 * B - l, 2 * B), slice(r, 2 * l + 1))):
                    t[:r, rows, cs] += part[:, prow, pc]
        else:
            t[:, c[:, None], c[None, :]] += part
    t *= sign
    t *= 2 * B * B / math.pi
    spec = torch.where(odd[None], _series(_trig(B, np.sin).T.contiguous(), t), _series(_trig(B, np.cos).T.contiguous(), t))
    del t
    return torch.fft.ifft2(spec, dim=(1, 2)).transpose(1, 2).contiguous()


def exact(case, seed):
    op = case["op"]
    x = _inputs(case, seed)
    if op.startswith("layers"):
        f = torch.fft.fft2 if op == "layers_dft2" else torch.fft.ifft2
        return f(x[0], dim=(1, 2), norm="ortho")
    out = [(_exact_idsoft if op.endswith("idsoft") else _exact_dsoft)(v, B) for v, B in zip(x, _bandwidths(case))]
    return out if op.startswith("batch") else out[0]
