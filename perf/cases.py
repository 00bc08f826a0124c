"""Timed cases of the framework: what its users have it do, through the public Python API.

A case is a dict of plain values; ``kind`` says which entry points it drives:

``mul``      ``Context.mul``: N products of la x lb limbs, ``form`` "pair" (N
             pairs), "square" (B is A) or "bcast" (one B for every row).
``ragged``   ``Context.mul_ragged``: N products with lengths log-uniform in
             [lo, hi] limbs per operand, rows packed.
``linear``   the linear-time operations of one merge step on N rows of L
             limbs: shift_add, sub, mul_small, exactdiv_small (rows of at most
             128 limbs), shift_bits, limblength_max.
``convert``  ``Context.convert_decimal``: a binary fraction to decimal digits.
``pi``       ``pi_compute`` with the digits and RET copied to pinned host
             buffers, as a program that wants the digits calls it.

Limbs are uniform random 32-bit words, the distribution the operations meet
inside the pi computation; every result is an exact integer.
"""
from __future__ import annotations

import decimal
import math
import sys

import numpy as np
import torch

import gpupi_b200 as g

SHIFT = 15             # bits of the merge step's shifts
FACTOR = 10005         # the single-limb factor (odd) of mul_small / exactdiv_small
EXACTDIV_MAX = 128     # limbs per row exactdiv_small accepts
PI_JITTER = 512        # a pi case asks for up to this many digits fewer, by seed

_ctx = None


def _context() -> g.Context:
    """A program opens one context and keeps it for its lifetime."""
    global _ctx
    if _ctx is None:
        _ctx = g.Context()
    return _ctx


def listed() -> list[dict]:
    return [
        # one product of two short numbers: the latency of a call
        {"name": "mul_one", "kind": "mul", "n": 1, "la": 180, "lb": 171, "form": "pair"},
        # a lower level of a splitting tree: very many products of a dozen limbs
        {"name": "mul_rows_14", "kind": "mul", "n": 262144, "la": 14, "lb": 13, "form": "pair"},
        # the middle levels: thousands of products of a few hundred limbs
        {"name": "mul_rows_431", "kind": "mul", "n": 8192, "la": 431, "lb": 397, "form": "pair"},
        # products just past the schoolbook sizes
        {"name": "mul_rows_2k", "kind": "mul", "n": 1024, "la": 2001, "lb": 1903, "form": "pair"},
        # the upper levels: tens of long products
        {"name": "mul_rows_20k", "kind": "mul", "n": 96, "la": 20011, "lb": 18003, "form": "pair"},
        # the largest product of the reference's API: 2^27 x 2^27 limbs
        {"name": "mul_2_27", "kind": "mul", "n": 1, "la": 1 << 27, "lb": 1 << 27, "form": "pair"},
        # independent products of uneven lengths in one call
        {"name": "ragged_4096", "kind": "ragged", "n": 4096, "lo": 8, "hi": 4096},
        # the linear operations of a merge level with many rows of a hundred limbs
        {"name": "linear_rows_101", "kind": "linear", "n": 65536, "l": 101},
        # the same on one very long number (the top of the tree)
        {"name": "linear_long", "kind": "linear", "n": 1, "l": (1 << 26) + 3},
        # decimal conversion of a 2^25-limb fraction to 322,961,408 digits
        {"name": "convert_2_25", "kind": "convert", "leaf": 308, "levels": 20},
        # pi at a million and at a billion digits, digits delivered to the host
        {"name": "pi_1e6", "kind": "pi", "digits": 1_000_000},
        {"name": "pi_1e9", "kind": "pi", "digits": 1_000_000_000},
    ]


def _log(rng, lo: float, hi: float) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["mul", "mul", "mul", "mul", "ragged", "linear", "convert", "pi"])
    if kind == "mul":
        la = _log(rng, 1, 1 << 26)
        lb = max(1, int(la * rng.uniform(0.4, 1.0)))
        most = max(1, (1 << 26) // (la + lb))
        n = min(1 << 21, _log(rng, 1, most))
        return {"kind": "mul", "n": n, "la": la, "lb": lb, "form": rng.choice(["pair", "pair", "pair", "square", "bcast"])}
    if kind == "ragged":
        lo = _log(rng, 1, 256)
        return {"kind": "ragged", "n": _log(rng, 16, 4096), "lo": lo, "hi": lo * _log(rng, 2, 64)}
    if kind == "linear":
        l = _log(rng, 2, 1 << 26)
        return {"kind": "linear", "n": _log(rng, 1, max(1, (1 << 26) // l)), "l": l}
    if kind == "convert":
        return {"kind": "convert", "leaf": rng.randint(288, 575), "levels": rng.randint(4, 19)}
    return {"kind": "pi", "digits": _log(rng, 20_000, 200_000_000)}


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _words(n: int, gen) -> torch.Tensor:
    return torch.randint(-(1 << 31), 1 << 31, (n,), dtype=torch.int32, device="cuda", generator=gen)


def _gen(seed: int):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    return gen


def _ragged_lengths(case: dict, seed: int):
    rng = np.random.default_rng(seed)
    lo, hi = math.log2(case["lo"]), math.log2(case["hi"])
    la, lb = (np.floor(2 ** rng.uniform(lo, hi, size=case["n"])).astype(np.uint32) for _ in range(2))

    def starts(lens):
        return np.concatenate([[0], np.cumsum(lens.astype(np.uint64))[:-1]]).astype(np.uint64)

    return la, lb, starts(la), starts(lb), starts(la.astype(np.uint64) + lb)


def _ragged_room(case: dict) -> int:
    """Limbs of an output buffer that holds any such batch."""
    return 2 * case["n"] * case["hi"]


def _pi_digits(case: dict, seed: int) -> int:
    return case["digits"] - (seed * 2654435761 % (1 << 32)) % PI_JITTER


def _convert_limbs(case: dict) -> tuple[int, int]:
    total = case["leaf"] << case["levels"]
    return total, (int(total * math.log2(10)) + 96 + 31) // 32


def _form(case: dict) -> tuple[int, int, int]:
    """Rows of B, limbs of B, stride of B."""
    if case["form"] == "square":
        return case["n"], case["la"], case["la"]
    if case["form"] == "bcast":
        return 1, case["lb"], 0
    return case["n"], case["lb"], case["lb"]


def prepare(case: dict, seed: int) -> dict:
    gen, kind = _gen(seed), case["kind"]
    s = {"case": case, "ctx": _context()}
    if kind == "mul":
        rows, lb, _ = _form(case)
        s["A"] = _words(case["n"] * case["la"], gen)
        s["B"] = s["A"] if case["form"] == "square" else _words(rows * lb, gen)
        s["C"] = torch.zeros(case["n"] * (case["la"] + lb), dtype=torch.int32, device="cuda")
    elif kind == "ragged":
        s["la"], s["lb"], s["oa"], s["ob"], s["oc"] = _ragged_lengths(case, seed)
        na, nb = int(s["la"].sum(dtype=np.uint64)), int(s["lb"].sum(dtype=np.uint64))
        s["A"], s["B"] = _words(na, gen), _words(nb, gen)
        s["C"] = torch.zeros(_ragged_room(case), dtype=torch.int32, device="cuda")
    elif kind == "linear":
        n, l = case["n"], case["l"]
        s["A"], s["B"] = _words(n * l, gen), _words(n * l, gen)
        for name, length in (("sum", l + 1), ("dif", l + 1), ("scaled", l + 1), ("shifted", l)):
            s[name] = torch.zeros(n * length, dtype=torch.int32, device="cuda")
    elif kind == "convert":
        total, limbs = _convert_limbs(case)
        s["X"] = _words(limbs, gen)
        s["out"] = torch.zeros(total, dtype=torch.uint8, device="cuda")
    else:
        s["digits"] = _pi_digits(case, seed)
        s["text"] = torch.zeros(case["digits"], dtype=torch.uint8, pin_memory=True)
        s["ret"] = torch.zeros(g.ret_limbs_bound(case["digits"]), dtype=torch.int32, pin_memory=True)
    return s


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
def run(s: dict):
    case, ctx, kind = s["case"], s["ctx"], s["case"]["kind"]
    if kind == "mul":
        n, la = case["n"], case["la"]
        _, lb, sb = _form(case)
        ctx.mul(n, s["A"].data_ptr(), la, la, s["B"].data_ptr(), lb, sb, s["C"].data_ptr(), la + lb, la + lb)
        return s["C"]
    if kind == "ragged":
        ctx.mul_ragged(s["A"].data_ptr(), s["oa"], s["la"], s["B"].data_ptr(), s["ob"], s["lb"], s["C"].data_ptr(),
                       s["oc"])
        return s["C"]
    if kind == "linear":
        n, l = case["n"], case["l"]
        A, B = s["A"].data_ptr(), s["B"].data_ptr()
        ctx.shift_add(n, A, l, l, B, l, l, SHIFT, s["sum"].data_ptr(), l + 1, l + 1)
        ctx.sub(n, s["sum"].data_ptr(), l + 1, l + 1, A, l, l, s["dif"].data_ptr(), l + 1, l + 1)
        ctx.mul_small(n, B, l, l, FACTOR, s["scaled"].data_ptr(), l + 1, l + 1)
        if l + 1 <= EXACTDIV_MAX:
            ctx.exactdiv_small(n, s["scaled"].data_ptr(), l + 1, l + 1, FACTOR)
        ctx.shift_bits(n, A, l, l, s["shifted"].data_ptr(), l, l, -SHIFT)
        longest = ctx.limblength_max(n, s["dif"].data_ptr(), l + 1, l + 1)
        return {"sum": s["sum"], "dif": s["dif"], "scaled": s["scaled"], "shifted": s["shifted"], "longest": longest}
    if kind == "convert":
        total, limbs = _convert_limbs(case)
        ctx.convert_decimal(s["X"].data_ptr(), limbs, 32 * limbs, total, case["leaf"], s["out"].data_ptr())
        return s["out"]
    g.pi_compute(s["digits"], ctx, host_digits=s["text"], host_ret=s["ret"])
    return {"digits": s["text"], "ret": s["ret"]}


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------
def _mul_ops(la: float, lb: float) -> float:
    """Two operations per 32-bit limb product by the schoolbook, or the
    n log n of three transforms modulo three word-size primes, if fewer."""
    n = la + lb
    return min(2.0 * la * lb, 3 * 3 * 3 * n * math.log2(max(n, 2.0)))


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "mul":
        rows, lb, _ = _form(case)
        n, la = case["n"], case["la"]
        b_read = 0 if case["form"] == "square" else rows * lb
        return {"bytes": 4.0 * (n * la + b_read + n * (la + lb)), "flops": n * _mul_ops(la, lb)}
    if kind == "ragged":
        la, lb = _ragged_lengths(case, 0)[:2]
        limbs = float(la.sum(dtype=np.float64) + lb.sum(dtype=np.float64))
        return {"bytes": 8.0 * limbs, "flops": sum(_mul_ops(float(a), float(b)) for a, b in zip(la, lb))}
    if kind == "linear":
        n, l = case["n"], case["l"]
        return {"bytes": 4.0 * n * (2.0 * l + 3.0 * (l + 1) + l), "flops": 6.0 * n * l}
    if kind == "convert":
        total, limbs = _convert_limbs(case)
        # one truncated product of half the bits per level and half
        flops = sum((1 << k) * _mul_ops(limbs / 2 ** (k + 1), limbs / 2 ** (k + 1)) for k in range(case["levels"]))
        return {"bytes": 4.0 * limbs + total, "flops": flops}
    limbs = case["digits"] * math.log2(10) / 32
    levels = max(1, int(math.log2(limbs)) - 4)
    # each level of the tree: four products over all of the level's limbs
    flops = sum(4 * (1 << k) * _mul_ops(limbs / 2 ** (k + 1), limbs / 2 ** (k + 1)) for k in range(levels))
    return {"bytes": 4.0 * limbs + case["digits"], "flops": flops}


def tolerance(case: dict):
    return "exact"   # integers and decimal digits, whatever the algorithm


# ---------------------------------------------------------------------------
# The same results without this repository's code
# ---------------------------------------------------------------------------
def _carry(c: torch.Tensor) -> torch.Tensor:
    """Rows of int64 byte coefficients (any sign) -> rows of bytes, modulo the row's width."""
    while True:
        over = c >> 8
        c = c & 255
        if not bool(over.any()):
            return c.to(torch.uint8)
        c[:, 1:] += over[:, :-1]


def _bytes(x: torch.Tensor, rows: int) -> torch.Tensor:
    return x.view(torch.uint8).view(rows, -1)


def _product(a: torch.Tensor, b: torch.Tensor) -> torch.Tensor:
    """Rows of bytes x rows of bytes by a 64-bit floating transform: the
    coefficients stay below 2^44, far inside what it resolves."""
    n = a.shape[1] + b.shape[1]
    size = 1 << (n - 1).bit_length()
    f = torch.fft.rfft(a.double(), size) * torch.fft.rfft(b.double(), size)
    return _carry(torch.fft.irfft(f, size)[:, :n].round().to(torch.int64))


def _limbs(rows: torch.Tensor) -> torch.Tensor:
    return rows.contiguous().view(torch.int32).view(-1)


def _pi_text(digits: int) -> str:
    """The digits after "3." from Chudnovsky's series in decimal arithmetic."""
    decimal.getcontext().prec = 4 * digits + 200
    decimal.getcontext().Emax = decimal.MAX_EMAX
    D = decimal.Decimal
    c3 = 640320 ** 3 // 24

    def split(a, b):
        if b - a == 1:
            p = (6 * a - 5) * (2 * a - 1) * (6 * a - 1) if a else 1
            q = a ** 3 * c3 if a else 1
            t = p * (13591409 + 545140134 * a)
            return p, q, -t if a & 1 else t
        m = (a + b) // 2
        p1, q1, t1 = split(a, m)
        p2, q2, t2 = split(m, b)
        if b - a > 256 >= m - a:   # long products in decimal, short ones as integers
            p1, q1, t1, p2, q2, t2 = map(D, (p1, q1, t1, p2, q2, t2))
        return p1 * p2, q1 * q2, q2 * t1 + p1 * t2

    _, q, t = split(0, digits // 14 + 2)
    decimal.getcontext().prec = digits + 30
    pi = (D(q) * 426880 * D(10005).sqrt()) / D(t)
    return str(pi)[2:2 + digits]


def exact(case: dict, seed: int):
    kind = case["kind"]
    sys.set_int_max_str_digits(0)
    if kind == "pi":
        if case["digits"] > 400_000:   # the decimal series would take too long
            return None
        want = _pi_digits(case, seed)
        text = np.zeros(case["digits"], dtype=np.uint8)
        text[:want] = np.frombuffer(_pi_text(want).encode(), dtype=np.uint8)
        return {"digits": torch.from_numpy(text), "ret": None}
    if kind == "convert":
        total, limbs = _convert_limbs(case)
        if total > 1_000_000:
            return None
        x = int.from_bytes(prepare(case, seed)["X"].cpu().numpy().tobytes(), "little")
        digits = str((x * 10 ** total) >> (32 * limbs)).rjust(total, "0")
        return torch.from_numpy(np.frombuffer(digits.encode(), dtype=np.uint8).copy())
    if kind == "mul":
        n, la = case["n"], case["la"]
        rows, lb, _ = _form(case)
        if n * (la + lb) > 1 << 24:
            return None
        s = prepare(case, seed)
        a, b = _bytes(s["A"], n), _bytes(s["B"], rows)
        return _limbs(_product(a, b))
    if kind == "ragged":
        s = prepare(case, seed)
        out, left = [], _ragged_room(case)
        for i in range(case["n"]):
            a = s["A"][int(s["oa"][i]):][:int(s["la"][i])]
            b = s["B"][int(s["ob"][i]):][:int(s["lb"][i])]
            out.append(_limbs(_product(_bytes(a.clone(), 1), _bytes(b.clone(), 1))))
            left -= out[-1].numel()
        out.append(torch.zeros(left, dtype=torch.int32, device="cuda"))
        return torch.cat(out)
    n, l = case["n"], case["l"]
    if n * l > 1 << 24:
        return None
    s = prepare(case, seed)
    a, b = (torch.nn.functional.pad(_bytes(s[x], n).to(torch.int64), (0, 4)) for x in "AB")
    low = a << SHIFT
    total = _carry(low + b)
    dif = _carry(total.to(torch.int64) - a)
    scaled = b.to(torch.uint8) if l + 1 <= EXACTDIV_MAX else _carry(b * FACTOR)
    down = a[:, :-4] << (16 - SHIFT)
    shifted = torch.nn.functional.pad(_carry(torch.nn.functional.pad(down, (0, 4)))[:, 2:4 * l], (0, 2))
    # A >> 15 = (A << 1) >> 16: two bytes down, the carry byte above the row kept
    top = _carry(torch.nn.functional.pad(down, (0, 4)))[:, 4 * l:4 * l + 2]
    shifted[:, 4 * l - 2:] = top
    words = dif.contiguous().view(torch.int32).view(n, l + 1) != 0
    used = words.any(dim=0).nonzero()
    return {"sum": _limbs(total), "dif": _limbs(dif), "scaled": _limbs(scaled), "shifted": _limbs(shifted),
            "longest": int(used[-1]) + 1 if len(used) else 0}
