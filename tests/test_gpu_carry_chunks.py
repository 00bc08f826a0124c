"""Carry-chain kernels at the edges of their four-limb chunks: lengths around
each lane-group size and the tile size, every alignment of the operands
against the 16-byte chunks of C, in-place use, and carries that run through
many tiles (looked back over 1024 tiles at a time).  All results bit-exact."""
import numpy as np
import pytest

import batch_ref as ref
from helpers import rand_buf, to_dev

pytestmark = pytest.mark.gpu

LENGTHS = [1, 3, 4, 5, 12, 13, 14, 28, 29, 30, 60, 61, 62, 124, 125, 126, 509, 512, 513, 4093, 4094, 4096, 4097, 8190]


@pytest.mark.parametrize("Lc", LENGTHS)
def test_lengths_and_alignments(ctx, Lc):
    """Every offset of A, B and C modulo four limbs; rows one limb apart in
    stride so that the alignment also changes from row to row."""
    rng = np.random.default_rng(Lc)
    N = 5
    La, Lb = max(Lc - 1, 0), max(Lc - 3, 1)
    sA, sB, sC = Lc + 1, Lc + 2, Lc + 1
    for oa, ob, oc in [(0, 0, 0), (1, 0, 0), (0, 2, 1), (3, 1, 2), (2, 3, 3)]:
        A, B, C = rand_buf(rng, N + 1, sA, La), rand_buf(rng, N + 1, sB, Lb), rand_buf(rng, N + 1, sC, 0)
        A[oa + 2 * sA: oa + 2 * sA + La] = 0xFFFFFFFF          # a row that carries all the way
        B[ob + 2 * sB: ob + 2 * sB + Lb] = 0
        B[ob + 2 * sB] = 1
        for op in ("add", "sub", "shift_add", "shift_sub", "mul_small"):
            dA, dB, dC = to_dev(A), to_dev(B), to_dev(C)
            a, b, c = (dA.at(oa), La, sA), (dB.at(ob), Lb, sB), (dC.at(oc), Lc, sC)
            if op == "mul_small":
                ctx.mul_small(N, *a, 0xFFFFFFFB, *c)
                want = ref.mul_small(N, A[oa:], La, sA, 0xFFFFFFFB, C[oc:], Lc, sC)
            elif op.startswith("shift"):
                getattr(ctx, op)(N, *a, *b, 45, *c)
                want = getattr(ref, op)(N, A[oa:], La, sA, B[ob:], Lb, sB, 45, C[oc:], Lc, sC)
            else:
                getattr(ctx, op)(N, *a, *b, *c)
                want = getattr(ref, op)(N, A[oa:], La, sA, B[ob:], Lb, sB, C[oc:], Lc, sC)
            got = dC.numpy()
            assert np.array_equal(got[oc:], want), (op, oa, ob, oc)
            assert np.array_equal(got[:oc], C[:oc])


IN_PLACE = [(N, L) for N in (1, 3, 150)
            for L in (5, 125, 126, 130, 144, 145, 254, 300, 509, 513, 1300, 4090, 4096, 4097, 13000, 70001)
            if N * L <= 1 << 20]


@pytest.mark.parametrize("N,L", IN_PLACE)
def test_small_in_place(ctx, N, L):
    """C is A: also for mul_small, whose limbs read the one below."""
    rng = np.random.default_rng(L + N)
    A = rand_buf(rng, N + 1, L + 1, L)
    A[2:2 + L // 2] = 0xFFFFFFFF
    for op in ("mul_small", "add_small", "sub_small"):
        dA = to_dev(A)
        getattr(ctx, op)(N, dA.at(1), L, L + 1, 0xFFFFFFFB, dA.at(1), L, L + 1)
        want = getattr(ref, op)(N, A[1:], L, L + 1, 0xFFFFFFFB, A[1:], L, L + 1)
        assert np.array_equal(dA.numpy()[1:], want), op


@pytest.mark.parametrize("L", [7, 61, 4095, 13000])
@pytest.mark.parametrize("op", ["add", "sub"])
def test_in_place_misaligned(ctx, op, L):
    rng = np.random.default_rng(L)
    N = 3
    A, B = rand_buf(rng, N + 1, L, L), rand_buf(rng, N + 1, L + 2, L)
    dA, dB = to_dev(A), to_dev(B)
    getattr(ctx, op)(N, dA.at(3), L, L, dB.at(1), L, L + 2, dA.at(3), L, L)
    assert np.array_equal(dA.numpy()[3:], getattr(ref, op)(N, A[3:], L, L, B[1:], L, L + 2, A[3:], L, L))


@pytest.mark.parametrize("tiles", [33, 1023, 1024, 1025, 3 * 1024 + 1])
@pytest.mark.parametrize("off", [0, 1])
def test_carry_through_many_tiles(ctx, tiles, off):
    """(2^(32 L) - 1) + 1 through every tile, then with one absorbing limb on the
    way; 0 - 1 through every tile, and up to one limb that absorbs it."""
    import torch
    L = tiles * 4096 - 5
    A = torch.full((L + off,), -1, dtype=torch.int32, device="cuda")
    B = torch.zeros(1 + off, dtype=torch.int32, device="cuda")
    B[off] = 1
    C = torch.full((L + 1 + off,), 7, dtype=torch.int32, device="cuda")
    a, b, c = A.data_ptr() + 4 * off, B.data_ptr() + 4 * off, C.data_ptr() + 4 * off
    ctx.add(1, a, L, L, b, 1, 1, c, L + 1, L + 1)
    assert int(C[off:off + L].ne(0).sum()) == 0 and int(C[off + L]) == 1
    stop = 4096 * (tiles // 2) + 77
    A[off + stop] = 41
    ctx.add(1, a, L, L, b, 1, 1, c, L + 1, L + 1)
    assert int(C[off:off + stop].ne(0).sum()) == 0 and int(C[off + stop]) == 42
    assert int(C[off + stop + 1:off + L].ne(-1).sum()) == 0 and int(C[off + L]) == 0
    # 0 - 1 borrows through every limb, or up to the first nonzero one
    A.zero_()
    ctx.sub(1, a, L, L, b, 1, 1, c, L + 1, L + 1)
    assert int(C[off:off + L + 1].ne(-1).sum()) == 0
    A[off + stop] = 41
    ctx.sub(1, a, L, L, b, 1, 1, c, L + 1, L + 1)
    assert int(C[off:off + stop].ne(-1).sum()) == 0 and int(C[off + stop]) == 40
    assert int(C[off + stop + 1:off + L + 1].ne(0).sum()) == 0


WARP_ROWS = [(5, Lc) for Lc in (127, 128, 129, 144, 145, 192, 193, 253, 254, 381, 382, 511, 1021, 1300)]
WARP_ROWS += [(148, 509), (148, 510), (149, 510), (149, 193), (4095, 254), (4096, 254), (4096, 381), (4096, 382)]


@pytest.mark.parametrize("N,Lc", WARP_ROWS)
def test_rows_of_a_warp(ctx, N, Lc):
    """Rows a warp handles one limb or four limbs per lane, either side of each
    change between the two and between 256 and 512 limbs per step, with rows
    that carry all the way and strides that change the alignment."""
    rng = np.random.default_rng(Lc * 5000 + N)
    La, Lb, sA, sB, sC = Lc - 1, Lc - 2, Lc, Lc + 1, Lc + 2
    A, B, C = rand_buf(rng, N, sA, La), rand_buf(rng, N, sB, Lb), rand_buf(rng, N, sC, 0)
    for r in range(0, N, 3):
        A[r * sA:r * sA + La] = 0xFFFFFFFF if r % 2 else 0
        B[r * sB:r * sB + Lb] = 0
        B[r * sB] = 1
    for op in ("add", "sub", "add_small", "sub_small", "mul_small", "shift_add", "shift_sub"):
        dA, dB, dC = to_dev(A), to_dev(B), to_dev(C)
        a, b, c = (dA.ptr, La, sA), (dB.ptr, Lb, sB), (dC.ptr, Lc, sC)
        if op.endswith("small"):
            getattr(ctx, op)(N, *a, 0xFFFFFFFB, *c)
            want = getattr(ref, op)(N, A, La, sA, 0xFFFFFFFB, C, Lc, sC)
        elif op.startswith("shift"):
            getattr(ctx, op)(N, *a, *b, 45, *c)
            want = getattr(ref, op)(N, A, La, sA, B, Lb, sB, 45, C, Lc, sC)
        else:
            getattr(ctx, op)(N, *a, *b, *c)
            want = getattr(ref, op)(N, A, La, sA, B, Lb, sB, C, Lc, sC)
        assert np.array_equal(dC.numpy(), want), op


@pytest.mark.parametrize("N,L", [(1, 1), (1, 33), (1, 128), (2, 33), (2, 128), (8, 8), (8, 9), (9, 31), (33, 32), (33, 33), (40, 40),
                                 (40, 41), (65, 102), ((1 << 18) - 1, 3), (1 << 18, 3), ((1 << 18) + 5, 1)])
def test_exactdiv_kernels(ctx, N, L):
    """Either side of the choice between the two kernels, and of their groups
    of eight limbs; rows need not be multiples of the divisor."""
    rng = np.random.default_rng(N + L)
    A = rand_buf(rng, N, L + 1, L)
    dA = to_dev(A)
    ctx.exactdiv_small(N, dA.ptr, L, L + 1, 0x13579BDF)
    assert np.array_equal(dA.numpy(), ref.exactdiv_small(N, A, L, L + 1, 0x13579BDF))
