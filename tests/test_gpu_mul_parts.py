"""NTT products of M K points, forced through the tune table: two-part
transforms (M with two bits set: K1 = K 2^floor(log2 M) points and the rest)
and equal cosets, at full and barely used sizes, with operands longer than a
part (folded), squares and broadcast rows; and the row kernels' segment counts
around their groups.  Exact against Python integers."""
import numpy as np
import pytest

import batch_ref as ref
from helpers import rand_buf, to_dev

pytestmark = pytest.mark.gpu

K = 1 << 13


@pytest.fixture
def shape():
    import gpupi_b200 as g

    def force(log_k, M):
        g.tune_load(text=f"mul 64 school\nntt 2 {M << log_k} {log_k} {M}\n")

    yield force
    g.tune_load(g.TUNE_TABLE_PATH)


def product(ctx, N, La, Lb, form, rng, ones=False):
    sB = Lb if form == "pair" else 0
    if form == "square":
        Lb, sB = La, La
    A = rand_buf(rng, N, La, La)
    B = A if form == "square" else rand_buf(rng, N if form == "pair" else 1, Lb, Lb)
    if ones:
        A[:] = 0xFFFFFFFF
        B[:] = 0xFFFFFFFF
    C = np.zeros(N * (La + Lb), dtype=np.uint32)
    dA, dC = to_dev(A), to_dev(C)
    dB = dA if form == "square" else to_dev(B)
    ctx.mul_ntt(N, dA.ptr, La, La, dB.ptr, Lb, sB, dC.ptr, La + Lb)
    assert np.array_equal(dC.numpy(), ref.mul(N, A, La, La, B, Lb, sB, C, La + Lb))


@pytest.mark.parametrize("M", [2, 3, 4, 5, 6, 7, 9, 10, 12, 17, 20])
@pytest.mark.parametrize("N,form", [(1, "pair"), (3, "pair"), (2, "square"), (3, "bcast")])
def test_shapes(ctx, shape, M, N, form):
    rng = np.random.default_rng(M * 10 + N)
    full = M * K + 1                       # L_a + L_b - 1 = M K
    shape(13, M)
    product(ctx, N, full // 2, full - full // 2, form, rng)
    product(ctx, N, full // 2, full - full // 2, "pair", rng, ones=True)
    if form != "square":
        product(ctx, N, full - 700, 700, form, rng)   # an operand longer than either part
        product(ctx, N, 700, full - 700, form, rng)
        product(ctx, N, K // 2, 5, form, rng)         # one short block in a large shape
    else:
        product(ctx, N, full // 2 - 33, 0, form, rng)


@pytest.mark.parametrize("log_k", [14, 15, 16, 17, 18])
@pytest.mark.parametrize("M", [3, 5])
def test_column_lengths(ctx, shape, log_k, M):
    """Column passes of 2 to 32 points and more, with the second part's twist."""
    rng = np.random.default_rng(log_k + M)
    shape(log_k, M)
    full = (M << log_k) + 1
    product(ctx, 1, full // 2 + 1234, full - full // 2 - 1234, "pair", rng)
    product(ctx, 1, full - 300, 300, "pair", rng)


@pytest.mark.parametrize("N", [1, 2, 49, 50, 99, 197, 198, 297])
def test_row_groups(ctx, N):
    """Rows of one 4096-point segment per prime, around a CTA per segment (148),
    two groups per CTA and 148 x 2 CTAs (3 N segments in all), and a prime
    change inside a CTA's run; operands longer than half a segment and not
    (the first level then only multiplies)."""
    rng = np.random.default_rng(N)
    product(ctx, N, 70, 4000, "pair", rng)
    product(ctx, N, 70, 4000, "bcast", rng)
    product(ctx, N, 2048, 2040, "pair", rng)
    product(ctx, N, 2047, 0, "square", rng)


@pytest.mark.parametrize("table", [None, "mul 24 school\n", "mul 48 school\nmul 3072 tc\n",
                                   "ntt 8100 8192 13 2\nntt 16385 40960 13 5\n"])
def test_ragged_in_place(ctx, table):
    """Uneven products read and written where they lie: every bucket from a
    few limbs to the column-pass sizes, with the last table equal cosets and
    two-part transforms too, empty operands, operands of very different
    lengths, unordered output places with gaps left alone."""
    import gpupi_b200 as g
    rng = np.random.default_rng(5)
    pairs = [(1, 1), (0, 7), (9, 0), (3, 40), (200, 3), (130, 126), (255, 2), (250, 260), (1000, 30), (700, 1300),
             (2040, 2056), (4095, 2), (3000, 3000), (8000, 192), (4097, 4096), (60, 20000), (9000, 9001), (33000, 500)]
    pairs += [(int(a), int(b)) for a, b in 2 ** rng.uniform(0, 12.5, size=(60, 2))]
    rng.shuffle(pairs)
    La = np.array([p[0] for p in pairs], dtype=np.uint32)
    Lb = np.array([p[1] for p in pairs], dtype=np.uint32)
    A = rng.integers(0, 1 << 32, size=int(La.sum()) + 1, dtype=np.uint64).astype(np.uint32)
    B = rng.integers(0, 1 << 32, size=int(Lb.sum()) + 1, dtype=np.uint64).astype(np.uint32)
    A[int(La[:9].sum()):int(La[:19].sum())] = 0xFFFFFFFF
    B[int(Lb[:9].sum()):int(Lb[:19].sum())] = 0xFFFFFFFF
    Lc = La.astype(np.uint64) + Lb
    oa, ob = (np.concatenate([[0], np.cumsum(x.astype(np.uint64))[:-1]]).astype(np.uint64) for x in (La, Lb))
    oc = np.zeros(len(pairs), dtype=np.uint64)
    at = 3
    for i in rng.permutation(len(pairs)):
        oc[i] = at
        at += int(Lc[i]) + int(rng.integers(0, 4))
    C = np.full(at + 5, 0x5A5A5A5A, dtype=np.uint32)
    want = C.copy()
    for i, (a, b) in enumerate(pairs):
        x = int.from_bytes(A[int(oa[i]):int(oa[i]) + a].tobytes(), "little")
        y = int.from_bytes(B[int(ob[i]):int(ob[i]) + b].tobytes(), "little")
        want[int(oc[i]):int(oc[i]) + a + b] = np.frombuffer((x * y).to_bytes(4 * (a + b), "little"), dtype=np.uint32)
    dA, dB, dC = to_dev(A), to_dev(B), to_dev(C)
    try:
        if table:
            g.tune_load(text=table)
        ctx.mul_ragged(dA.ptr, oa, La, dB.ptr, ob, Lb, dC.ptr, oc)
    finally:
        g.tune_load(g.TUNE_TABLE_PATH)
    assert np.array_equal(dC.numpy(), want)


@pytest.mark.parametrize("last", [1366, 1370, 2041])
def test_ragged_carry_to_a_short_rows_end(ctx, last):
    """(2^(32m) + 1)(2^(64m) - 2^(32m) + 1) = 2^(96m) + 1, 3m + 1 limbs: its
    coefficient sums leave all-ones limbs that a carry runs through to the
    row's last limbs, in a bucket whose longest product is longer; the
    product with m = `last` ends the output."""
    rng = np.random.default_rng(last)
    ms = [1366, 1367, 1400, 2100, last]
    A, B = [], []
    for m in ms:
        a, b = np.zeros(m + 1, dtype=np.uint32), np.zeros(2 * m, dtype=np.uint32)
        a[0] = a[m] = b[0] = 1
        b[m:] = 0xFFFFFFFF
        A.append(a)
        B.append(b)
    A.insert(1, rand_buf(rng, 1, 4001, 4001))
    B.insert(1, rand_buf(rng, 1, 4100, 4100))
    La, Lb = (np.array([len(x) for x in v], dtype=np.uint32) for v in (A, B))
    oa, ob, oc = (np.concatenate([[0], np.cumsum(x)[:-1]]).astype(np.uint64) for x in (La, Lb, La + Lb))
    want = []
    for a, b in zip(A, B):
        x, y = (int.from_bytes(v.tobytes(), "little") for v in (a, b))
        want.append(np.frombuffer((x * y).to_bytes(4 * (len(a) + len(b)), "little"), dtype=np.uint32))
    want = np.concatenate(want)
    dA, dB, dC = to_dev(np.concatenate(A)), to_dev(np.concatenate(B)), to_dev(np.zeros_like(want))
    ctx.mul_ragged(dA.ptr, oa, La, dB.ptr, ob, Lb, dC.ptr, oc)
    assert np.array_equal(dC.numpy(), want)


def test_ragged_tensor_products_in_one_launch(ctx):
    import gpupi_b200 as g
    rng = np.random.default_rng(2)
    La, Lb = (rng.integers(70, 1200, size=40).astype(np.uint32) for _ in range(2))
    A, B = rand_buf(rng, 1, int(La.sum()), int(La.sum())), rand_buf(rng, 1, int(Lb.sum()), int(Lb.sum()))
    oa, ob, oc = (np.concatenate([[0], np.cumsum(x)[:-1]]).astype(np.uint64) for x in (La, Lb, La + Lb))
    dA, dB, dC = to_dev(A), to_dev(B), to_dev(np.zeros(int((La + Lb).sum()), dtype=np.uint32))
    try:
        g.tune_load(text="mul 2560 tc\n")
        g.timer_reset()
        g.timer_enable(True)
        ctx.mul_ragged(dA.ptr, oa, La, dB.ptr, ob, Lb, dC.ptr, oc)
        g.timer_enable(False)
        assert g.timer_report()["schoolbook_tc"][0] == 1
    finally:
        g.timer_enable(False)
        g.timer_reset()
        g.tune_load(g.TUNE_TABLE_PATH)
    got = dC.numpy()
    for i in range(40):
        x, y, z = (int.from_bytes(v[int(o[i]):int(o[i]) + int(n)].tobytes(), "little")
                   for v, o, n in ((A, oa, La[i]), (B, ob, Lb[i]), (got, oc, La[i] + Lb[i])))
        assert z == x * y
