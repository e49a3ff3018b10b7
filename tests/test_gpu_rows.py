"""GPU parity of the row kernels that the binning picks by structure, at the edges
of their ranges, bit for bit against the CPU oracle; the kernels that ran are
read from the engine's per-kernel profile."""
import numpy as np
import pytest

import oracle
from appt_spgemm_b200 import csr
from parity import assert_same_csr

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.fixture(scope="module", params=["default", "binned"])
def eng(request):
    from appt_spgemm_b200.engine import Engine
    e = Engine("cuda:0", **({} if request.param == "default" else {"small_max_nnz": -1}))
    e.binned = request.param == "binned"
    yield e
    e.check_device_status()
    e.close()


def product(eng, A, task):
    """The product twice from one plan (the second re-derives what depends on
    A's values), compared both times; returns the kernel labels."""
    from appt_spgemm_b200.engine import CsrDevice
    eng.profile_enable(True)
    eng.profile_reset()
    p = eng.plan(CsrDevice.from_host(A, "cuda:0"), task)
    ref = oracle.multiply(A, task)
    for _ in range(2):
        C = p.execute()
        torch.cuda.synchronize()
        assert_same_csr(C.to_host(), ref, task)
    p.close()
    labels = set(eng.profile_read()["kernels"])
    eng.profile_enable(False)
    eng.check_device_status()
    return labels


def from_rows(n, rows, seed):
    """CSR of the given column lists (sorted here), values uniform(-1, 1)."""
    rows = [np.unique(np.asarray(r, dtype=np.int64)) for r in rows]
    rp = np.zeros(n + 1, dtype=np.int32)
    rp[1:len(rows) + 1] = np.cumsum([len(r) for r in rows])
    rp[len(rows) + 1:] = rp[len(rows)]
    col = np.concatenate(rows).astype(np.int32)
    return csr.CsrHost(n, rp, col, np.random.default_rng(seed).uniform(-1, 1, len(col)))


# rows of exactly d·d products over 20,011 columns: either side of the kernel's
# smallest row (8), of each row capacity and of the largest (4096)
@pytest.mark.parametrize("d", [2, 3, 6, 7, 11, 12, 16, 17, 19, 20, 22, 23, 27, 28, 32, 33, 39, 45, 46, 55,
                               64, 65])
def test_sorted_rows(eng, d):
    labels = product(eng, csr.uniform(20011, d, seed=d), "AA")
    if eng.binned:
        assert any(x.startswith("num/sort") for x in labels) == (3 <= d <= 64)


def test_sorted_rows_uneven(eng):
    # empty B rows between others, rows of very different lengths, repeated columns
    rng = np.random.default_rng(5)
    n = 6007
    rows = [rng.integers(0, n, rng.choice([0, 0, 1, 2, 30, 70])) for _ in range(n)]
    for task in ("AA", "AAt", "AAtS"):
        product(eng, from_rows(n, rows, 6), task)


@pytest.mark.parametrize("width", [1, 60, 700])
def test_sorted_rows_clustered(eng, width):
    # a row's products fall into a few columns at one end of a wide span, so one
    # bucket holds them all
    n = 50021
    rng = np.random.default_rng(width)
    rows = [np.concatenate([rng.integers(0, 40, 9), [n - 1 - i % 5]]) for i in range(400)]
    rows += [[n - 1 - i % 3, i % width] for i in range(400, 3000)]
    rows[:40] = [np.concatenate([rng.integers(1000, 1000 + width, 12), [n - 3]]) for _ in range(40)]
    product(eng, from_rows(n, rows, 7), "AA")


def hub_rows(n, hubs, width, seed):
    """`hubs` rows of `width` random columns each, the first of them 3·width, among
    rows of 8 and empty rows; columns skewed to the low end."""
    rng = np.random.default_rng(seed)
    rows = []
    for i in range(n):
        if i % (n // hubs) == 1:
            k = 3 * width if i == 1 else width
        else:
            k = 0 if i % 7 == 3 else 8
        rows.append((n * rng.random(k) ** 2).astype(np.int64))
    return from_rows(n, rows, seed)


# spans below one panel, of a panel and a bit, ragged and many; panels of 256,
# 512 and 1024 columns (few or many tasks)
@pytest.mark.parametrize("n,hubs,width", [(601, 30, 90), (1025, 40, 200), (3001, 60, 300),
                                          (16411, 300, 400)])
@pytest.mark.parametrize("task", ["AA", "AAt", "AAtS"])
def test_paneled_rows(eng, n, hubs, width, task):
    labels = product(eng, hub_rows(n, hubs, width, seed=n), task)
    assert "num/panels" in labels or n < 1024  # (up to 1024 columns: narrow rows)


def test_paneled_rows_signed_zeros():
    # products of −0.0, cancelled sums and underflow stay entries, with the
    # oracle's signs; every row through panels that search for their slices or
    # read them from the table
    from appt_spgemm_b200.engine import Engine
    A = hub_rows(2003, 50, 200, seed=9)
    rng = np.random.default_rng(10)
    A.val = rng.choice([0.0, -0.0, 1.0, -1.0, 1e-200, -1e-200], A.nnz)
    with Engine("cuda:0", small_max_nnz=-1, force_heavy=1) as e:
        e.binned = True
        for task in ("AA", "AAt", "AAtS"):
            assert "num/panels" in product(e, A, task)


def test_paneled_rows_without_table():
    # many columns and a small C: the slice bounds would take more memory than
    # they may, so the panels search for them
    from appt_spgemm_b200.engine import Engine
    n, hubs = 262144, 280
    rng = np.random.default_rng(11)
    ids = rng.choice(n, hubs, replace=False)
    rows = [[i] for i in range(n)]
    for i in ids:
        rows[i] = np.concatenate([ids, rng.integers(0, n, 240)])
    with Engine("cuda:0", small_max_nnz=-1) as e:
        e.binned = True
        assert "num/panels" in product(e, from_rows(n, rows, 12), "AA")


def by_offsets(n, offsets, seed):
    """Row i holds the columns i + o that lie in the matrix: runs of shifted rows."""
    return from_rows(n, [[i + o for o in offsets if 0 <= i + o < n] for i in range(n)], seed)


# whether runs are taken: enough rows (8), products (768) and room for the rows of
# B, which lie side by side or not; runs are cut at 256 rows
@pytest.mark.parametrize("n,offsets,taken", [
    (7, [0], False), (9, [0], True), (300, [0], True), (261, [-1, 0, 1], True),
    (1000, [-30, -1, 0, 1, 30], True), (1500, list(range(-13, 14)), True),
    (1501, list(range(-13, 15)), False), (700, list(range(-60, 60, 5)), False),
    (2600, [-700, -3, 0, 1, 2, 50, 51, 900], True), (70001, [-30000, -1, 0, 1, 33000], True)])
@pytest.mark.parametrize("task", ["AA", "AAt"])
def test_shifted_rows(n, offsets, taken, task):
    from appt_spgemm_b200.engine import Engine
    with Engine("cuda:0", small_max_nnz=-1) as e:
        e.binned = True
        labels = product(e, by_offsets(n, offsets, seed=n), task)
        assert any(x.startswith("num/runs") for x in labels) == taken


@pytest.mark.parametrize("side", [8, 9, 21, 34, 45])
def test_shifted_rows_stencil(eng, side):
    product(eng, csr.stencil27(side, seed=side), "AAt")
    product(eng, csr.laplace2d(side * side // 3), "AA")


def test_shifted_rows_interrupted(eng):
    # single entries dropped, added and moved break the runs; consecutive instances
    # of a batch must not be taken for one run's columns
    rng = np.random.default_rng(13)
    rows = [[i + o for o in (-90, -1, 0, 1, 2, 90) if 0 <= i + o < 3000] for i in range(3000)]
    for i in rng.integers(0, 3000, 40):
        rows[i] = rows[i][1:] if i % 2 else rows[i] + [int(rng.integers(0, 3000))]
    A = from_rows(3000, rows, 14)
    product(eng, A, "AA")
    product(eng, A, "AAt")
    from appt_spgemm_b200.engine import CsrDevice
    As = [by_offsets(n, [-1, 0, 1], n) for n in (40, 41, 300, 7)] + [csr.stencil27(9, seed=2)]
    R = eng.multiply_batched([CsrDevice.from_host(M, "cuda:0") for M in As], "AA")
    for b, M in enumerate(As):
        rp, col, val = R.instance(b)
        assert_same_csr((rp.cpu().numpy(), col.cpu().numpy(), val.cpu().numpy()),
                        oracle.multiply(M, "AA"), f"instance {b}")


# spans either side of each width (128 … 1024 columns) and beyond the last, B rows
# of less than half a warp, of a warp and of several segments
@pytest.mark.parametrize("bw,fill", [(8, 0.9), (16, 0.5), (31, 0.4), (32, 0.4), (33, 0.9),
                                     (63, 0.2), (64, 0.3), (65, 0.8), (127, 0.1), (128, 0.5),
                                     (129, 0.3), (255, 0.2), (256, 0.3), (257, 0.3), (300, 0.1)])
def test_narrow_rows(eng, bw, fill):
    A = csr.banded(3001, bw, fill, bw)
    labels = product(eng, A, "AA")
    if eng.binned:  # (at the edges of the matrix the widest bands have narrow rows too)
        assert any(x.startswith("num/narrow") for x in labels)
    product(eng, A, "AAt")


def test_narrow_rows_signed_zeros(eng):
    # every product a zero of either sign, or an underflow: all stay entries
    A = csr.banded(2000, 40, 0.4, 3)
    A.val = np.random.default_rng(4).choice([0.0, -0.0, 1e-200, -1e-200, 1.0], A.nnz)
    product(eng, A, "AA")
    product(eng, from_rows(3006, [[(i // 9) * 9 + 8 - i % 3] if i % 5 else [] for i in range(3000)],
                           5), "AAt")


def test_row_pointers_and_bins_of_many_tiles(eng):
    # rows of every kind next to one another, n over several scan tiles and binning
    # blocks and not a multiple of either
    rng = np.random.default_rng(15)
    n = 9001
    rows = []
    for i in range(n):
        kind = (i // 37) % 5
        if kind == 0:
            rows.append([j for j in (i - 70, i - 1, i, i + 1, i + 70) if 0 <= j < n])
        elif kind == 1:
            rows.append(i // 2 + rng.integers(0, 200, 30))
        elif kind == 2:
            rows.append(rng.integers(0, n, 25))
        elif kind == 3:
            rows.append([])
        else:
            rows.append(rng.integers(0, n, 300 if i % 50 == 0 else 3))
    A = from_rows(n, rows, 16)
    for task in ("AA", "AAt", "AAtS"):
        product(eng, A, task)


# runs of few entries a row: either side of what teams of one warp take in span
# (32,768 columns) and in room for their operands
@pytest.mark.parametrize("n,offsets,label", [
    (40001, [0, 16383], "num/runs1"), (40001, [0, 16384], "num/runs2"),
    (999, [0, 50, 100], "num/runs1"), (999, [0, 50, 100, 150], "num/runs2"),
    (999, list(range(8)), "num/runs1"), (999, list(range(9)), "num/runs2")])
def test_shifted_rows_short(n, offsets, label):
    from appt_spgemm_b200.engine import Engine
    with Engine("cuda:0", small_max_nnz=-1) as e:
        e.binned = True
        assert label in product(e, by_offsets(n, offsets, seed=n), "AA")


def test_prepass_of_short_rows():
    # few entries a row on average: rows on either side of what a thread, a warp and
    # a piece of a long row take, next to one another and to empty ones
    from appt_spgemm_b200.engine import Engine
    rng = np.random.default_rng(17)
    n = 9001
    rows = [np.arange(i, min(i + 3, n)) for i in range(n)]
    lengths = [0, 1, 3, 4, 5, 15, 16, 17, 31, 32, 33, 125, 126, 127, 255, 256, 257, 1023, 1024, 1025]
    for at, length in enumerate(lengths):
        for i in (at, 300 + 32 * at, n - 1 - at):
            rows[i] = rng.choice(n, length, replace=False)
        start = int(rng.integers(0, n - length - 40))
        for i in range(2000 + 40 * at, 2003 + 40 * at):  # shifted rows of this length
            rows[i] = start + i - 2000 - 40 * at + np.arange(length)
    A = from_rows(n, rows, 18)
    assert A.nnz <= 8 * n
    with Engine("cuda:0", small_max_nnz=-1) as e:
        e.binned = True
        product(e, A, "AA")
        product(e, A, "AAt")
