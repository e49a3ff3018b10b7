"""GPU cases at the edges of the row kernels' launches: several contexts at once,
launch shapes, scratch limits and special values, against the CPU oracle."""
import threading

import numpy as np
import pytest

import oracle
from appt_spgemm_b200 import csr
from parity import assert_same_csr

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def dev(A):
    from appt_spgemm_b200.engine import CsrDevice
    return CsrDevice.from_host(A, "cuda:0")


def kernels(eng, call):
    """The kernel labels of call()."""
    eng.profile_enable(True)
    eng.profile_reset()
    call()
    torch.cuda.synchronize()
    labels = set(eng.profile_read()["kernels"])
    eng.profile_enable(False)
    return labels


def in_threads(*bodies):
    """Runs the bodies at once, a thread each, and raises the first error."""
    errors, start = [], threading.Barrier(len(bodies))

    def run(body):
        try:
            start.wait()
            body()
        except Exception as e:  # noqa: BLE001 (reported below)
            errors.append(e)

    threads = [threading.Thread(target=run, args=(b,)) for b in bodies]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    if errors:
        raise errors[0]


def long_rows(n, rows, length, seed):
    """`rows` rows of `length` random columns, and as many that hold all of those."""
    rng = np.random.default_rng(seed)
    lists = [np.unique(rng.integers(2 * rows, n, length)) for _ in range(rows)]
    lists += [np.arange(rows)] * rows
    rp = np.zeros(n + 1, dtype=np.int32)
    rp[1:2 * rows + 1] = np.cumsum([len(x) for x in lists])
    rp[2 * rows + 1:] = rp[2 * rows]
    col = np.concatenate(lists).astype(np.int32)
    return csr.CsrHost(n, rp, col, rng.uniform(-1, 1, len(col)))


def test_heavy_rows_of_different_shapes_in_several_contexts():
    # a context per thread: panels of 256 columns beside panels of 1024, and bitmap
    # windows of 2^11 columns beside 2^20; the shared memory that one thread's launch
    # asks for must not limit another's
    from appt_spgemm_b200.engine import Engine
    binned = dict(small_max_nnz=-1)
    wide = dict(binned, force_heavy=1, heavy_split=1)
    jobs = [(long_rows(3000, 70, 300, 1), binned), (long_rows(65536, 70, 500, 2), binned),
            (long_rows(3000, 70, 300, 3), dict(wide, window_bits=1 << 11)),
            (long_rows(3000, 70, 300, 3), dict(wide, window_bits=1 << 20))]

    def body(A, cfg):
        def run():
            stream = torch.cuda.Stream()
            with torch.cuda.stream(stream), Engine("cuda:0", **cfg) as e:
                p = e.plan(dev(A), "AA")
                C = p.execute()
                for _ in range(1500):
                    p.execute(C)
                stream.synchronize()
                e.check_device_status()
                assert_same_csr(C.to_host(), oracle.multiply(A, "AA"), str(cfg))
                p.close()
        return run

    in_threads(*(body(*j) for j in jobs))


def most_entries(total, tail_rows, degree, seed):
    """A matrix of `total` entries on the device, whose last `tail_rows` rows are a
    random product of their own and whose other entries point at empty rows; with it
    those rows as a matrix of their own."""
    from appt_spgemm_b200.engine import CsrDevice
    n = 1 << 26
    tail = csr.uniform(tail_rows, degree, seed)
    first, end = 40, n - tail_rows           # the empty rows
    rest = total - tail.nnz
    counts = np.zeros(n, dtype=np.int64)
    counts[:rest // (end - first)] = end - first
    counts[rest // (end - first)] = rest % (end - first)
    counts[end:] = np.diff(tail.rowptr)
    rp = np.zeros(n + 1, dtype=np.int32)
    rp[1:] = np.cumsum(counts)
    col = torch.empty(total, dtype=torch.int32, device="cuda:0")
    for r in range(first):
        if counts[r]:
            col[rp[r]:rp[r + 1]] = torch.arange(first, first + int(counts[r]), dtype=torch.int32,
                                                device="cuda:0")
    col[rest:] = torch.from_numpy(tail.col + np.int32(end)).to("cuda:0")
    val = torch.zeros(total, dtype=torch.float64, device="cuda:0")
    val[rest:] = torch.from_numpy(tail.val).to("cuda:0")
    return CsrDevice(n, torch.from_numpy(rp).to("cuda:0"), col, val), tail


def needs_memory(bytes_):
    torch.cuda.empty_cache()
    if torch.cuda.mem_get_info()[0] < bytes_:
        pytest.skip("not enough device memory")


def check_last_rows(e, A, tail, label):
    C, end = e.multiply(A, "AA"), A.n - tail.n
    e.check_device_status()
    assert int(C.rowptr[end]) == 0
    assert_same_csr((C.rowptr[end:].cpu().numpy(), C.col.cpu().numpy() - end,
                     C.val.cpu().numpy()), oracle.multiply(tail, "AA"), label)


def test_searches_beyond_two_to_the_thirty_entries():
    # the middle of two positions above 2^30: panels that search for their slices
    # (the table of their bounds would be as large as C many times), and the
    # descriptors' look for each entry's mirror
    from appt_spgemm_b200.engine import Engine
    needs_memory(90 << 30)
    A, tail = most_entries((1 << 31) - (1 << 16), 3000, 90, seed=5)
    with Engine("cuda:0") as e:
        assert "num/panels" in kernels(e, lambda: check_last_rows(e, A, tail, "last rows"))
        d = e.describe(A)
        assert d["products_aa"] == int(np.diff(tail.rowptr)[tail.col].sum())
        mirrored = len(np.intersect1d(
            *(lambda r: (r * tail.n + tail.col, tail.col * tail.n + r))(
                np.repeat(np.arange(tail.n, dtype=np.int64), np.diff(tail.rowptr)))))
        assert abs(d["pattern_symmetry"] * A.nnz - mirrored) < 0.5


FORCED = dict(force_heavy=1, heavy_split=1)


# the last row, up to the last entry that 32-bit row pointers can count, through each
# row kernel: a step past its end must not wrap round
@pytest.mark.parametrize("tail_rows,degree,configs", [
    (12, 5, [{}]), (900, 60, [{}]), (3000, 9, [{}]),
    (1500, 40, [dict(heavy_split=1 << 30), dict(heavy_split=1 << 30, lanes_per_row=16)]),
    (3000, 60, [{}, FORCED, dict(FORCED, heavy_split=1 << 30), dict(FORCED, heavy_vcap=8192),
                dict(heavy_split=1, dense_max_words=2048)]),
    (3000, 400, [{}])])
def test_the_last_entries_of_a_full_matrix(tail_rows, degree, configs):
    from appt_spgemm_b200._capi import SpgemmError
    from appt_spgemm_b200.engine import Engine
    needs_memory(90 << 30)
    A, tail = most_entries((1 << 31) - 1, tail_rows, degree, seed=degree)
    for cfg in configs:
        with Engine("cuda:0", **cfg) as e:
            check_last_rows(e, A, tail, str(cfg))
    A.col[-1] = A.col[-2]  # not increasing
    with Engine("cuda:0") as e, pytest.raises(SpgemmError, match="strictly increase"):
        e.multiply(A, "AA")


def from_rows(n, rows, seed):
    rows = [np.unique(np.asarray(r, dtype=np.int64)) for r in rows]
    rp = np.zeros(n + 1, dtype=np.int32)
    rp[1:len(rows) + 1] = np.cumsum([len(r) for r in rows])
    rp[len(rows) + 1:] = rp[len(rows)]
    col = np.concatenate(rows).astype(np.int32)
    return csr.CsrHost(n, rp, col, np.random.default_rng(seed).uniform(-1, 1, len(col)))


def unknowns(A, k):
    """k unknowns per node of A's mesh: every entry a k x k block."""
    rows = []
    for i in range(A.n):
        c = A.col[A.rowptr[i]:A.rowptr[i + 1]].astype(np.int64)
        rows += [(c[:, None] * k + np.arange(k)).ravel()] * k
    return from_rows(A.n * k, rows, k)


def long_b_rows(n, rows, entries, length):
    """`rows` rows of `entries` entries, which point at 400 rows of `length`."""
    rng = np.random.default_rng(n + entries)
    lists = [rng.integers(400, n, length) for _ in range(400)]
    lists += [rng.choice(400, entries, replace=False) for _ in range(rows)]
    return from_rows(n, lists, 3)


def renumbered(A, window, seed):
    """A's nodes shuffled within windows of the order: an unstructured mesh's rows."""
    rng = np.random.default_rng(seed)
    q = np.lexsort((rng.random(A.n), np.arange(A.n) // window))
    to = np.empty(A.n, dtype=np.int64)
    to[q] = np.arange(A.n)
    rows = [None] * A.n
    for i in range(A.n):
        rows[to[i]] = to[A.col[A.rowptr[i]:A.rowptr[i + 1]]]
    return from_rows(A.n, rows, seed)


def arrowhead(n, width):
    rows = [np.concatenate([[0], np.arange(max(0, i - width), min(n, i + width + 1))])
            for i in range(n)]
    rows[0] = np.arange(0, n, 7)
    return from_rows(n, rows, 5)


# which rows are worth a panel: meshes with several unknowns per node keep their tables
# (one panel's products merge into few entries), as do long rows with few products per
# panel; random rows and hubs take panels, all of an arrowhead's
@pytest.mark.parametrize("A,panels,windows", [
    (lambda: unknowns(csr.laplace2d(60), 6), False, False),
    (lambda: unknowns(csr.laplace2d(40), 8), False, False),
    (lambda: unknowns(csr.stencil27(20, 1), 2), False, False),
    (lambda: unknowns(csr.stencil27(14, 1), 3), True, None),
    (lambda: csr.erdos_renyi(3000, 40.0, 1), True, None),
    (lambda: long_b_rows(200000, 500, 32, 500), False, None),
    (lambda: long_b_rows(200000, 500, 64, 800), True, None),
    (lambda: long_b_rows(50000, 500, 64, 100), True, None),
    (lambda: renumbered(csr.stencil27(24, 1), 64, 2), False, None),
    (lambda: csr.erdos_renyi(1100, 28.0, 1), True, None),
    (lambda: arrowhead(6000, 3), True, False)],
    ids=["grid6", "grid8", "cube2", "cube3", "random", "few-products", "many-products",
         "many-entries", "mesh", "random-small", "arrowhead"])
def test_rows_worth_a_panel(A, panels, windows):
    from appt_spgemm_b200.engine import Engine
    A = A()
    with Engine("cuda:0", small_max_nnz=-1) as e:
        for task in ("AA", "AAt"):
            got = []
            ran = kernels(e, lambda: got.append(e.multiply(dev(A), task)))
            e.check_device_status()
            assert_same_csr(got[0].to_host(), oracle.multiply(A, task), task)
            if task == "AA":
                assert ("num/panels" in ran) == panels, ran
                assert windows is None or ("num/heavy_w32" in ran) == windows, ran


def dense(n):
    return csr.CsrHost(n, (np.arange(n + 1) * n).astype(np.int32),
                       np.tile(np.arange(n, dtype=np.int32), n),
                       np.random.default_rng(n).uniform(-1, 1, n * n))


def test_marking_rows_that_merge():
    # rows whose products fall on a few columns time after time are marked with a look
    # before the atomic: no slower than their sums; rows either side of that line
    from appt_spgemm_b200.engine import Engine
    with Engine("cuda:0") as e:
        A = dev(dense(2000))
        for _ in range(2):
            e.profile_enable(True)
            e.profile_reset()
            e.multiply(A, "AA")
            torch.cuda.synchronize()
            ms = {k: v["ms"] for k, v in e.profile_read()["kernels"].items()}
        assert ms["sym/heavy"] < ms["num/panels"], ms
    with Engine("cuda:0", force_heavy=1) as e:
        for B in (dense(63), dense(64), dense(65), dense(300), csr.erdos_renyi(300, 140.0, 3)):
            C = e.multiply(dev(B), "AA")
            e.check_device_status()
            assert_same_csr(C.to_host(), oracle.multiply(B, "AA"), str(B.n))


def test_prepass_of_longer_rows_together():
    # 2,000 rows of 64 entries next to one another among rows of two: the pre-pass takes
    # no longer than with the same rows spread over the matrix
    from appt_spgemm_b200.engine import Engine
    n, step = 100000, 47
    rng = np.random.default_rng(1)
    longer = [np.unique(rng.integers(0, n, 64)) for _ in range(2000)]
    took = {}
    with Engine("cuda:0", small_max_nnz=-1) as e:
        for name, at in (("together", np.arange(400, 2400)), ("spread", np.arange(2000) * step)):
            rows = [[i, (i * 7) % n] for i in range(n)]
            for i, r in zip(at, longer):
                rows[i] = r
            A = from_rows(n, rows, 2)
            C = e.multiply(dev(A), "AA")
            assert_same_csr(C.to_host(), oracle.multiply(A, "AA"), name)
            d = dev(A)
            e.profile_enable(True)
            times = []
            for _ in range(9):
                e.profile_reset()
                e.multiply(d, "AA")
                torch.cuda.synchronize()
                times.append(e.profile_read()["kernels"]["plan/prepass"]["ms"])
            e.profile_enable(False)
            took[name] = np.median(times)
        e.check_device_status()
    assert took["together"] < 1.7 * took["spread"], took


def test_symmetric_small_plan_gathers_its_transpose():
    # a plan of the symmetric variant executed again: the values of A^T by one launch
    # (its pattern is A's), then the product; an unsymmetric one transposes
    from appt_spgemm_b200.engine import Engine
    sym, unsym = csr.laplace2d(50), csr.erdos_renyi(900, 5.0, 3)
    with Engine("cuda:0") as e:
        launches = {}
        for name, A in (("sym", sym), ("unsym", unsym)):
            A.val = np.random.default_rng(4).uniform(-1, 1, A.nnz)
            d = dev(A)
            p = e.plan(d, "AAtS")
            assert p.info["symmetric_pattern"] == (name == "sym")
            C = p.execute()
            d.val.copy_(torch.from_numpy(A.val[::-1].copy()))  # other values, same pattern
            e.profile_reset()
            p.execute(C)
            launches[name] = e.profile_read()["launches"]
            e.check_device_status()
            B = csr.CsrHost(A.n, A.rowptr, A.col, A.val[::-1].copy())
            assert_same_csr(C.to_host(), oracle.multiply(B, "AAtS"), name)
            p.close()
    assert launches["sym"] == 2 < launches["unsym"], launches


def table_bytes(n):
    return 4 * n * (((n - 1) >> 10) + 2)


# the table of the panels' slice bounds, an int per row of B and panel of 1024 columns:
# taken where its bounds are read often, not for a few rows among many
@pytest.mark.parametrize("n,rows,table", [(60000, 2, False), (60000, 2000, True)])
def test_panel_table_only_where_it_is_used(n, rows, table):
    from appt_spgemm_b200.engine import Engine
    A = long_b_rows(n, rows, 40, 800)
    with Engine("cuda:0", small_max_nnz=-1) as e:
        p = e.plan(dev(A), "AA")
        assert (p.info["exec_workspace_bytes"] >= table_bytes(n)) == table, p.info
        got = []
        assert "num/panels" in kernels(e, lambda: got.append(p.execute()))
        e.check_device_status()
        assert_same_csr(got[0].to_host(), oracle.multiply(A, "AA"), str(rows))
        p.close()


def test_panels_without_memory_for_their_table():
    # the table is taken for speed alone: an execute that cannot have it searches
    from appt_spgemm_b200.engine import Engine
    A = long_b_rows(120000, 1000, 60, 800)
    ref = oracle.multiply(A, "AA")
    torch.cuda.empty_cache()
    with Engine("cuda:0", small_max_nnz=-1, pool_release_bytes=1) as e:
        p = e.plan(dev(A), "AA")
        nnz = int(p.info["nnz_c"])
        assert p.info["exec_workspace_bytes"] >= table_bytes(A.n) > 50 << 20
        from appt_spgemm_b200.engine import CsrResult
        C = CsrResult(A.n, nnz, torch.zeros(A.n + 1, dtype=torch.int64, device="cuda:0"),
                      torch.zeros(nnz, dtype=torch.int32, device="cuda:0"),
                      torch.zeros(nnz, dtype=torch.float64, device="cuda:0"))
        torch.cuda.synchronize()
        hog, chunk = [], 1 << 34
        while chunk >= 1 << 21:  # the rest of the memory, down to a few MB
            try:
                hog.append(torch.empty(chunk, dtype=torch.uint8, device="cuda:0"))
            except torch.OutOfMemoryError:
                chunk >>= 1
        try:
            p.execute(C)
            torch.cuda.synchronize()
        finally:
            hog.clear()
            torch.cuda.empty_cache()
        e.check_device_status()
        assert_same_csr(C.to_host(), ref, "without the table")
        p.close()


def test_server_runs_what_fits_without_the_table():
    from appt_spgemm_b200.engine import Engine, Server
    A = long_b_rows(60000, 2000, 40, 800)
    d = dev(A)
    with Engine("cuda:0") as e:
        p = e.plan(d, "AA")
        need = sum(p.info[k] for k in ("workspace_bytes", "exec_workspace_bytes", "output_bytes"))
        p.close()
    with Server(workers=1, memory_budget_bytes=need - table_bytes(A.n) // 2, batch_rows=1) as srv:
        rid = srv.submit(d, "AA")
        info = srv.wait(rid)
        assert info["status"] == 0
        assert_same_csr(srv.result(rid).to_host(), oracle.multiply(A, "AA"), "served")
        srv.release(rid)
        st = srv.stats()
        assert st["rejected"] == 0 and st["peak_held_bytes"] <= st["budget_bytes"]


def test_panels_leave_their_sms():
    # grid_sms: CTAs leave after their share of the work, so that a small product on a
    # stream of higher priority is done long before a large one that started first
    from appt_spgemm_b200.engine import Engine
    small, large = dev(csr.laplace2d(64)), dev(csr.erdos_renyi(40000, 150.0, 1))
    low, high = torch.cuda.Stream(priority=0), torch.cuda.Stream(priority=-5)
    with Engine("cuda:0", grid_sms=1 << 16) as el, Engine("cuda:0") as es:
        A = csr.erdos_renyi(6000, 80.0, 2)
        C = el.multiply(dev(A), "AA")  # the same values with a warp per panel
        assert_same_csr(C.to_host(), oracle.multiply(A, "AA"), "retiring")
        p = el.plan(large, "AA", stream=low)
        C = p.execute(stream=low)
        es.multiply(small, "AA", stream=high)
        torch.cuda.synchronize()
        start, mid, end = (torch.cuda.Event(enable_timing=True) for _ in range(3))
        start.record(low)
        assert "num/panels" in kernels(el, lambda: p.execute(C, stream=low))
        torch.cuda.synchronize()
        start.record(low)
        p.execute(C, stream=low)
        end.record(low)
        es.multiply(small, "AA", stream=high)
        mid.record(high)
        torch.cuda.synchronize()
        el.check_device_status()
        es.check_device_status()
        p.close()
        assert start.elapsed_time(mid) < 0.5 * start.elapsed_time(end), (
            start.elapsed_time(mid), start.elapsed_time(end))


@pytest.mark.parametrize("split,panels", [(0, True), (128, True), (127, False), (1 << 30, False)])
def test_the_default_split_written_out(split, panels):
    from appt_spgemm_b200.engine import Engine
    A = csr.rmat(12, 16, seed=2)
    with Engine("cuda:0", heavy_split=split) as e:
        got = []
        ran = kernels(e, lambda: got.append(e.multiply(dev(A), "AA")))
        assert ("num/panels" in ran) == panels, ran
        assert_same_csr(got[0].to_host(), oracle.multiply(A, "AA"), str(split))


# infinities, NaN and both zeros through each row kernel: what a place or a slot holds
# to say that it has no entry must not be taken for a value, nor the reverse
@pytest.mark.parametrize("A,kernel", [
    (lambda: csr.erdos_renyi(3000, 45.0, 1), "num/panels"),
    (lambda: csr.banded(3000, 40, 0.4, 2), "num/narrow"),
    (lambda: csr.uniform(20011, 20, 3), "num/sort"),
    (lambda: csr.stencil27(14, 4), "num/runs"),
    (lambda: csr.uniform(3000, 2, 5), "num/bin")],
    ids=["panels", "narrow", "sorted", "runs", "tables"])
def test_special_values(A, kernel):
    from appt_spgemm_b200.engine import Engine
    A = A()
    A.val = np.random.default_rng(6).choice(
        [0.0, -0.0, 1.0, -1.0, 1e308, -1e308, 5e-324, np.inf, -np.inf, np.nan], A.nnz,
        p=[0.2, 0.2, 0.2, 0.2, 0.05, 0.05, 0.05, 0.02, 0.02, 0.01])
    with Engine("cuda:0", small_max_nnz=-1) as e:
        for task in ("AA", "AAt", "AAtS"):
            got = []
            ran = kernels(e, lambda: got.append(e.multiply(dev(A), task)))
            assert task != "AA" or any(x.startswith(kernel) for x in ran), ran
            e.check_device_status()
            rp, ci, cx = got[0].to_host()
            orp, oci, ocx = oracle.multiply(A, task)
            assert np.array_equal(rp, orp) and np.array_equal(ci, oci), task
            nan = np.isnan(ocx)  # (which NaN is the hardware's choice)
            assert nan.any() and np.isinf(ocx).any() and np.array_equal(np.isnan(cx), nan), task
            assert np.array_equal(cx[~nan].view(np.int64), ocx[~nan].view(np.int64)), task


def test_knobs_with_many_runs_per_bin():
    # concurrent bins and retiring CTAs over thousands of runs, and panels beside them
    from appt_spgemm_b200.engine import Engine
    grid, side = csr.laplace2d(220), csr.stencil27(26, 2)
    for cfg in (dict(bin_streams=4), dict(grid_sms=1 << 16), dict(bin_streams=4, grid_sms=1 << 16)):
        with Engine("cuda:0", small_max_nnz=-1, **cfg) as e:
            for A in (grid, side, csr.rmat(12, 16, seed=4)):
                for task in ("AA", "AAt"):
                    C = e.multiply(dev(A), task)
                    e.check_device_status()
                    assert_same_csr(C.to_host(), oracle.multiply(A, task), str(cfg))


# A·Aᵀ plans that cannot be small (a row of it has the squared mean degree of products or
# more, against 1536) are not tried as such; either side of the line
@pytest.mark.parametrize("degree,tried", [(39, True), (40, False), (60, False)])
def test_hopeless_small_plans_are_not_tried(degree, tried):
    from appt_spgemm_b200.engine import Engine
    A = csr.uniform(2000, degree, degree)
    with Engine("cuda:0") as e:
        for task in ("AAt", "AAtS"):
            got = []
            ran = kernels(e, lambda: got.append(e.multiply(dev(A), task)))
            assert ("sym/small" in ran) == tried, ran
            e.check_device_status()
            assert_same_csr(got[0].to_host(), oracle.multiply(A, task), task)


def test_meshes_of_a_batch_keep_their_tables():
    # rows of one or two panels: in a batch there are enough of them to fill the GPU, and
    # tables serve a renumbered mesh's rows better
    from appt_spgemm_b200.engine import Engine
    As = [renumbered(csr.stencil27(16, 1), 64, i) for i in range(4)]
    with Engine("cuda:0") as e:
        got = []
        ran = kernels(e, lambda: got.append(e.multiply_batched([dev(A) for A in As], "AA")))
        assert "sym/heavy" not in ran and "num/panels" not in ran, ran
        for b, A in enumerate(As):
            rp, col, val = got[0].instance(b)
            assert_same_csr((rp.cpu().numpy(), col.cpu().numpy(), val.cpu().numpy()),
                            oracle.multiply(A, "AA"), f"instance {b}")


# whole runs of shifted rows: shorter ones are hashed.  (Grid lines of a power of two
# lie whole in the blocks of 256 rows that runs are looked for in; of a line that a
# block cuts, parts of 8 rows are runs too.)
@pytest.mark.parametrize("grid,count,taken", [
    (lambda i: csr.stencil27(16, i), 8, False), (lambda i: csr.stencil27(32, i), 2, True),
    (lambda i: csr.laplace2d(16), 90, False), (lambda i: csr.laplace2d(32), 30, True),
    (lambda i: csr.laplace2d(27), 30, True)],
    ids=["12", "28", "12-short", "28-short", "cut"])
def test_whole_runs_worth_their_setup(grid, count, taken):
    from appt_spgemm_b200.engine import Engine
    As = [grid(i) for i in range(count)]
    for i, A in enumerate(As):
        A.val = np.random.default_rng(i).uniform(-1, 1, A.nnz)
    with Engine("cuda:0") as e:
        for task in ("AA", "AAt"):
            got = []
            ran = kernels(e, lambda: got.append(e.multiply_batched([dev(A) for A in As], task)))
            e.check_device_status()
            for b, A in enumerate(As):
                rp, col, val = got[0].instance(b)
                assert_same_csr((rp.cpu().numpy(), col.cpu().numpy(), val.cpu().numpy()),
                                oracle.multiply(A, task), f"instance {b}")
            assert any(x.startswith("num/runs") for x in ran) == taken, ran


def blocks(n, b):
    """Dense blocks of b on the diagonal."""
    k = n // b
    col = np.repeat(np.arange(k) * b, b * b).reshape(k, b, b) + np.arange(b)
    return csr.CsrHost(k * b, (np.arange(k * b + 1) * b).astype(np.int32),
                       col.ravel().astype(np.int32),
                       np.random.default_rng(b).uniform(-1, 1, col.size))


# rows of a few columns: tables unless B's rows fill the lanes that would sum them
@pytest.mark.parametrize("b,narrow", [(7, False), (8, False), (9, True), (10, True), (11, False),
                                      (16, False), (17, True), (33, True)])
def test_narrow_rows_of_few_columns(b, narrow):
    from appt_spgemm_b200.engine import Engine
    A = blocks(3000, b)
    for cfg in (dict(), dict(small_max_nnz=-1)):
        with Engine("cuda:0", **cfg) as e:
            for task in ("AA", "AAt"):
                got = []
                ran = kernels(e, lambda: got.append(e.multiply(dev(A), task)))
                assert not cfg or any(x.startswith("num/narrow") for x in ran) == narrow, ran
                e.check_device_status()
                assert_same_csr(got[0].to_host(), oracle.multiply(A, task), task)


def communities(n, size, inside, seed):
    """Rows of `inside` columns of their own community and one of anywhere."""
    rng = np.random.default_rng(seed)
    return from_rows(n, [np.concatenate([i // size * size + rng.integers(0, size, inside),
                                         rng.integers(0, n, 1)]) for i in range(n)], seed)


# sorted rows are hashed where their columns crowd together: communities of a hundredth of
# the columns and less, one readback or two; not those of a tenth, nor a random graph
@pytest.mark.parametrize("A,crowded", [
    (lambda: communities(40000, 200, 12, 1), True), (lambda: communities(40000, 400, 20, 2), True),
    (lambda: communities(40000, 4000, 20, 3), False),
    (lambda: csr.erdos_renyi(40000, 16.0, 4), False)],
    ids=["200", "400", "4000", "random"])
def test_crowded_rows_are_not_sorted(A, crowded):
    from appt_spgemm_b200.engine import Engine
    A = A()
    for cfg in (dict(small_max_nnz=-1), dict()):
        with Engine("cuda:0", **cfg) as e:
            for task in ("AA", "AAt", "AAtS"):
                got = []
                ran = kernels(e, lambda: got.append(e.multiply(dev(A), task)))
                if cfg:
                    assert any(x.startswith("num/sort") for x in ran) != crowded, (task, ran)
                e.check_device_status()
                assert_same_csr(got[0].to_host(), oracle.multiply(A, task), task)
