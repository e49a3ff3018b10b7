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
