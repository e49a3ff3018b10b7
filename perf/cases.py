"""Performance cases: the products that users of the engine ask for, through its
public Python entry points (Engine.multiply, Engine.multiply_batched, and the
replay of a captured batched execute), over the matrix families and sizes of
the benchmark workloads.

A case is a dict of plain values:
  family  laplace (2-D 5-point grid), stencil (3-D 27-point grid), banded
          (random in-band fill), er (Erdős–Rényi), rmat (power law), or mix
          (a batch, alternately banded and er, sizes log-uniform)
  task    AA, AAt or AAtS (A·Aᵀ through the symmetric Gram path)
  call    multiply (plan + execute with a newly allocated C, one call),
          batched (the same for many matrices in one call), replay (a CUDA
          graph of a batched plan's execute, relaunched)
and the family's sizes, with the seed of a random pattern.
"""
import functools
import math

import numpy as np
import torch

from appt_spgemm_b200 import csr
from appt_spgemm_b200.engine import CsrDevice, Engine


def listed():
    return [
        # One small sparse operator per call (setup of a 2-D multigrid level,
        # one request of a serving stream): launch and host latency.
        {"name": "laplace_64_AA", "family": "laplace", "side": 64, "task": "AA",
         "call": "multiply"},
        {"name": "laplace_64_AAt", "family": "laplace", "side": 64, "task": "AAt",
         "call": "multiply"},
        # A large 2-D operator with an odd side: few products per row, a million rows.
        {"name": "laplace_1009_AA", "family": "laplace", "side": 1009, "task": "AA",
         "call": "multiply"},
        # The 3-D FEM-like operator: the headline product, its A·Aᵀ (structurally
        # symmetric, numerically not) and the Gram form, at full and ragged sides.
        {"name": "stencil_96_AA", "family": "stencil", "side": 96, "task": "AA",
         "call": "multiply"},
        {"name": "stencil_61_AAt", "family": "stencil", "side": 61, "task": "AAt",
         "call": "multiply"},
        {"name": "stencil_47_AAtS", "family": "stencil", "side": 47, "task": "AAtS",
         "call": "multiply"},
        # One wide random band: many products per output entry.
        {"name": "banded_50021_AA", "family": "banded", "n": 50021, "bw": 48, "pattern": 3,
         "task": "AA", "call": "multiply"},
        # Random graphs, whose products hardly merge: a mid-sized one, and a
        # larger one against its transpose (unsymmetric pattern).
        {"name": "er_40009_AA", "family": "er", "n": 40009, "degree": 20.0, "pattern": 3,
         "task": "AA", "call": "multiply"},
        {"name": "er_262147_AAt", "family": "er", "n": 262147, "degree": 9.0, "pattern": 3,
         "task": "AAt", "call": "multiply"},
        # A power-law graph: hub rows with up to millions of products.
        {"name": "rmat_16_AA", "family": "rmat", "scale": 16, "pattern": 3, "task": "AA",
         "call": "multiply"},
        # Many matrices of uneven size at once, planned and multiplied in one
        # call, and with the plan kept and its execute replayed on the values at hand.
        {"name": "batch_48_AA", "family": "mix", "count": 48, "n_min": 1000, "n_max": 64000,
         "pattern": 4, "task": "AA", "call": "batched"},
        {"name": "replay_24_AA", "family": "mix", "count": 24, "n_min": 1000, "n_max": 64000,
         "pattern": 4, "task": "AA", "call": "replay"},
    ]


def draw(rng):
    def logint(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["laplace", "stencil", "banded", "er", "er_large", "rmat", "batched",
                       "replay"])
    task = rng.choice(["AA", "AAt", "AAtS"])
    pattern = rng.randint(1, 1 << 30)
    if kind == "laplace":
        return {"family": "laplace", "side": logint(16, 1100), "task": task, "call": "multiply"}
    if kind == "stencil":
        return {"family": "stencil", "side": logint(6, 80), "task": task, "call": "multiply"}
    if kind == "banded":
        return {"family": "banded", "n": logint(1000, 64000), "bw": rng.randint(3, 64),
                "pattern": pattern, "task": task, "call": "multiply"}
    if kind == "er":
        return {"family": "er", "n": logint(1000, 64000), "degree": rng.uniform(4.0, 32.0),
                "pattern": pattern, "task": task, "call": "multiply"}
    if kind == "er_large":
        return {"family": "er", "n": logint(64000, 400000), "degree": rng.uniform(4.0, 12.0),
                "pattern": pattern, "task": task, "call": "multiply"}
    if kind == "rmat":
        return {"family": "rmat", "scale": rng.randint(10, 15), "pattern": pattern, "task": task,
                "call": "multiply"}
    return {"family": "mix", "count": logint(3, 40), "n_min": 1000, "n_max": 32000,
            "pattern": pattern, "call": kind,
            "task": "AA" if kind == "replay" else rng.choice(["AA", "AAt"])}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _matrices(case, seed):
    """The case's matrices on the host (one, or the batch's).  The case fixes the
    pattern (`pattern` seeds the random ones), as the mesh or the graph of a user's
    program does; the seed draws the values."""
    fam, pattern = case["family"], case.get("pattern", 0)
    if fam == "laplace":
        As = [csr.laplace2d(case["side"])]
    elif fam == "stencil":
        As = [csr.stencil27(case["side"], seed=1)]
    elif fam == "banded":
        As = [csr.banded(case["n"], case["bw"], 0.3, pattern)]
    elif fam == "er":
        As = [csr.erdos_renyi(case["n"], case["degree"], pattern)]
    elif fam == "rmat":
        As = [csr.rmat(case["scale"], 16, seed=pattern)]
    else:
        As, _ = csr.batch_mix(case["count"], seed=pattern, n_min=case["n_min"],
                              n_max=case["n_max"])
    rng = np.random.default_rng(seed)
    for A in As:
        if fam == "laplace":  # a variable-coefficient operator: 4 and -1, scaled per entry
            A.val = A.val * rng.uniform(0.5, 1.5, A.nnz)
        else:
            A.val = rng.uniform(0.0 if fam == "rmat" else -1.0, 1.0, A.nnz)
    return As


_engine = None


def _shared_engine():
    """The one engine context that a program keeps for all of its products."""
    global _engine
    if _engine is None:
        _engine = Engine("cuda:0")
    return _engine


def prepare(case, seed):
    eng = _shared_engine()
    As = [CsrDevice.from_host(A, "cuda:0") for A in _matrices(case, seed)]
    state = {"call": case["call"], "task": case["task"], "engine": eng, "A": As}
    if case["call"] == "replay":
        plan = eng.plan_batched(As, case["task"])
        out = plan.execute()
        state["offsets"] = plan.offsets()
        stream = torch.cuda.Stream()
        stream.wait_stream(torch.cuda.current_stream())
        state["graph"] = plan.capture_graph(out, stream)
        torch.cuda.current_stream().wait_stream(stream)
    return state


def run(state):
    if state["call"] == "multiply":
        C = state["engine"].multiply(state["A"][0], state["task"])
        return {"rowptr": C.rowptr, "col": C.col, "val": C.val}
    if state["call"] == "batched":
        R = state["engine"].multiply_batched(state["A"], state["task"])
        return {"rowptr": R.C.rowptr, "col": R.C.col, "val": R.C.val,
                "row_off": R.row_off, "nnz_off": R.nnz_off}
    C = state["graph"].launch()
    row_off, nnz_off = state["offsets"]
    return {"rowptr": C.rowptr, "col": C.col, "val": C.val,
            "row_off": row_off, "nnz_off": nnz_off}


# ---------------------------------------------------------------------------
# what the product cannot do without, and its values in 64 bits
# ---------------------------------------------------------------------------
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _chunks(A, B, max_products):
    """Yields (first row, end row, sorted keys row·n+col, products in key order)
    of C = A·B by expanding the rows' products, a bounded number at a time."""
    dev = _device()
    n = A.n
    arp, ac, av = (torch.from_numpy(x).to(dev) for x in (A.rowptr, A.col, A.val))
    brp, bc, bv = (torch.from_numpy(x).to(dev) for x in (B.rowptr, B.col, B.val))
    arp, ac, brp, bc = arp.long(), ac.long(), brp.long(), bc.long()
    blen = brp[1:] - brp[:-1]
    per_entry = blen[ac]
    upto = torch.zeros(A.nnz + 1, dtype=torch.int64, device=dev)
    torch.cumsum(per_entry, 0, out=upto[1:])
    row_upto = upto[arp].cpu().numpy()
    arow = torch.repeat_interleave(torch.arange(n, device=dev), arp[1:] - arp[:-1])
    r0 = 0
    while r0 < n:
        r1 = int(np.searchsorted(row_upto, row_upto[r0] + max_products, side="right")) - 1
        r1 = min(n, max(r0 + 1, r1))
        e0, e1 = int(arp[r0]), int(arp[r1])
        cnt = per_entry[e0:e1]
        entry = torch.repeat_interleave(torch.arange(e0, e1, device=dev), cnt)
        within = torch.arange(entry.numel(), device=dev) + (upto[e0] - upto[entry])
        src = brp[ac[entry]] + within
        key = arow[entry] * n + bc[src]
        prod = av[entry] * bv[src]
        key, order = torch.sort(key, stable=True)
        yield r0, r1, key, prod[order]
        r0 = r1


def _product(case, A, values=True, max_products=1 << 26):
    """(rowptr, col, val) of the case's product of one matrix, and its products."""
    B = A if case["task"] == "AA" else A.transpose()
    counts = np.zeros(A.n, dtype=np.int64)
    cols, vals, products = [], [], 0
    for r0, r1, key, prod in _chunks(A, B, max_products):
        products += key.numel()
        uniq, inverse = torch.unique_consecutive(key, return_inverse=True)
        rows = torch.div(uniq, A.n, rounding_mode="floor")
        counts[r0:r1] = torch.bincount(rows - r0, minlength=r1 - r0).cpu().numpy()
        if values:
            out = torch.zeros(uniq.numel(), dtype=torch.float64, device=key.device)
            out.index_add_(0, inverse, prod)
            vals.append(out.cpu().numpy())
            cols.append((uniq - rows * A.n).to(torch.int32).cpu().numpy())
    rowptr = np.zeros(A.n + 1, dtype=np.int64)
    np.cumsum(counts, out=rowptr[1:])
    cat = (lambda x, t: np.concatenate(x) if x else np.zeros(0, t))
    return rowptr, cat(cols, np.int32), cat(vals, np.float64), products


@functools.lru_cache(maxsize=None)
def _work(key):
    case = dict(key)
    nbytes = flops = 0
    for A in _matrices(case, 1):
        rowptr, _, _, products = _product(case, A, values=False)
        nbytes += 4 * (A.n + 1) + 12 * A.nnz + 8 * (A.n + 1) + 12 * int(rowptr[-1])
        flops += 2 * products
    return nbytes, flops


def work(case):
    """A read once and C written once (int32 indices, int64 row pointers, 64-bit
    values); a multiply and an add per product."""
    nbytes, flops = _work(tuple(sorted((k, v) for k, v in case.items() if k != "name")))
    return {"bytes": nbytes, "flops": flops}


def exact(case, seed):
    parts = [_product(case, A)[:3] for A in _matrices(case, seed)]
    if case["call"] == "multiply":
        rowptr, col, val = parts[0]
        return {"rowptr": rowptr, "col": col, "val": val}
    row_off = np.cumsum([0] + [p[0].size - 1 for p in parts]).astype(np.int64)
    nnz_off = np.cumsum([0] + [p[1].size for p in parts]).astype(np.int64)
    rowptr = np.concatenate([p[0][:-1] + o for p, o in zip(parts, nnz_off)] + [nnz_off[-1:]])
    return {"rowptr": rowptr, "col": np.concatenate([p[1] for p in parts]),
            "val": np.concatenate([p[2] for p in parts]),
            "row_off": row_off, "nnz_off": nnz_off}
