"""Performance cases of the library: what its users call, over the sizes they call it with.

Every case goes through the public entry points (the C ABI, by the thin wrappers of
libxstream_b200.acc where there is one) on device-resident data and a stream of the library, as
DBCSR, CP2K's DBM or a dense FP64 caller drives it. Kinds of work:

  stack        one libsmm_acc_process call: C[c] += A[a] * B[b] over a stack of S triples
  dbm          the same multiplication as 6-int DBM task records with a factor alpha
  batch        all stacks of one mixed-shape multiplication in one libxstream_b200_process_batch call
  multiply     a DBCSR-like multiplication from start to end: block norms, B upload and transpose,
               cleared C, several stacks
  ozaki_stack  the int8 tensor-core form of the stack path
  dgemm, ozaki1, ozaki2   dense FP64 GEMM: plain, int8 slices (scheme 1), int8 residues (scheme 2)

Calls that accumulate (C += ...) do so from pass to pass, as repeated calls on one C pool do.
"""
from __future__ import annotations

import ctypes
import math

import torch

from libxstream_b200 import StackDesc, acc, check, lib

# block sizes of the mixed-shape workload and of the published single-shape results
BLOCK_SIZES = (4, 5, 9, 13, 16, 22, 23, 26, 32, 45, 64)
MAX_KERNEL_DIM = 80
LARGEST = 64 * 64 * 64 * 200000  # m*n*k*S of the largest stack


# ------------------------------------------------------------------------------------- the cases

def listed() -> list[dict]:
    return [
        # A stack that was flushed early or belongs to a thin matrix: a few hundred blocks, where the
        # latency of the call counts.
        {"name": "stack_small", "kind": "stack", "m": 13, "n": 13, "k": 13, "S": 400, "zipf": 0.0, "grouped": True,
         "spread": 0},
        # Minimal basis sets: tiny blocks, many of them.
        {"name": "stack_tiny_blocks", "kind": "stack", "m": 5, "n": 5, "k": 5, "S": 100000, "zipf": 1.1, "grouped": False,
         "spread": 0},
        # The headline: water in a double-zeta basis, 23 x 23 x 23, one full stack of 30000.
        {"name": "stack_23", "kind": "stack", "m": 23, "n": 23, "k": 23, "S": 30000, "zipf": 1.1, "grouped": False,
         "spread": 0},
        # Several atomic kinds: odd rectangular blocks with no common factor.
        {"name": "stack_ragged", "kind": "stack", "m": 17, "n": 29, "k": 11, "S": 20000, "zipf": 1.1, "grouped": False,
         "spread": 0},
        # Larger basis, full stack, entries over 40 binary orders, in the order of the C blocks.
        {"name": "stack_45", "kind": "stack", "m": 45, "n": 45, "k": 45, "S": 30000, "zipf": 1.1, "grouped": True,
         "spread": 20},
        # The largest blocks and the longest stack in use.
        {"name": "stack_64_large", "kind": "stack", "m": 64, "n": 64, "k": 64, "S": 200000, "zipf": 1.1, "grouped": False,
         "spread": 20},
        # One multiplication of a matrix with mixed blocks: twelve stacks from hundreds to 10^5 triples.
        {"name": "batch_mixed", "kind": "batch", "stacks": 12, "smin": 100, "smax": 200000, "total": 186000, "pick": 25071975},
        # One multiplication from start to end: norms for the filter, B brought in and transposed, C
        # cleared, four stacks that share the pools.
        {"name": "multiply_22", "kind": "multiply", "m": 22, "n": 22, "k": 22, "S": 15000, "stacks": 4, "nblocks": 8192},
        # The int8 form of the stack path on entries of widely spread magnitude.
        {"name": "ozaki_stack_64", "kind": "ozaki_stack", "m": 64, "n": 64, "k": 64, "S": 30000, "slices": 7, "trim": 6},
        # Dense FP64 products: plain, by slices, by residues.
        {"name": "dgemm_2048", "kind": "dgemm", "M": 2048, "N": 2048, "K": 2048, "beta": 0.0},
        {"name": "ozaki1_4096", "kind": "ozaki1", "M": 4096, "N": 4096, "K": 4096, "ta": "N", "tb": "N", "slices": 7,
         "trim": 6, "beta": 0.0},
        {"name": "ozaki2_4096", "kind": "ozaki2", "M": 4096, "N": 4096, "K": 4096, "ta": "N", "tb": "N", "moduli": 0,
         "beta": 0.0},
    ]


def _logint(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _block(rng) -> int:
    """A block size: one in practical use, or any up to the largest kernel's."""
    return rng.choice(BLOCK_SIZES) if rng.random() < 0.5 else rng.randint(3, 72)


def draw(rng) -> dict:
    kind = rng.choice(("stack",) * 8 + ("dbm", "batch", "batch", "multiply", "ozaki_stack", "dgemm", "ozaki1", "ozaki2", "ozaki2"))
    if kind in ("stack", "dbm"):
        square = rng.random() < 0.4
        m, n, k = (_block(rng),) * 3 if square else (_block(rng), _block(rng), _block(rng))
        S = min(_logint(rng, 200, 200000), LARGEST // (m * n * max(k, 16)))
        case = {"kind": kind, "m": m, "n": n, "k": k, "S": S, "zipf": rng.choice((0.0, 1.1)), "grouped": rng.random() < 0.5}
        if kind == "stack":
            return {**case, "spread": rng.choice((0, 20))}
        return {**case, "alpha": round(rng.uniform(-2.0, 2.0), 3)}
    if kind == "batch":
        return {"kind": kind, "stacks": rng.randint(2, 16), "smin": 100, "smax": 200000, "total": _logint(rng, 5000, 400000),
                "pick": rng.randrange(1 << 30)}
    if kind == "multiply":
        m, n, k = _block(rng) % 33 + 3, _block(rng) % 33 + 3, _block(rng) % 33 + 3
        return {"kind": kind, "m": m, "n": n, "k": k, "S": _logint(rng, 500, 30000), "stacks": rng.randint(1, 6),
                "nblocks": _logint(rng, 256, 16384)}
    if kind == "ozaki_stack":
        m, n, k = rng.randint(16, 64), rng.randint(16, 64), rng.randint(16, 64)
        slices = rng.randint(5, 8)
        return {"kind": kind, "m": m, "n": n, "k": k, "S": _logint(rng, 500, 30000), "slices": slices, "trim": slices - 1}
    M, N, K = (_logint(rng, 200, 3000 if kind == "dgemm" else 4096) for _ in range(3))
    if kind == "dgemm":
        return {"kind": kind, "M": M, "N": N, "K": K, "beta": rng.choice((0.0, 1.0))}
    case = {"kind": kind, "M": M, "N": N, "K": K, "ta": rng.choice("NT"), "tb": rng.choice("NT"), "beta": rng.choice((0.0, 1.0))}
    if kind == "ozaki1":
        slices = rng.randint(5, 8)
        return {**case, "slices": slices, "trim": slices - 1}
    return {**case, "moduli": rng.choice((0, 14))}


# --------------------------------------------------------------------------- what a program keeps

class Buf:
    """A device buffer of the caller's, as the wrappers of libxstream_b200.acc take it."""

    def __init__(self, t: torch.Tensor):
        self.t = t
        self.ptr = t.data_ptr()
        self.nbytes = t.numel() * t.element_size()


_stream = None


def _the_stream() -> acc.Stream:
    global _stream
    if _stream is None:
        acc.init()
        _stream = acc.Stream("perf")
    return _stream


def _gen(seed: int) -> torch.Generator:
    return torch.Generator(device="cuda").manual_seed(seed)


def _values(g, count: int, spread: int = 0) -> torch.Tensor:
    """Uniform in [-1, 1), or mantissa U[1, 2) times 2^e with e uniform in [-spread, spread]."""
    u = torch.rand(count, generator=g, device="cuda", dtype=torch.float64)
    if spread == 0:
        return u * 2.0 - 1.0
    e = torch.randint(-spread, spread + 1, (count,), generator=g, device="cuda")
    sign = torch.randint(0, 2, (count,), generator=g, device="cuda") * 2 - 1
    return torch.ldexp((u + 1.0) * sign, e)


def _blocks(S: int) -> tuple[int, int]:
    """Blocks in the A and B pools, and in the C pool, for a stack of S triples."""
    return min(8192, max(16, S // 8)), min(2048, max(8, S // 32))


def _indices(g, S: int, nab: int, nc: int, zipf: float, grouped: bool):
    a = torch.randint(0, nab, (S,), generator=g, device="cuda")
    b = torch.randint(0, nab, (S,), generator=g, device="cuda")
    if zipf > 0.0:
        w = torch.arange(1, nc + 1, device="cuda", dtype=torch.float64) ** -zipf
        cdf = torch.cumsum(w, 0) / w.sum()
        u = torch.rand(S, generator=g, device="cuda", dtype=torch.float64)
        rank = torch.searchsorted(cdf, u).clamp_(max=nc - 1)
        c = torch.randperm(nc, generator=g, device="cuda")[rank]
    else:
        c = torch.randint(0, nc, (S,), generator=g, device="cuda")
    if grouped:
        c = torch.sort(c).values
    return a, b, c


def _triples(a, b, c, m: int, n: int, k: int) -> torch.Tensor:
    return torch.stack((a * (m * k) + 1, b * (k * n) + 1, c * (m * n) + 1), 1).to(torch.int32).contiguous()


def _stack_inputs(g, m, n, k, S, zipf, grouped, spread=0) -> dict:
    nab, nc = _blocks(S)
    idx = _indices(g, S, nab, nc, zipf, grouped)
    return {"m": m, "n": n, "k": k, "S": S, "nab": nab, "nc": nc, "idx": idx,
            "a": _values(g, nab * m * k, spread), "b": _values(g, nab * k * n, spread),
            "c": _values(g, nc * m * n), "stack": _triples(*idx, m, n, k)}


def _batch_stacks(case: dict) -> list[tuple[int, int, int, int]]:
    """(m, n, k, S) of every stack of a batch: shapes from BLOCK_SIZES, sizes log-uniform in
    [smin, smax] scaled by one factor to `total` triples."""
    import random

    r = random.Random(case["pick"])
    shapes = [tuple(r.choice(BLOCK_SIZES) for _ in range(3)) for _ in range(case["stacks"])]
    sizes = [math.exp(r.uniform(math.log(case["smin"]), math.log(case["smax"]))) for _ in shapes]
    f = case["total"] / sum(sizes)
    return [(*s, max(1, int(round(S * f)))) for s, S in zip(shapes, sizes)]


def _inputs(case: dict, seed: int) -> dict:
    g = _gen(seed)
    kind = case["kind"]
    if kind in ("stack", "dbm"):
        s = _stack_inputs(g, case["m"], case["n"], case["k"], case["S"], case["zipf"], case["grouped"], case.get("spread", 0))
        if kind == "dbm":  # (m, n, k, a, b, c) with 0-based offsets
            m, n, k = case["m"], case["n"], case["k"]
            shape = torch.tensor([m, n, k], device="cuda", dtype=torch.int32).expand(case["S"], 3)
            s["stack"] = torch.cat((shape, s["stack"] - 1), 1).contiguous()
        return s
    if kind == "batch":
        return {"parts": [_stack_inputs(g, m, n, k, S, 1.1, False) for m, n, k, S in _batch_stacks(case)]}
    if kind == "multiply":
        m, n, k, nb = case["m"], case["n"], case["k"], case["nblocks"]
        nc = max(8, nb // 8)
        s = {"nc": nc, "a": _values(g, nb * m * k), "b": _values(g, nb * k * n)}  # both column-major blocks
        s["idx"] = [_indices(g, case["S"], nb, nc, 1.1, False) for _ in range(case["stacks"])]
        s["stacks"] = [_triples(*i, m, n, k) for i in s["idx"]]
        at = torch.arange(nb, device="cuda", dtype=torch.int32)
        s["at_a"], s["at_b"] = at * (m * k), at * (k * n)
        return s
    if kind == "ozaki_stack":
        return _stack_inputs(g, case["m"], case["n"], case["k"], case["S"], 1.1, False, 20)
    M, N, K = case["M"], case["N"], case["K"]
    # column-major operands; entries uniform, rows of op(A) and columns of op(B) at magnitudes of their own
    op_a, op_b = _values(g, M * K).view(M, K), _values(g, K * N).view(K, N)
    if kind != "dgemm":
        op_a = op_a * torch.ldexp(torch.ones((), device="cuda", dtype=torch.float64),
                                  torch.randint(-8, 9, (M, 1), generator=g, device="cuda"))
        op_b = op_b * torch.ldexp(torch.ones((), device="cuda", dtype=torch.float64),
                                  torch.randint(-8, 9, (1, N), generator=g, device="cuda"))
    a = op_a if case.get("ta", "N") == "T" else op_a.T
    b = op_b if case.get("tb", "N") == "T" else op_b.T
    return {"op_a": op_a, "op_b": op_b, "a": a.contiguous(), "b": b.contiguous(), "c": _values(g, M * N).view(N, M)}


def prepare(case: dict, seed: int) -> dict:
    stream = _the_stream()
    x = _inputs(case, seed)
    kind = case["kind"]
    state = {"case": case, "stream": stream}
    if kind in ("stack", "dbm", "ozaki_stack"):
        state.update({name: Buf(x[name]) for name in ("stack", "a", "b", "c")}, nab=x["nab"])
    elif kind == "batch":
        descs = [StackDesc(p["stack"].data_ptr(), p["S"], p["m"], p["n"], p["k"], p["a"].data_ptr(), p["b"].data_ptr(),
                           p["c"].data_ptr()) for p in x["parts"]]
        state.update(parts=[(p["stack"], p["a"], p["b"], p["c"]) for p in x["parts"]],
                     descs=(StackDesc * len(descs))(*descs))
    elif kind == "multiply":
        state.update(a=Buf(x["a"]), b_in=Buf(x["b"]), b=Buf(torch.empty_like(x["b"])),
                     c=Buf(torch.empty(x["nc"] * case["m"] * case["n"], device="cuda", dtype=torch.float64)),
                     at_a=Buf(x["at_a"]), at_b=Buf(x["at_b"]), stacks=[Buf(t) for t in x["stacks"]],
                     ne_a=Buf(torch.full_like(x["at_a"], case["m"] * case["k"])),
                     ne_b=Buf(torch.full_like(x["at_b"], case["k"] * case["n"])),
                     norms_a=Buf(torch.empty(case["nblocks"], device="cuda", dtype=torch.float32)),
                     norms_b=Buf(torch.empty(case["nblocks"], device="cuda", dtype=torch.float32)))
    else:
        state.update(a=Buf(x["a"]), b=Buf(x["b"]), c=Buf(x["c"]))
    torch.cuda.synchronize()  # the inputs are made on torch's stream, the calls use the library's
    return state


# ------------------------------------------------------------------------------------- one pass

def run(s: dict):
    case, stream, kind = s["case"], s["stream"], s["case"]["kind"]
    if kind == "stack":
        check(acc.process(s["stack"], case["S"], s["a"], s["b"], s["c"], case["m"], case["n"], case["k"], stream,
                          MAX_KERNEL_DIM), "process")
        return s["c"].t
    if kind == "dbm":
        shape = case["m"] | case["n"] << 8 | case["k"] << 16
        check(lib().libxstream_b200_dbm_launch(stream.handle, case["alpha"], case["S"], shape, None, s["stack"].ptr,
                                               s["a"].ptr, s["b"].ptr, s["c"].ptr), "dbm_launch")
        return s["c"].t
    if kind == "batch":
        check(lib().libxstream_b200_process_batch(ctypes.cast(s["descs"], ctypes.c_void_p), len(s["descs"]), MAX_KERNEL_DIM,
                                                  stream.handle), "process_batch")
        return [p[3] for p in s["parts"]]
    if kind == "multiply":
        m, n, k, nb = case["m"], case["n"], case["k"], case["nblocks"]
        check(acc.norms(s["a"], nb, s["at_a"], s["ne_a"], s["norms_a"], stream), "norms")
        check(acc.norms(s["b_in"], nb, s["at_b"], s["ne_b"], s["norms_b"], stream), "norms")
        check(lib().c_dbcsr_acc_memcpy_d2d(s["b_in"].ptr, s["b"].ptr, s["b"].nbytes, stream.handle), "memcpy")
        check(acc.transpose(s["at_b"], 0, nb, s["b"], k, n, stream), "transpose")
        check(lib().c_dbcsr_acc_memset_zero(s["c"].ptr, 0, s["c"].nbytes, stream.handle), "memset")
        for st in s["stacks"]:
            check(acc.process(st, case["S"], s["a"], s["b"], s["c"], m, n, k, stream, MAX_KERNEL_DIM), "process")
        return {"c": s["c"].t, "b": s["b"].t, "norms_a": s["norms_a"].t, "norms_b": s["norms_b"].t}
    if kind == "ozaki_stack":
        check(acc.process_ozaki(s["stack"], case["S"], case["m"], case["n"], case["k"], s["a"], s["nab"], s["b"], s["nab"],
                                s["c"], case["slices"], case["trim"], stream), "process_ozaki")
        return s["c"].t
    M, N, K = case["M"], case["N"], case["K"]
    if kind == "dgemm":
        check(acc.dgemm(M, N, K, 1.0, s["a"], M, s["b"], K, case["beta"], s["c"], M, stream), "dgemm")
        return s["c"].t
    lda, ldb = (M if case["ta"] == "N" else K), (K if case["tb"] == "N" else N)
    if kind == "ozaki1":
        check(acc.ozaki_gemm(case["ta"], case["tb"], M, N, K, 1.0, s["a"], lda, s["b"], ldb, case["beta"], s["c"], M,
                             case["slices"], case["trim"], stream), "ozaki_gemm")
    else:
        check(acc.ozaki2_gemm(case["ta"], case["tb"], M, N, K, 1.0, s["a"], lda, s["b"], ldb, case["beta"], s["c"], M,
                              case["moduli"], stream), "ozaki2_gemm")
    return s["c"].t


# ----------------------------------------------------------------- what a pass cannot do without

def _stack_work(m, n, k, S, nab, nc) -> tuple[float, float]:
    nab, nc = min(nab, S), min(nc, S)
    return 12.0 * S + 8.0 * (nab * (m * k + k * n) + 2 * nc * m * n), 2.0 * m * n * k * S


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind in ("stack", "dbm", "ozaki_stack"):
        b, f = _stack_work(case["m"], case["n"], case["k"], case["S"], *_blocks(case["S"]))
        b += 12.0 * case["S"] if kind == "dbm" else 0.0
    elif kind == "batch":
        parts = [_stack_work(m, n, k, S, *_blocks(S)) for m, n, k, S in _batch_stacks(case)]
        b, f = sum(p[0] for p in parts), sum(p[1] for p in parts)
    elif kind == "multiply":
        m, n, k, S, nb = case["m"], case["n"], case["k"], case["S"], case["nblocks"]
        # A and B read, B transposed written, norms and offsets, C written, the stacks
        b = 8.0 * nb * (m * k + 2 * k * n) + 24.0 * nb + 8.0 * max(8, nb // 8) * m * n + 12.0 * S * case["stacks"]
        f = 2.0 * m * n * k * S * case["stacks"] + 2.0 * nb * (m * k + k * n)
    else:
        M, N, K = case["M"], case["N"], case["K"]
        b = 8.0 * (M * K + K * N + (2 if case["beta"] else 1) * M * N)
        f = 2.0 * M * N * K
    return {"bytes": b, "flops": f}


# ------------------------------------------------------------------- the same values by plain torch

def _exact_stack(c, idx, a, b, m, n, k, alpha=1.0) -> torch.Tensor:
    """c + alpha * sum of A[a] B[b] per C block; A m x k column-major, B k x n row-major, C column-major."""
    av, bv = a.view(-1, k, m), b.view(-1, k, n)
    out = c.clone().view(-1, n * m)
    ia, ib, ic = idx
    step = max(1, (1 << 26) // max(m * n, m * k, k * n))
    for i in range(0, ia.numel(), step):
        # (A B)^T = B^T A^T: row index n, column index m, which is the column-major block
        p = torch.bmm(bv[ib[i:i + step]].transpose(1, 2), av[ia[i:i + step]])
        out.index_add_(0, ic[i:i + step], p.reshape(-1, n * m), alpha=alpha)
    return out.view(-1)


def exact(case: dict, seed: int):
    x = _inputs(case, seed)
    kind = case["kind"]
    if kind in ("stack", "dbm", "ozaki_stack"):
        return _exact_stack(x["c"], x["idx"], x["a"], x["b"], case["m"], case["n"], case["k"], case.get("alpha", 1.0))
    if kind == "batch":
        return [_exact_stack(p["c"], p["idx"], p["a"], p["b"], p["m"], p["n"], p["k"]) for p in x["parts"]]
    if kind == "multiply":
        m, n, k, nb = case["m"], case["n"], case["k"], case["nblocks"]
        bt = x["b"].view(nb, n, k).transpose(1, 2).contiguous().view(-1)
        c = torch.zeros(x["nc"] * m * n, device="cuda", dtype=torch.float64)
        for idx in x["idx"]:
            c = _exact_stack(c, idx, x["a"], bt, m, n, k)
        return {"c": c, "b": bt, "norms_a": x["a"].view(nb, -1).square().sum(1).sqrt(),
                "norms_b": x["b"].view(nb, -1).square().sum(1).sqrt()}
    c = (x["op_a"] @ x["op_b"]).T.contiguous()
    return c + x["c"] if case["beta"] else c
