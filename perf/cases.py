"""The work a user of this library has it do, as cases that can be timed.

A case is a sampling pattern (its family, size and row lengths), an inner dimension K, a storage / arithmetic mode and a
flow, i.e. which public calls make up one pass:

  run      the pattern is planned once and held, every pass computes P on the device: Engine.run() + Engine.sync(), what
           run_csr() of the competitor does inside the benchmark loop
  device   a new problem every pass, operands already on the GPU (one process per GPU with a broadcast B, a sampled
           subgraph): Engine.upload_csr_device() + run() + sync()
  host     the drop-in sequence init_csr / run_csr / cleanup_csr on pageable host arrays: Engine.upload_csr() + run() +
           download()
  iterate  an ALS-style step on a held pattern: new S values, A and B from pinned host memory, P = SDDMM, Y = P B, Y back
           to pinned host memory: Engine.update_raw() + run() + spmm_raw()

Families (the five configurations of the benchmark and what lies between them): uniform (small, random positions),
blocks (64 x 64 blocks 70 % full on the 64-grid), offset_blocks (the same at arbitrary offsets), banded (3 x 3 blocks in
a band), powerlaw (Zipf(2) rows and columns), poisson (Poisson row lengths, uniform columns).
"""
import math

import numpy as np
import torch

from dphpc_b200.capi import Engine


def listed():
    return [
        # the smallest configuration: a 656 x 656 mesh-sized matrix; launches and latency are all there is
        {"name": "small", "flow": "run", "family": "uniform", "mode": "fp32", "M": 656, "N": 656, "nnz": 18964, "K": 32},
        # clustered rows, fp32-grade results from the tensor cores
        {"name": "clustered fp32_tc", "flow": "run", "family": "blocks", "mode": "fp32_tc", "M": 14340, "N": 14340, "nnz": 18070000, "K": 32},
        # the same matrix in the default mode: plain fp32 arithmetic
        {"name": "clustered fp32", "flow": "run", "family": "blocks", "mode": "fp32", "M": 14340, "N": 14340, "nnz": 18070000, "K": 32},
        # blocks wherever they fall, bf16 operands
        {"name": "clustered bf16 offset K64", "flow": "run", "family": "offset_blocks", "mode": "bf16", "M": 14340, "N": 14340, "nnz": 18070000, "K": 64},
        # a stiffness-like matrix: three unknowns per node, short band
        {"name": "banded K64", "flow": "run", "family": "banded", "mode": "fp32", "M": 503712, "N": 503712, "nnz": 36800000, "K": 64},
        # a social-graph-like matrix: rows of 1 to 50 000 nonzeros, popular columns
        {"name": "powerlaw", "flow": "run", "family": "powerlaw", "mode": "fp32", "M": 2601977, "N": 2601977, "nnz": 36200000, "K": 32},
        # the benchmark's default workload: no reuse but through the caches
        {"name": "poisson", "flow": "run", "family": "poisson", "mode": "fp32", "M": 1453908, "N": 1453908, "nnz": 37500000, "K": 32},
        # the K sweep's bf16 half: the most bytes per nonzero of the list
        {"name": "poisson bf16 K128", "flow": "run", "family": "poisson", "mode": "bf16", "M": 1453908, "N": 1453908, "nnz": 37500000, "K": 128},
        # odd sizes throughout: a rectangular rating matrix and a rank that is no multiple of four
        {"name": "ragged K50", "flow": "run", "family": "poisson", "mode": "fp32", "M": 60013, "N": 17771, "nnz": 2400000, "K": 50},
        # a subgraph of a larger training set, another one in every step
        {"name": "device subgraph K64", "flow": "device", "family": "poisson", "mode": "fp32", "M": 200003, "N": 200003, "nnz": 5200000, "K": 64},
        # the drop-in call on host containers
        {"name": "host banded", "flow": "host", "family": "banded", "mode": "fp32", "M": 50373, "N": 50373, "nnz": 3680000, "K": 32},
        # alternating least squares on a rating matrix: factors from and to the host
        {"name": "iterate powerlaw K64", "flow": "iterate", "family": "powerlaw", "mode": "fp32", "M": 100003, "N": 50021, "nnz": 4000000, "K": 64},
    ]


# ranges: nonzeros from a small mesh to the largest configuration, mean row lengths of each family's configurations
MOST_GATHER = 37500000 * 128 * 2  # nonzeros * K * bytes per stored element of the largest listed case
FAMILIES = {  # family: (mean row length from, to; smallest M)
    "uniform": (5.0, 40.0, 200),
    "blocks": (100.0, 1300.0, 1024),
    "offset_blocks": (100.0, 1300.0, 1024),
    "banded": (30.0, 90.0, 3000),
    "powerlaw": (8.0, 40.0, 2000),
    "poisson": (8.0, 60.0, 500),
}


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    flow = rng.choice(["run"] * 7 + ["device", "host", "iterate"])
    family = rng.choice(["uniform", "blocks", "offset_blocks", "banded", "banded", "powerlaw", "powerlaw", "poisson", "poisson", "poisson"])
    clustered = family in ("blocks", "offset_blocks")
    mode = rng.choice(["fp32", "fp32_tc", "tf32", "bf16"] if clustered else ["fp32", "fp32", "fp32", "bf16"])
    if flow != "run":
        mode = "fp32_tc" if clustered else "fp32"
    K = rng.choice([32, 32, 32, 64, 64, 128, 256, 48, 96, 16, 100, 50, 33])
    if mode == "bf16":
        K = max(8, K // 8 * 8)
    if clustered:
        K = max(32, K // 32 * 32)
    if family == "banded" and flow == "run":
        K = rng.choice([32, 64, K])
    if flow == "iterate":
        K = max(16, K // 4 * 4)  # what the consumer of P takes
    lo, hi, small = FAMILIES[family]
    most = 200000 if family == "uniform" else 37500000 if flow == "run" and K % 4 == 0 else 5200000
    nnz = _log(rng, 15000 if family == "uniform" else 100000, most)
    nnz = min(nnz, MOST_GATHER / (K * (2 if mode == "bf16" else 4)))
    mean = _log(rng, lo, hi)
    M = max(small, int(nnz / mean)) + rng.randrange(7)
    if clustered:  # between a twentieth and a third of the matrix is covered
        M = max(small, int(math.sqrt(nnz / _log(rng, 0.03, 0.25)))) + rng.randrange(7)
    N = M if rng.random() < 0.5 or family == "banded" else max(small, int(M * _log(rng, 0.4, 2.0))) + rng.randrange(7)
    nnz = int(min(nnz, 0.25 * M * N, 90.0 * M if family == "banded" else nnz))
    return {"flow": flow, "family": family, "mode": mode, "M": M, "N": N, "nnz": nnz, "K": K}


# ---- patterns, made on the GPU from the seed alone ----------------------------------------------------------------------
def _csr(keys, M, N):
    """Sorted distinct keys row * N + column -> row_ptr, col_idx."""
    row = torch.div(keys, N, rounding_mode="floor")
    col = (keys - row * N).to(torch.int32)
    row_ptr = torch.zeros(M + 1, dtype=torch.int64, device="cuda")
    row_ptr[1:] = torch.cumsum(torch.bincount(row, minlength=M), 0)
    return row_ptr.to(torch.int32), col


def _rand(g, n):
    return torch.rand(int(n), generator=g, device="cuda")


def _below(g, n, high):
    return torch.randint(0, int(high), (int(n),), generator=g, device="cuda", dtype=torch.int64)


def _distinct(keys):
    return torch.unique_consecutive(torch.sort(keys).values)


def _zipf2(g, n, most):
    """Ranks 1 .. most with P(rank >= x) = 1 / x."""
    u = torch.clamp(_rand(g, n).double(), min=1e-9)
    return torch.clamp((1.0 / u).long(), 1, int(most))


def _rows_of(lens):
    return torch.repeat_interleave(torch.arange(lens.numel(), device="cuda"), lens)


def _exactly(g, keys, n, space):
    """n of the sorted distinct keys, chosen at random; where there are fewer, others below `space` join them."""
    while keys.numel() < n:
        keys = _distinct(torch.cat([keys, _below(g, 2 * (n - keys.numel()), space)]))
    drop = keys.numel() - n
    if drop == 0:
        return keys
    keep = torch.ones(keys.numel(), dtype=torch.bool, device="cuda")
    keep[torch.randperm(keys.numel(), generator=g, device="cuda")[:drop]] = False
    return keys[keep]


def _uniform(g, M, N, nnz):
    return _distinct(_below(g, int(nnz * 1.1) + 64, M * N))


def _poisson(g, M, N, nnz):
    lens = torch.clamp(torch.poisson(torch.full((M,), 1.005 * nnz / M, device="cuda"), generator=g).long(), max=N)
    rows = _rows_of(lens)
    return _distinct(rows * N + _below(g, rows.numel(), N))


def _powerlaw(g, M, N, nnz):
    most = min(50000, N // 2)
    raw = _zipf2(g, M, most).double()
    scale = 1.0
    for _ in range(12):  # the factor that makes the lengths, clipped to [1, most], add up to nnz
        lens = torch.clamp((scale * raw + 0.5).long(), 1, most)
        scale *= nnz / float(lens.sum())
    lens = torch.clamp((scale * raw + 0.5).long(), 1, most)
    perm = torch.randperm(N, generator=g, device="cuda")  # popularity rank -> column
    keys = torch.empty(0, dtype=torch.int64, device="cuda")
    for attempt in range(9):  # draw what a row still misses: by popularity at first, then anywhere
        have = torch.bincount(torch.div(keys, N, rounding_mode="floor"), minlength=M)
        rows = _rows_of(lens - have)
        if rows.numel() == 0:
            break
        cols = perm[_zipf2(g, rows.numel(), N) - 1] if attempt < 6 else _below(g, rows.numel(), N)
        keys = _distinct(torch.cat([keys, rows * N + cols]))
    return keys


def _blocks(g, M, N, nnz, offset):
    cell = 128 if offset else 64  # at offsets: one block somewhere in each chosen 128 x 128 cell, so blocks never overlap
    gr, gc = M // cell, N // cell
    n = min(gr * gc, math.ceil(1.001 * nnz / (0.7 * 64 * 64)))
    cells = torch.randperm(gr * gc, generator=g, device="cuda")[:n]
    r0, c0 = torch.div(cells, gc, rounding_mode="floor") * cell, cells % gc * cell
    if offset:
        r0, c0 = r0 + _below(g, n, 65), c0 + _below(g, n, 65)
    at = (_rand(g, n * 4096) < 0.7).nonzero().squeeze(1)
    block, r, c = at >> 12, (at >> 6) & 63, at & 63
    return torch.sort((r0[block] + r) * N + c0[block] + c).values


def _banded(g, M, N, nnz):
    nb = (M + 2) // 3
    half = max(1, min(2000, M // 4) // 3)
    rows = torch.arange(nb, device="cuda").repeat_interleave(math.ceil(1.1 * nnz / 9 / nb) + 1)
    cols = rows + _below(g, rows.numel(), 2 * half + 1) - half
    inside = (cols >= 0) & (cols < nb)
    pairs = _exactly(g, _distinct(rows[inside] * nb + cols[inside]), min(nb * half, -(-nnz // 9) + 64), nb * nb)
    rows, cols = torch.div(pairs, nb, rounding_mode="floor") * 3, pairs % nb * 3
    i = torch.arange(3, device="cuda")
    rows, cols = (rows[:, None, None] + i[None, :, None]), (cols[:, None, None] + i[None, None, :])
    rows, cols = rows.expand(-1, 3, 3).reshape(-1), cols.expand(-1, 3, 3).reshape(-1)
    inside = (rows < M) & (cols < N)
    return torch.sort(rows[inside] * N + cols[inside]).values[:nnz]  # whole blocks, but for the last few


def _problem(case, seed):
    """row_ptr, col_idx, S values, A, B on the GPU."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 1000003 + 17)
    M, N, K, nnz, family = (case[k] for k in ("M", "N", "K", "nnz", "family"))
    if family == "uniform":
        keys = _uniform(g, M, N, nnz)
    elif family == "poisson":
        keys = _poisson(g, M, N, nnz)
    elif family == "powerlaw":
        keys = _powerlaw(g, M, N, nnz)
    elif family == "banded":
        keys = _banded(g, M, N, nnz)
    else:
        keys = _blocks(g, M, N, nnz, family == "offset_blocks")
    row_ptr, col = _csr(_exactly(g, keys, nnz, M * N), M, N)
    val = torch.ones(col.numel(), device="cuda") if family == "powerlaw" else _rand(g, col.numel())
    A = 2.0 * _rand(g, M * K) - 1.0
    B = 2.0 * _rand(g, N * K) - 1.0
    return row_ptr, col, val, A, B


class _Device:
    """The engine's P.val as an array on the GPU; a tensor made from it keeps the engine, whose memory it is."""

    def __init__(self, engine, n):
        self.engine = engine
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": "<f4", "data": (engine.p_device(), False), "version": 3}


def prepare(case, seed):
    M, N, K = case["M"], case["N"], case["K"]
    problem = _problem(case, seed)
    torch.cuda.synchronize()  # the engine works on streams of its own
    nnz = problem[1].numel()
    engine = Engine(0, case["mode"])
    state = {"flow": case["flow"], "engine": engine, "dims": (M, N, K)}
    if case["flow"] == "host":
        state["arrays"] = [t.cpu().numpy() for t in problem]
        state["out"] = np.zeros(nnz, dtype=np.float32)
        return state
    if case["flow"] == "device":
        state["arrays"] = problem
        state["nnz"] = nnz
        return state
    engine.upload_csr_device(M, N, K, nnz, *(t.data_ptr() for t in problem))
    if case["flow"] == "iterate":
        state["arrays"] = [t.cpu().pin_memory() for t in problem[2:]]
        state["out"] = torch.zeros(M, K).pin_memory()
        return state
    state["out"] = torch.as_tensor(_Device(engine, nnz), device="cuda")
    return state


def run(state):
    engine, flow = state["engine"], state["flow"]
    if flow == "run":
        engine.run()
        engine.sync()
        return state["out"]
    M, N, K = state["dims"]
    if flow == "device":
        engine.upload_csr_device(M, N, K, state["nnz"], *(t.data_ptr() for t in state["arrays"]))
        engine.run()
        engine.sync()
        return torch.as_tensor(_Device(engine, state["nnz"]), device="cuda")
    if flow == "host":
        engine.upload_csr(M, N, K, *state["arrays"])
        engine.run()
        return engine.download(state["out"])
    val, A, B = state["arrays"]
    engine.update_raw(A.data_ptr(), B.data_ptr(), val.data_ptr())
    engine.run()
    engine.spmm_raw(K, 0, state["out"].data_ptr())
    return state["out"]


def work(case):
    """Each operand row that is needed once, column index and S value once, the result once."""
    M, N, K, nnz = case["M"], case["N"], case["K"], case["nnz"]
    e = 2 if case["mode"] == "bf16" else 4
    spread = 0.6 if case["family"] == "powerlaw" else 1.0  # popular columns are drawn again and again
    rows, cols = M * -math.expm1(-nnz / M), N * -math.expm1(-spread * nnz / N)
    done = {"bytes": e * K * (rows + cols) + 12 * nnz + 4 * (M + 1), "flops": 2 * nnz * K}
    if case["flow"] == "iterate":
        done["bytes"] += 4 * nnz + 4 * K * (M + cols)  # P and B again, Y
        done["flops"] += 2 * nnz * K
    return done


def tolerance(case):
    # tf32: 11 significand bits in the operands (truncated or rounded); every other mode sums exact or fp32-grade products
    # in 32 bits (bf16 storage rounds the operands one defined way)
    return {"rel": 1e-3} if case["mode"] == "tf32" else {"rel": 1e-5}
