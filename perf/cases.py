"""Performance cases: the work that users of the sparse attention operators have them do.

Every case is one forward of one mask family through the torch modules that a program imports (`spfa_<mask>.forward`
and their `plan` / `forward_planned`), on seeded N(0, 1) inputs that lie on the GPU. A program that calls the operators
for every layer and head keeps its (m, l, O) buffers: it resets (m, l) to the empty state with one copy before each
call, which also voids what O holds (a row's old O counts with weight l = 0). That reset is part of the pass; nothing
else is. Kinds:

  chain    Local, then Global-no-local, then a random CSR mask on one state: the three-call composition, small
  csr      diagonal + Bernoulli entries as CSR, float32
  csr16    power-law graph as CSR, float16 / bfloat16
  local    sliding window, float32
  local16  sliding window, float16 / bfloat16
  batched  sliding window over [batch * heads, L, d], float32
  l1d      1D-dilated window
  gnl      global rows and columns, local window excluded
  l2d      block-diagonal with intra-block dilation, rows without keys NaN-filled
  bigbird  window + globals + random CSR entries in one fused call
  coo      power-law graph united with a band, row-sorted COO, mask analysed inside the call
  planned  the same graph from a stored plan (a mask applied by many layers)
"""
import functools
import importlib
import math

import numpy as np
import torch

PACKAGE = "graph-processing-attention-ipdps-2025_b200"
MAX_DEGREE = 8192
DTYPES = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}


@functools.lru_cache(maxsize=None)
def module(name):
    return importlib.import_module(PACKAGE).binding("spfa_" + name)


def listed():
    return [
        # latency: the three chained calls at the size of the verification script of the operators
        {"name": "chain_256", "kind": "chain", "L": 256, "d": 32, "w": 10, "globals": 8, "random": 4},
        # the small explicit-mask configuration: one short launch
        {"name": "csr_4096", "kind": "csr", "L": 4096, "d": 64, "random": 41},
        # a mid-size graph in half precision (16-bit storage is what models hold), a ragged number of nodes
        {"name": "csr_f16_50021", "kind": "csr16", "L": 50021, "d": 64, "random": 48, "dtype": "f16"},
        # the sliding-window configuration
        {"name": "local_65536", "kind": "local", "L": 65536, "d": 64, "w": 256},
        # a sliding-window layer of a half-precision model, one wide head
        {"name": "local_bf16_32768", "kind": "local16", "L": 32768, "d": 128, "w": 512, "dtype": "bf16"},
        # all heads of a small batch in one call, length not a multiple of any tile
        {"name": "local_heads_24x4001", "kind": "batched", "slices": 24, "L": 4001, "d": 64, "w": 128},
        # the dilated-window configuration
        {"name": "l1d_131072", "kind": "l1d", "L": 131072, "d": 128, "w": 512, "dilation": 1},
        # the global-token configuration
        {"name": "gnl_131072", "kind": "gnl", "L": 131072, "d": 128, "w": 256, "globals": 64},
        # the block-dilated configuration, dead rows NaN-filled
        {"name": "l2d_262144", "kind": "l2d", "L": 262144, "d": 64, "block": 256, "dilation": 4},
        # window + globals + random keys, fused
        {"name": "bigbird_131072", "kind": "bigbird", "L": 131072, "d": 64, "w": 256, "globals": 64, "random": 32},
        # the million-token graph as a one-shot call
        {"name": "coo_1048576", "kind": "coo", "L": 1048576, "d": 64, "band": 64, "random": 32},
        # the same graph, analysed once and applied many times
        {"name": "planned_1048576", "kind": "planned", "L": 1048576, "d": 64, "band": 64, "random": 32},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice([c["kind"] for c in listed()])
    c = {"kind": kind, "d": rng.choice([32, 64, 64, 128])}
    if kind == "chain":
        c.update(L=_log_int(rng, 128, 4096), w=rng.randint(4, 24), globals=rng.randint(4, 16), random=rng.randint(2, 8))
    elif kind == "csr":
        c.update(L=_log_int(rng, 1000, 16384), random=_log_int(rng, 8, 128), d=rng.choice([16, 32, 64, 64, 96, 128]))
    elif kind == "csr16":
        c.update(L=_log_int(rng, 8192, 262144), random=_log_int(rng, 12, 64), dtype=rng.choice(["f16", "bf16"]))
    elif kind == "local":
        c.update(L=_log_int(rng, 2048, 262144), w=_log_int(rng, 16, 1024))
    elif kind == "local16":
        c.update(L=_log_int(rng, 2048, 131072), w=_log_int(rng, 16, 1024), dtype=rng.choice(["f16", "bf16"]))
    elif kind == "batched":
        c.update(slices=rng.randint(4, 48), L=_log_int(rng, 500, 8192), w=_log_int(rng, 32, 512))
    elif kind == "l1d":
        c.update(L=_log_int(rng, 8192, 262144), w=_log_int(rng, 32, 1024), dilation=rng.randint(1, 7))
    elif kind == "gnl":
        c.update(L=_log_int(rng, 8192, 262144), w=_log_int(rng, 32, 512), globals=_log_int(rng, 8, 256))
    elif kind == "l2d":
        block = rng.choice([64, 128, 256, 512])
        c.update(L=max(1, _log_int(rng, 8192, 524288) // block) * block, block=block, dilation=rng.randint(1, 7))
    elif kind == "bigbird":
        c.update(L=_log_int(rng, 8192, 131072), w=_log_int(rng, 32, 512), globals=_log_int(rng, 8, 128),
                 random=_log_int(rng, 8, 48))
    else:
        c.update(L=_log_int(rng, 32768, 1000000), d=rng.choice([32, 64]), band=rng.randint(16, 64), random=rng.randint(8, 32))
    return c


# ---- masks ----------------------------------------------------------------------------------------------------------
@functools.lru_cache(maxsize=8)
def _degrees(L, mean):
    """Row degrees of a power-law graph (tail exponent 2.1), stratified so that their multiset depends on (L, mean) alone."""
    z = np.floor(((np.arange(L) + 0.5) / L) ** (-1.0 / 1.1))
    return np.minimum(np.minimum(MAX_DEGREE, L // 2), np.rint(z * (mean / z.mean()))).astype(np.int64)


def _offsets(rows, L):
    off = torch.zeros(L + 1, dtype=torch.int64, device=rows.device)
    off[1:] = torch.cumsum(torch.bincount(rows, minlength=L), 0)
    return off


def _csr(keys, L):
    """Sorted unique keys row * L + column -> (offsets, columns) in the operators' index types."""
    return _offsets(keys // L, L).view(torch.uint64), (keys % L).to(torch.int32).view(torch.uint32)


def _graph(L, mean, band, g, dev):
    deg = torch.from_numpy(_degrees(L, mean)).to(dev)[torch.randperm(L, device=dev, generator=g)]
    rows = torch.repeat_interleave(torch.arange(L, device=dev), deg)
    parts = [rows * L + torch.randint(0, L, (rows.numel(),), device=dev, generator=g)]
    if band >= 0:
        i = torch.arange(L, device=dev).unsqueeze(1)
        j = i + torch.arange(-band, band + 1, device=dev)
        parts.append((i * L + j)[(j >= 0) & (j < L)])
    return torch.unique(torch.cat(parts))


def _random_part(L, w, listed_rows, per_row, g, dev):
    """Random keys per row outside the window and off the global rows and columns (the three parts stay disjoint)."""
    rows = torch.arange(L, device=dev).repeat_interleave(per_row)
    cols = torch.randint(0, L, (L * per_row,), device=dev, generator=g)
    is_global = torch.zeros(L, dtype=torch.bool, device=dev)
    is_global[listed_rows.long()] = True
    keep = ((rows - cols).abs() > w) & ~is_global[rows] & ~is_global[cols]
    return torch.unique(rows[keep] * L + cols[keep])


# ---- a program's state ----------------------------------------------------------------------------------------------
def prepare(case, seed):
    dev, kind, L, d = torch.device("cuda"), case["kind"], case["L"], case["d"]
    dtype = DTYPES[case.get("dtype", "f32")]
    g = torch.Generator(device=dev).manual_seed(seed)
    shape = (case["slices"], L) if kind == "batched" else (L,)
    s = {"case": case}
    for t in "QKV":
        s[t] = torch.randn(*shape, d, device=dev, generator=g).to(dtype)
    s["empty"] = torch.zeros(2, *shape, device=dev, dtype=dtype)
    s["empty"][0] = -math.inf
    s["ml"] = s["empty"].clone()
    s["m"], s["l"] = s["ml"][0], s["ml"][1]
    s["O"] = torch.zeros(*shape, d, device=dev, dtype=dtype)
    if kind in ("chain", "gnl", "bigbird"):
        s["G"] = torch.sort(torch.randperm(L, device=dev, generator=g)[: case["globals"]]).values.to(torch.int32)
    if kind in ("chain", "bigbird"):
        s["off"], s["col"] = _csr(_random_part(L, case["w"], s["G"], case["random"], g, dev), L)
    elif kind == "csr":
        mask = torch.rand(L, L, device=dev, generator=g) < case["random"] / L
        mask.fill_diagonal_(True)
        at = mask.nonzero()
        s["off"], s["col"] = _csr(at[:, 0] * L + at[:, 1], L)
    elif kind == "csr16":
        s["off"], s["col"] = _csr(_graph(L, case["random"], 0, g, dev), L)
    elif kind in ("coo", "planned"):
        keys = _graph(L, case["random"], case["band"], g, dev)
        s["row"], s["col"] = (keys // L).view(torch.uint64), (keys % L).to(torch.int32).view(torch.uint32)
        if kind == "planned":
            s["nnz"] = keys.numel()
            s["plan"] = module("coo").plan(s.pop("row"), s.pop("col"), L, L, d)
    if "col" in s:
        s["val"] = torch.ones(s["col"].numel(), device=dev, dtype=dtype)  # the mask's values: an argument, not a factor
    return s


def run(s):
    c, kind = s["case"], s["case"]["kind"]
    s["ml"].copy_(s["empty"])
    Q, K, V, m, l, O = s["Q"], s["K"], s["V"], s["m"], s["l"], s["O"]
    if kind == "chain":
        module("local").forward(Q, K, V, m, l, O, c["w"])
        module("global_no_local").forward(Q, K, V, m, l, O, s["G"], c["w"])
        module("csr").forward(Q, K, V, s["off"], s["col"], s["val"], m, l, O, False)
    elif kind in ("csr", "csr16"):
        module("csr").forward(Q, K, V, s["off"], s["col"], s["val"], m, l, O, False)
    elif kind in ("local", "local16", "batched"):
        module("local").forward(Q, K, V, m, l, O, c["w"])
    elif kind == "l1d":
        module("local_1d_dilated").forward(Q, K, V, m, l, O, c["w"], c["dilation"])
    elif kind == "gnl":
        module("global_no_local").forward(Q, K, V, m, l, O, s["G"], c["w"])
    elif kind == "l2d":
        module("local_2d_dilated").forward(Q, K, V, m, l, O, c["block"], c["dilation"], True)
    elif kind == "bigbird":
        module("bigbird").forward(Q, K, V, m, l, O, s["G"], c["w"], s["off"], s["col"])
    elif kind == "coo":
        module("coo").forward(Q, K, V, s["row"], s["col"], s["val"], m, l, O, False)
    else:
        module("coo").forward_planned(Q, K, V, s["plan"], s["nnz"], m, l, O, False)
    return {"O": O, "m": m, "l": l}


# ---- what a pass cannot do without ----------------------------------------------------------------------------------
def _window(L, w):
    """Pairs |i - j| <= w within [0, L)."""
    w = min(w, L - 1)
    return L * (2 * w + 1) - w * (w + 1)


def work(case):
    kind, L, d = case["kind"], case["L"], case["d"]
    size = 4 if case.get("dtype", "f32") == "f32" else 2
    n = case.get("slices", 1)
    live, index, window, random = L, 0, 0, 0  # rows with keys, bytes of the mask, keys of the closed-form part / the rest
    if kind in ("chain", "bigbird"):
        window = _window(L, case["w"])
        random = L * case["random"]
    if kind in ("gnl", "chain", "bigbird"):
        window += max(0, 2 * case["globals"] * (L - 2 * case["w"]))
        index += 4 * case["globals"]
    if kind in ("local", "local16", "batched"):
        window = n * _window(L, case["w"])
    if kind == "l1d":
        s = case["dilation"] + 1
        window = sum(_window((L - r + s - 1) // s, case["w"]) for r in range(s))
    if kind == "l2d":
        keys = (case["block"] - 1) // (case["dilation"] + 1) + 1
        live = L // case["block"] * keys
        window = live * keys
    if kind == "csr":
        random = L * (case["random"] + 1)
    if kind in ("csr16", "coo", "planned"):
        random = int(_degrees(L, case["random"]).sum())
        band = _window(L, case.get("band", 0))
        if kind == "csr16":
            random += band
        elif kind == "coo":
            index += 12 * (random + band)  # 64-bit rows, 32-bit columns
        else:  # a plan: a bit for each pair of the band's 64-key tiles, the other columns as they are
            index += (L // 128 + 1) * 1024 * ((127 + 2 * case["band"]) // 64 + 1) + 4 * random
        window = band if kind != "csr16" else 0
    if kind in ("csr", "csr16", "chain", "bigbird"):
        index += 8 * (L + 1) + 4 * random
    rows = n * (live if kind == "l2d" else L)
    # Q, K, V read, O written (2D-dilated: dead rows are written and not read), (m, l) read and written
    return {"bytes": size * (3 * rows * d + n * L * d) + 4 * size * rows + index, "flops": 4.0 * d * (window + random)}


def tolerance(case):
    kind, d = case["kind"], case["d"]
    if case.get("dtype") == "bf16":
        return {"rel": 1e-2}  # results are stored with 8 bits
    if case.get("dtype") == "f16":
        return {"rel": 2e-3}  # results are stored with 11 bits
    window = kind in ("local", "batched", "l1d") and case["w"] >= 32
    if d in (32, 64, 128) and (window or kind in ("chain", "gnl", "bigbird", "coo", "planned")):
        return {"rel": 2e-3}  # tensor-core products of operands with 11 significant bits (TF32)
    return {"rel": 1e-5}  # float32 throughout
