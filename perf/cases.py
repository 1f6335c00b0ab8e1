"""What a program does with this library, as cases that can be timed.

A case is a dict of plain values; `prepare` makes the inputs it names on the GPU (pinned host memory for the
host-buffer calls), `run` is one pass through the package's public entry points.  Everything is fp32 CSR, the
only data type the library takes.  `kind` says which call a case makes:

  spmm          Context.spmm, or Context.spmm_planned with a plan kept by the caller (`planned`)
  sddmm         Context.sddmm, or Context.sddmm_masked with the mask's values as factors (`masked`)
  fused         Context.fused on a band mask with uniform extra entries
  attention     Context.attention with softmax on such a mask
  spmm_batch    Batch.launch on a prepared batch of independent SpMMs
  spmm_group, sddmm_group, fused_group    the one-shot grouped calls
  spmm_host     Context.spmm_batched_host on problems in pinned host memory
"""
import importlib
import math
import random

import torch

pkg = importlib.import_module("dlspm-esimd_b200")

# the shape / sparsity / width grid of pruned CNN and Transformer weights that the benchmark's batch is drawn
# from, and the inner dimensions of its grouped SDDMM and fused calls
SHAPES = [(64, 64), (256, 256), (512, 2048), (2048, 512), (1024, 4096)]
SPARSITIES = [0.5, 0.7, 0.8, 0.9, 0.95, 0.98]
WIDTHS = [256, 1024, 3136]
INNER = [32, 128, 256]
COV = 0.4  # spread of the row lengths of such weights (standard deviation over mean)


def listed():
    return [
        # one small layer, the first configuration of the benchmark: latency and the launch itself
        {"name": "spmm 512x512 n128", "kind": "spmm", "M": 512, "K": 512, "N": 128, "density": 0.1, "cov": 0.0, "planned": False},
        # a pruned Transformer layer on its own, the largest shape of the sweep
        {"name": "spmm 1024x4096 n1024", "kind": "spmm", "M": 1024, "K": 4096, "N": 1024, "density": 0.1, "cov": COV, "planned": False},
        # ragged sizes: the last stages of a CNN have 7 x 7 = 49 columns, so no row of B is 16-byte aligned
        {"name": "spmm 1003x1531 n49", "kind": "spmm", "M": 1003, "K": 1531, "N": 49, "density": 0.2, "cov": COV, "planned": False},
        # the single very large product of the multi-GPU configuration
        {"name": "spmm 65536 1% n512", "kind": "spmm", "M": 65536, "K": 65536, "N": 512, "density": 0.01, "cov": 0.0, "planned": False},
        # a pattern that is used again and again: plan made once, uneven rows
        {"name": "planned 8192x2048 n256", "kind": "spmm", "M": 8192, "K": 2048, "N": 256, "density": 0.1, "cov": COV, "planned": True},
        # the SDDMM configuration of the benchmark
        {"name": "sddmm 2048x512 n128", "kind": "sddmm", "M": 2048, "K": 512, "N": 128, "density": 0.2, "masked": False},
        # the largest square pattern of the reference's grid, the mask's values as factors (the gradient of a pruned layer)
        {"name": "sddmm masked 8192 n64", "kind": "sddmm", "M": 8192, "K": 8192, "N": 64, "density": 0.1, "masked": True},
        # the fused configuration of the benchmark: attention-like band plus 5 % extra entries
        {"name": "fused 4096 d64", "kind": "fused", "M": 4096, "N": 64, "half_band": 32, "density": 0.05},
        # sparse attention over a long sequence
        {"name": "attention 16384 d128", "kind": "attention", "M": 16384, "N": 128, "half_band": 32, "density": 0.01},
        # the benchmark's batch: a prepared batch drawn from the whole grid, one grouped launch a pass
        {"name": "batch of 256 spmm", "kind": "spmm_batch", "count": 256, "mix": 1},
        # patterns seen once: grouped SDDMM with its tables built by the call
        {"name": "group of 96 sddmm", "kind": "sddmm_group", "count": 96, "mix": 2},
        # problems that live in pinned host memory, copies both ways included
        {"name": "host batch of 24 spmm", "kind": "spmm_host", "count": 24, "mix": 3},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _width(rng, lo, hi):
    """Widths as they come up: most a multiple of 32 or of 4, some odd."""
    n = _log_int(rng, lo, hi)
    step = rng.choice([1, 4, 32, 32])
    return max(step, n // step * step)


def draw(rng):
    kind = rng.choice(["spmm", "spmm", "spmm", "sddmm", "sddmm", "fused", "attention", "spmm_batch", "spmm_group", "sddmm_group",
                       "fused_group", "spmm_host"])
    if kind in ("spmm_batch", "spmm_group"):
        return {"kind": kind, "count": _log_int(rng, 8, 200), "mix": rng.randrange(1 << 30)}
    if kind in ("sddmm_group", "fused_group"):
        return {"kind": kind, "count": _log_int(rng, 8, 150), "mix": rng.randrange(1 << 30)}
    if kind == "spmm_host":
        return {"kind": kind, "count": _log_int(rng, 4, 24), "mix": rng.randrange(1 << 30)}
    if kind in ("fused", "attention"):
        M = _log_int(rng, 256, 16384)
        return {"kind": kind, "M": M, "N": _width(rng, 16, 256), "half_band": rng.choice([8, 16, 32, 64]),
                "density": round(math.exp(rng.uniform(math.log(0.005), math.log(0.08))), 4)}
    M, K = _log_int(rng, 64, 16384), _log_int(rng, 64, 8192)
    density = round(1.0 - rng.choice(SPARSITIES), 2)
    if kind == "spmm":
        N = _width(rng, 16, 3136)
        case = {"kind": kind, "M": M, "K": K, "N": N, "density": density, "cov": rng.choice([0.0, COV]), "planned": rng.random() < 0.4}
    else:
        N = _width(rng, 16, 1024)
        case = {"kind": kind, "M": M, "K": K, "N": N, "density": density, "masked": rng.random() < 0.5}
    while 2.0 * case["M"] * K * N * density > 2e10:  # no more work than the large listed ones
        case["M"] = max(1, int(case["M"] * 0.7))
    return case


def _problems(case):
    """(M, K, N, sparsity) of every problem of a batch; a matter of the case, not of the seed."""
    rng = random.Random(case["mix"])
    widths = WIDTHS if case["kind"] in ("spmm_batch", "spmm_group", "spmm_host") else INNER
    return [(*rng.choice(SHAPES), rng.choice(widths), rng.choice(SPARSITIES)) for _ in range(case["count"])]


# ---- inputs -------------------------------------------------------------------------------------------------

_context = None


def _ctx():
    global _context
    if _context is None:
        _context = pkg.Context(0)
    return _context


def _pattern(gen, M, K, density, cov=0.0, half_band=-1):
    """CSR arrays of a random pattern: every row draws its columns with a probability of its own, which spreads
    the row lengths by `cov`; half_band >= 0 adds every column within that distance of the diagonal."""
    dev = gen.device
    p = torch.full((M, 1), float(density), device=dev)
    if cov > 0.0:
        p = (p * (1.0 + cov * torch.randn(M, 1, generator=gen, device=dev))).clamp_(0.0, 1.0)
    step = max(1, (1 << 27) // K)
    lengths, cols = [], []
    j = torch.arange(K, device=dev) if half_band >= 0 else None
    for r in range(0, M, step):
        n = min(step, M - r)
        keep = torch.rand(n, K, generator=gen, device=dev) < p[r:r + n]
        if half_band >= 0:
            i = torch.arange(r, r + n, device=dev)
            keep |= (i[:, None] - j[None, :]).abs() <= half_band
        lengths.append(keep.sum(1, dtype=torch.int32))
        cols.append((keep.view(-1).nonzero().view(-1) % K).to(torch.int32))
    ro = torch.zeros(M + 1, dtype=torch.int32, device=dev)
    ro[1:] = torch.cumsum(torch.cat(lengths), 0)
    ci = torch.cat(cols)
    return ro, ci, int(ci.numel())


def _uniform(gen, *shape):
    return torch.rand(*shape, generator=gen, device=gen.device).mul_(2.0).sub_(1.0)


def _normal(gen, *shape):
    return torch.randn(*shape, generator=gen, device=gen.device)


def _pad(n):
    return (n + 63) // 64 * 64


def _room(M, K, density, cov=0.0):
    """Entries that a pattern of _pattern stays below: an SDDMM's results go to the front of a buffer of this size,
    so that the buffer depends on the case and not on the seed."""
    spread = math.sqrt(M * K * density * (1.0 - density)) + math.sqrt(M) * cov * density * K
    return min(M * K, int(M * K * density + 10.0 * spread) + 64)


def prepare(case, seed):
    kind = case["kind"]
    dev = torch.device("cuda", 0)
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    ctx = _ctx()
    s = {"case": dict(case), "ctx": ctx}
    if kind == "spmm":
        M, K, N = case["M"], case["K"], case["N"]
        ro, ci, nnz = _pattern(gen, M, K, case["density"], case["cov"])
        s.update(args=(M, K, N, nnz), ro=ro, ci=ci, values=_uniform(gen, nnz), B=_uniform(gen, K, N),
                 out=torch.empty(M, N, device=dev))
        if case["planned"]:
            s["plan"] = ctx.plan_create(M, K, nnz, ro, ci)
    elif kind == "sddmm":
        M, K, N = case["M"], case["K"], case["N"]
        ro, ci, nnz = _pattern(gen, M, K, case["density"])
        s.update(args=(M, K, N, nnz), ro=ro, ci=ci, lhs=_normal(gen, M, N), rhs=_normal(gen, K, N),
                 mask=_uniform(gen, nnz) if case["masked"] else None, out=torch.zeros(_room(M, K, case["density"]), device=dev))
        s["out_values"] = s["out"][:nnz]
    elif kind in ("fused", "attention"):
        M, N = case["M"], case["N"]
        ro, ci, nnz = _pattern(gen, M, M, case["density"], half_band=case["half_band"])
        s.update(args=(M, M, N, nnz), ro=ro, ci=ci, q=_normal(gen, M, N), k=_normal(gen, M, N), v=_normal(gen, M, N),
                 out=torch.empty(M, N, device=dev))
    elif kind in ("spmm_batch", "spmm_group", "spmm_host"):
        problems = _problems(case)
        patterns = [_pattern(gen, M, K, 1.0 - sp, COV) for (M, K, N, sp) in problems]
        # one pool for the results: the problems' outputs one after the other
        total = sum(_pad(M * N) for (M, K, N, sp) in problems)
        if kind == "spmm_host":
            _prepare_host(s, gen, problems, patterns, total)
        else:
            out = torch.zeros(total, device=dev)
            arr, off = pkg.ProblemArray(len(problems)), 0
            for i, ((M, K, N, sp), (ro, ci, nnz)) in enumerate(zip(problems, patterns)):
                arr.set(i, M, K, N, nnz, _uniform(gen, nnz), ro, ci, _uniform(gen, K, N), out[off:off + M * N])
                off += _pad(M * N)
            s.update(array=arr, out=out)
            if kind == "spmm_batch":
                torch.cuda.synchronize()
                s["batch"] = ctx.batch_create(arr)
    else:
        problems = _problems(case)
        patterns = [_pattern(gen, M, K, 1.0 - sp, COV) for (M, K, N, sp) in problems]
        fused = kind == "fused_group"
        sizes = [_pad(M * N if fused else _room(M, K, 1.0 - sp, COV)) for (M, K, N, sp) in problems]
        out = torch.zeros(sum(sizes), device=dev)
        arr, off = pkg.RowProblemArray("fused" if fused else "sddmm", len(problems)), 0
        for i, ((M, K, N, sp), (ro, ci, nnz)) in enumerate(zip(problems, patterns)):
            q, k = _normal(gen, M, N), _normal(gen, K, N)
            if fused:
                arr.set_fused(i, M, K, N, nnz, ro, ci, q, k, _normal(gen, K, N), out[off:off + M * N])
            else:
                arr.set_sddmm(i, M, K, N, nnz, ro, ci, q, k, out[off:off + nnz])
            off += sizes[i]
        s.update(array=arr, out=out)
    torch.cuda.synchronize()
    return s


def _prepare_host(s, gen, problems, patterns, total):
    """Inputs in one pinned arena in the order of the library's staging layout (row_offsets, column_indices,
    values, B per problem, each padded to 256 bytes) and results in a second one, as dlspm.h advises."""
    words = sum(_pad(M + 1) + 2 * _pad(nnz) + _pad(K * N) for (M, K, N, sp), (ro, ci, nnz) in zip(problems, patterns))
    arena = torch.zeros(words, dtype=torch.int32, pin_memory=True)
    out = torch.zeros(total, pin_memory=True)
    arr, off, ooff = pkg.ProblemArray(len(problems)), 0, 0
    for i, ((M, K, N, sp), (ro, ci, nnz)) in enumerate(zip(problems, patterns)):
        at = []
        for t in (ro, ci, _uniform(gen, nnz), _uniform(gen, K * N)):
            part = arena[off:off + t.numel()]
            part.copy_(t.view(torch.int32))
            at.append(part)
            off += _pad(t.numel())
        arr.set(i, M, K, N, nnz, at[2].view(torch.float32), at[0], at[1], at[3].view(torch.float32),
                out[ooff:ooff + M * N], host=True)
        ooff += _pad(M * N)
    s.update(array=arr, arena=arena, out=out)


# ---- one pass -----------------------------------------------------------------------------------------------

def run(s):
    kind, ctx, out = s["case"]["kind"], s["ctx"], s["out"]
    if kind == "spmm":
        if "plan" in s:
            ctx.spmm_planned(s["plan"], s["args"][2], s["values"], s["ro"], s["ci"], s["B"], out)
        else:
            ctx.spmm(*s["args"], s["values"], s["ro"], s["ci"], s["B"], out)
    elif kind == "sddmm":
        if s["mask"] is not None:
            ctx.sddmm_masked(*s["args"], s["ro"], s["ci"], s["mask"], s["lhs"], s["rhs"], s["out_values"])
        else:
            ctx.sddmm(*s["args"], s["ro"], s["ci"], s["lhs"], s["rhs"], s["out_values"])
    elif kind == "fused":
        ctx.fused(*s["args"], s["ro"], s["ci"], s["q"], s["k"], s["v"], out)
    elif kind == "attention":
        ctx.attention(*s["args"], s["ro"], s["ci"], s["q"], s["k"], s["v"], out, scale=1.0 / math.sqrt(s["args"][2]),
                      flags=pkg.ATTN_SOFTMAX)
    elif kind == "spmm_batch":
        s["batch"].launch()
    elif kind == "spmm_group":
        ctx.spmm_batched(s["array"])
    elif kind == "sddmm_group":
        ctx.sddmm_batched(s["array"])
    elif kind == "fused_group":
        ctx.fused_batched(s["array"])
    else:
        ctx.spmm_batched_host(s["array"])
    return out


# ---- what a pass cannot do without --------------------------------------------------------------------------

def _work(op, M, K, N, nnz, masked=False):
    """(bytes, flops): every input read once, every output written once; the multiply-adds of the stored entries."""
    csr = 4.0 * (M + 1) + 4.0 * nnz
    if op == "spmm":
        return csr + 4.0 * nnz + 4.0 * K * N + 4.0 * M * N, 2.0 * nnz * N
    if op == "sddmm":
        return csr + (8.0 if masked else 4.0) * nnz + 4.0 * M * N + 4.0 * K * N, 2.0 * nnz * N
    return csr + 4.0 * N * (2.0 * M + 2.0 * K), 4.0 * nnz * N


def work(case):
    kind = case["kind"]
    if kind in ("spmm", "sddmm"):
        parts = [_work(kind, case["M"], case["K"], case["N"], case["M"] * case["K"] * case["density"], case.get("masked", False))]
    elif kind in ("fused", "attention"):
        M, b = case["M"], min(case["half_band"], case["M"] - 1)
        band = M * (2.0 * b + 1.0) - b * (b + 1.0)
        parts = [_work("fused", M, M, case["N"], band + (float(M) * M - band) * case["density"])]
    else:
        op = kind.split("_")[0]
        parts = [_work(op, M, K, N, M * K * (1.0 - sp)) for (M, K, N, sp) in _problems(case)]
    return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}


def tolerance(case):
    """Sums of up to a few thousand fp32 products in an order of the kernel's own."""
    return {"rel": 1e-5}
