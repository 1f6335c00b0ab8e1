"""GPU parity of the tensor-core SDDMM (csrc/sddmm_mma.cuh) against the CPU oracle: sizes around its tiles (128 rows,
256 columns, 64 of the inner dimension), dense enough to be taken by the dispatch."""
import numpy as np
import pytest

from cases import csr_bernoulli, csr_rowlen_normal, dense, shuffle_rows_columns
from conftest import TOL, to_dev

pytestmark = pytest.mark.gpu


def check(oracle, ro, ci, lhs, rhs, M, N, out, mask=None, tol=TOL / 50):
    ref = oracle.sddmm(ro, ci, lhs, rhs, M, N)
    scale = oracle.sddmm_scale(ro, ci, lhs, rhs, M, N)
    if mask is not None:
        ref, scale = ref * mask, scale * np.abs(mask)
    assert not np.isnan(out).any()
    bad, worst = oracle.violations(ref.astype(np.float32), out, scale.astype(np.float32), tol)
    assert bad == 0, worst


def lone_run(ctx, dev, M, K, N, ro, ci, lhs, rhs, mask=None):
    import torch

    nnz, guard = int(ci.size), 64
    buf = torch.full((nnz + 2 * guard,), float("nan"), device=dev)
    ctx.sddmm_masked(M, K, N, nnz, to_dev(ro, dev), to_dev(ci, dev), to_dev(mask, dev) if mask is not None else None,
                     to_dev(lhs, dev), to_dev(rhs, dev), buf[guard:guard + nnz])
    torch.cuda.synchronize()
    out = buf.cpu().numpy()
    assert np.isnan(out[:guard]).all() and np.isnan(out[guard + nnz:]).all(), "wrote outside the results"
    return out[guard:guard + nnz]


@pytest.mark.parametrize("M,K,N,density,kind", [(1024, 4096, 256, 0.5, "plain"), (1000, 4000, 300, 0.6, "masked"),
                                                (900, 3001, 255, 0.4, "masked"), (1024, 4096, 256, 0.5, "reversed"),
                                                (1024, 4096, 256, 0.5, "infinite"), (1024, 4096, 256, 0.5, "tiny"),
                                                (1024, 2048, 512, 0.5, "reversed"), (1024, 2048, 512, 0.5, "infinite"),
                                                (1024, 2048, 512, 0.5, "tiny"), (2048, 512, 512, 0.5, "masked"),
                                                (1500, 1000, 516, 0.4, "masked"), (1024, 2048, 512, 0.5, "tiny rows")])
def test_lone_launches(pkg, oracle, ctx, dev, M, K, N, density, kind):
    seed = M + N
    ro, ci = csr_rowlen_normal(pkg, M, K, 1.0 - density, seed)
    if kind == "reversed":
        for i in (0, 130, M - 1):  # a few rows: entries out of order are computed one by one
            ci[ro[i]:ro[i + 1]] = ci[ro[i]:ro[i + 1]][::-1]
    lhs = dense(pkg, M, N, seed, 11, kind=pkg.KIND_NORMAL)
    rhs = dense(pkg, K, N, seed, 12, kind=pkg.KIND_NORMAL)
    mask = pkg.gen_dense_host(int(ci.size), seed, 2) if kind == "masked" else None
    if kind == "tiny rows":  # each converted by one block of a pair, and looked up by both
        lhs, rhs = lhs.copy(), (rhs * np.float32(1e20)).astype(np.float32)
        lhs[[0, 9, 20, 31, 500, 1023]] *= np.float32(1e-36)
    if kind == "tiny":
        lhs, rhs = (lhs * np.float32(1e-36)).astype(np.float32), (rhs * np.float32(1e20)).astype(np.float32)
    if kind == "infinite":
        rhs = rhs.copy()
        rhs[77, 3] = np.inf
        out = lone_run(ctx, dev, M, K, N, ro, ci, lhs, rhs)
        hit = ci == 77
        assert hit.any() and np.isinf(out[hit]).all() and np.isfinite(out[~hit]).all()
        rhs[77, 3] = 0
        out[hit] = oracle.sddmm(ro, ci, lhs, rhs, M, N)[hit]
        check(oracle, ro, ci, lhs, rhs, M, N, out)
        return
    check(oracle, ro, ci, lhs, rhs, M, N, lone_run(ctx, dev, M, K, N, ro, ci, lhs, rhs, mask), mask)


def test_grouped_call_over_tile_edges(pkg, oracle, ctx, dev):
    """Problems that the tensor cores take (together they fill the device) next to some that they do not."""
    import torch

    shapes = [(385, 256, 256), (512, 257, 512), (513, 1000, 68), (640, 127, 1024), (1000, 2048, 128), (400, 129, 260),
              (2048, 512, 256), (100, 300, 64)] * 3
    arr = pkg.RowProblemArray("sddmm", len(shapes))
    keep = []
    for i, (M, K, N) in enumerate(shapes):
        ro, ci = csr_bernoulli(pkg, M, K, (0.5, 0.9, 0.3)[i // 8], 50 + i)
        if i == 8:
            ci = shuffle_rows_columns(ro, ci, i)
        nnz = int(ci.size)
        lhs = dense(pkg, M, N, 50 + i, 11, kind=pkg.KIND_NORMAL)
        rhs = dense(pkg, K, N, 50 + i, 12, kind=pkg.KIND_NORMAL)
        mask = pkg.gen_dense_host(nnz, 50 + i, 2) if i % 2 else None
        out = torch.full((nnz,), float("nan"), device=dev)
        arr.set_sddmm(i, M, K, N, nnz, to_dev(ro, dev), to_dev(ci, dev), to_dev(lhs, dev), to_dev(rhs, dev), out,
                      mask_values=to_dev(mask, dev) if mask is not None else None)
        keep.append((ro, ci, lhs, rhs, M, N, out, mask))
    ctx.sddmm_batched(arr)
    ctx.sddmm_batched(arr)
    torch.cuda.synchronize()
    for ro, ci, lhs, rhs, M, N, out, mask in keep:
        check(oracle, ro, ci, lhs, rhs, M, N, out.cpu().numpy(), mask)
