"""One-shot grouped SpMM calls whose denser problems go to the tensor cores: against the CPU oracle, with columns in and out
of order, and the allocation-free form against the allocating one."""
import numpy as np
import pytest

from cases import csr_rowlen_normal, dense, shuffle_rows_columns
from conftest import TOL, to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("density", [0.5, 0.2])
def test_one_shot_group(pkg, oracle, ctx, dev, density):
    import torch

    shapes = [(512, 512, 512), (300, 200, 36), (513, 640, 768), (64, 64, 64), (1000, 257, 1028), (700, 300, 33)] * 3
    a, b = pkg.ProblemArray(len(shapes)), pkg.ProblemArray(len(shapes))
    keep = []
    for i, (M, K, N) in enumerate(shapes):
        d = density if i < 12 else 0.9  # both builds of the kernel in one call
        ro, ci = csr_rowlen_normal(pkg, M, K, 1.0 - d, 70 + i)
        if i in (2, 4):
            ci = shuffle_rows_columns(ro, ci, i)
        vals = pkg.gen_dense_host(int(ci.size), 70 + i, 2)
        B = dense(pkg, K, N, 70 + i, 10)
        outs = [torch.full((M * N,), float("nan"), device=dev) for _ in range(2)]
        d = [to_dev(x, dev) for x in (vals, ro, ci, B)]
        a.set(i, M, K, N, int(ci.size), *d, outs[0])
        b.set(i, M, K, N, int(ci.size), *d, outs[1])
        keep.append((M, N, ro, ci, vals, B, outs))
    ctx.spmm_batched(a)
    ctx.spmm_batched(a)
    ctx.spmm_batched_static(b)
    torch.cuda.synchronize()
    for M, N, ro, ci, vals, B, outs in keep:
        out, other = (o.cpu().numpy().reshape(M, N) for o in outs)
        assert np.array_equal(out.view(np.uint32), other.view(np.uint32))
        bad, worst = oracle.violations(oracle.spmm(vals, ro, ci, B, M, N), out, oracle.spmm_scale(vals, ro, ci, B, M, N), TOL / 50)
        assert bad == 0, worst


@pytest.mark.parametrize("density", [0.2, 0.9])  # the two builds of the kernel
def test_many_tiles_with_columns_out_of_order(pkg, oracle, ctx, dev, density):
    """More tiles for every pair of blocks than are planned ahead.  Every third problem is out of order as a whole (its
    tiles are passed over), the others in a few rows that the kernel does not look at beforehand; those rows must be
    computed again, and the rest must have been multiplied on the tensor cores: their bits differ from the gather's."""
    import torch

    shapes = [(700 + 37 * i, 257 + 30 * (i % 4), 1028 + 256 * (i % 2)) for i in range(18)]
    tiles = sum(-(-M // 128) * -(-N // 256) for i, (M, K, N) in enumerate(shapes) if i % 3)
    assert tiles > 5 * 74
    arr, keep = pkg.ProblemArray(len(shapes)), []
    for i, (M, K, N) in enumerate(shapes):
        ro, ci = csr_rowlen_normal(pkg, M, K, 1.0 - density, 200 + i, cov=0.1)
        mixed = []
        if i % 3 == 0:
            ci = shuffle_rows_columns(ro, ci, i)
        else:
            looked_at = {M * lane // 32 for lane in range(32)}
            for n, r in enumerate(r for r in range(5, M, 7) if r not in looked_at):
                start, end = int(ro[r]), int(ro[r + 1])
                at = (start, (start + end) // 2, end - 2)[n % 3]
                if n % 2:
                    ci[at + 1] = ci[at]
                else:
                    ci[at], ci[at + 1] = ci[at + 1], ci[at]
                mixed.append(r)
        vals, B = pkg.gen_dense_host(int(ci.size), 200 + i, 2), dense(pkg, K, N, 200 + i, 10)
        out = torch.full((M * N,), float("nan"), device=dev)
        arr.set(i, M, K, N, int(ci.size), to_dev(vals, dev), to_dev(ro, dev), to_dev(ci, dev), to_dev(B, dev), out)
        keep.append((ro, ci, vals, B, mixed, out))
    ctx.spmm_batched(arr)
    torch.cuda.synchronize()
    outs = [out.cpu().numpy().reshape(M, N) for (M, K, N), (*_, out) in zip(shapes, keep)]
    ctx.set_option(pkg.OPT_TILE_MIN_DENSITY, 0)  # with a threshold one-shot calls gather
    try:
        ctx.spmm_batched(arr)
        torch.cuda.synchronize()
    finally:
        ctx.set_option(pkg.OPT_TILE_MIN_DENSITY, -1)
    for i, ((M, K, N), (ro, ci, vals, B, mixed, out)) in enumerate(zip(shapes, keep)):
        bad, worst = oracle.violations(oracle.spmm(vals, ro, ci, B, M, N), outs[i], oracle.spmm_scale(vals, ro, ci, B, M, N), TOL / 50)
        assert bad == 0, (i, worst)
        if i % 3:
            same = (outs[i] == out.cpu().numpy().reshape(M, N)).all(axis=1)
            same[mixed] = False
            assert not same.any(), "rows not multiplied"
