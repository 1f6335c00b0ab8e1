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
