"""GPU parity of the tensor-core SpMM (csrc/spmm_mma.cuh) against the CPU oracle at the edges of its tiles: 128 rows,
256 columns, 64 columns of the sparse matrix per step, eight lanes per row."""
import numpy as np
import pytest

from cases import csr_bernoulli, csr_from_lengths, csr_rowlen_normal, dense, shuffle_rows_columns
from conftest import TOL, to_dev

pytestmark = pytest.mark.gpu


def batch_run(pkg, ctx, dev, M, K, N, ro, ci, vals, B):
    """One problem as a prepared batch that takes the tensor cores whatever its density."""
    import torch

    ctx.set_option(pkg.OPT_TILE_MIN_DENSITY, 0)
    try:
        arr = pkg.ProblemArray(1)
        guard = 64
        buf = torch.full((M * N + 2 * guard,), float("nan"), device=dev)
        arr.set(0, M, K, N, int(ci.size), to_dev(vals, dev), to_dev(ro, dev), to_dev(ci, dev), to_dev(B, dev),
                buf[guard:guard + M * N])
        batch = ctx.batch_create(arr)
        batch.launch()
        torch.cuda.synchronize()
        info = batch.info(check_device=True)
        batch.close()
    finally:
        ctx.set_option(pkg.OPT_TILE_MIN_DENSITY, -1)
    assert info == (0, 1, 0)
    out = buf.cpu().numpy()
    assert np.isnan(out[:guard]).all() and np.isnan(out[guard + M * N:]).all(), "wrote outside C"
    return out[guard:guard + M * N].reshape(M, N)


def lone_run(ctx, dev, M, K, N, ro, ci, vals, B, plan=False):
    import torch

    out = torch.full((M, N), float("nan"), device=dev)
    d = [to_dev(x, dev) for x in (vals, ro, ci, B)]
    if plan:
        p = ctx.plan_create(M, K, int(ci.size), d[1], d[2])
        ctx.spmm_planned(p, N, *d, out)
        torch.cuda.synchronize()
        p.close()
    else:
        ctx.spmm(M, K, N, int(ci.size), *d, out)
    torch.cuda.synchronize()
    return out.cpu().numpy()


def check(oracle, ro, ci, vals, B, M, N, out, tol=TOL / 50):
    assert not np.isnan(out).any()
    bad, worst = oracle.violations(oracle.spmm(vals, ro, ci, B, M, N), out, oracle.spmm_scale(vals, ro, ci, B, M, N), tol)
    assert bad == 0, worst


@pytest.mark.parametrize("M,K,N,density", [(16, 64, 64, 0.3), (17, 1, 64, 1.0), (64, 63, 132, 0.5), (127, 65, 256, 0.1), (128, 64, 260, 0.9),
                                           (129, 127, 252, 0.02), (300, 200, 516, 0.25), (31, 1000, 128, 1.0), (1000, 129, 68, 0.4)])
def test_tile_edges(pkg, oracle, ctx, dev, M, K, N, density):
    seed = M + K + N
    ro, ci = csr_bernoulli(pkg, M, K, density, seed)
    vals = pkg.gen_dense_host(int(ci.size), seed, 2)
    B = dense(pkg, K, N, seed, 10)
    check(oracle, ro, ci, vals, B, M, N, batch_run(pkg, ctx, dev, M, K, N, ro, ci, vals, B))


def test_row_lengths_around_the_lane_group(pkg, oracle, ctx, dev):
    """Empty and full rows, and rows of up to 64 entries inside one step in front of rows with none."""
    K, N = 256, 64
    lengths = [0, 1, 7, 8, 9, 15, 16, 17, 31, 33, 39, 40, 41, 63, 64, 65, 128, 255, 256, 0, 0, 3]
    ro, ci = csr_from_lengths(pkg, K, lengths, seed=3)
    ci[ro[12]:ro[13]] = np.arange(20, 20 + lengths[12])  # all in one step
    ci[ro[14]:ro[15]] = np.arange(64, 64 + lengths[14])
    vals = pkg.gen_dense_host(int(ci.size), 3, 2)
    B = dense(pkg, K, N, 3, 10)
    out = batch_run(pkg, ctx, dev, len(lengths), K, N, ro, ci, vals, B)
    check(oracle, ro, ci, vals, B, len(lengths), N, out)
    assert (out[[0, 19, 20]] == 0).all()


@pytest.mark.parametrize("M,K,N,density,order", [(1024, 2048, 512, 0.3, "sorted"), (1000, 2000, 510, 0.4, "sorted"),
                                                 (1024, 2048, 512, 0.3, "shuffled"), (2048, 512, 1028, 0.3, "doubled"),
                                                 (900, 4100, 301, 0.5, "sorted")])
def test_lone_launches(pkg, oracle, ctx, dev, M, K, N, density, order):
    """With and without parts of K in blocks of their own, aligned and ragged widths; columns out of order and
    repeated columns are found by the kernel."""
    seed = M + N
    ro, ci = csr_rowlen_normal(pkg, M, K, 1.0 - density, seed)
    if order == "shuffled":
        ci = shuffle_rows_columns(ro, ci, seed)
    if order == "doubled":
        ci[ro[5] + 1] = ci[ro[5]]
        ci[ro[70] + 9] = ci[ro[70] + 8]
    vals = pkg.gen_dense_host(int(ci.size), seed, 2)
    B = dense(pkg, K, N, seed, 10)
    check(oracle, ro, ci, vals, B, M, N, lone_run(ctx, dev, M, K, N, ro, ci, vals, B))
    check(oracle, ro, ci, vals, B, M, N, lone_run(ctx, dev, M, K, N, ro, ci, vals, B, plan=True))


def gather_run(ctx, dev, M, K, N, ro, ci, vals, B):
    """The row-gather kernel whatever the sizes: a plan made when no row was sorted (entries may be permuted inside rows since)."""
    import torch

    out = torch.full((M, N), float("nan"), device=dev)
    d = [to_dev(x, dev) for x in (vals, ro, ci, B)]
    p = ctx.plan_create(M, K, int(ci.size), d[1], to_dev(np.concatenate([ci[s:e][::-1] for s, e in zip(ro, ro[1:])]), dev))
    ctx.spmm_planned(p, N, *d, out)
    torch.cuda.synchronize()
    p.close()
    return out.cpu().numpy()


def looks_sorted(ro, ci, M):
    """The kernel's look at the order of columns: eight entries from the middle of 32 rows."""
    for row in (M * lane // 32 for lane in range(32)):
        start, end = int(ro[row]), int(ro[row + 1])
        c = ci[start + (end - start) // 2:end][:8]
        if (np.diff(c) <= 0).any():
            return False
    return True


@pytest.mark.parametrize("M,K,N", [(12900, 200, 1028), (9800, 200, 1029), (900, 4100, 300), (900, 4100, 301)])
def test_order_of_columns_is_seen_in_every_tile_of_a_lone_launch(pkg, oracle, ctx, dev, M, K, N):
    """More tiles for every pair of blocks than are planned ahead, and one tile in four parts of K, with 16- and 4-byte
    copies of B; empty rows among them.  Columns repeated at the start, in the middle and at the end of rows, rows that run
    backwards, and columns exchanged or repeated where the parts of K meet.  The rows that the kernel looks at before it
    multiplies are in order, so that no launch is left to its gather loop."""
    seed = M + N
    rng = np.random.default_rng(seed)
    lengths = rng.integers(K // 4, K // 2, M)
    lengths[rng.integers(0, M, M // 8)] = 0
    lengths[:3] = 0
    lengths[-1] = 0
    ro, ci = csr_from_lengths(pkg, K, [int(x) for x in lengths], seed=seed)
    chunks = -(-K // 64)
    seams = [64 * (chunks * part // 4) for part in (1, 2, 3)]
    looked_at = {M * lane // 32 for lane in range(32)}
    mixed = np.zeros(M, dtype=bool)
    for n, i in enumerate(i for i in range(M) if lengths[i] and i not in looked_at):
        start, end = int(ro[i]), int(ro[i + 1])
        at = {0: start, 1: start + int(lengths[i]) // 2, 2: end - 2}.get(n % 11)
        if n % 11 in (4, 5, 6):  # the last entry in front of a seam and the first one behind it
            at = start + int(np.searchsorted(ci[start:end], seams[n % 11 - 4])) - 1
            if not start <= at < end - 1:
                continue
        if n % 11 == 3:
            ci[start:end] = ci[start:end][::-1].copy()
        elif at is None:
            continue
        elif n % 22 in (4, 5, 6):
            ci[at], ci[at + 1] = ci[at + 1], ci[at]
        else:
            ci[at + 1] = ci[at]
        mixed[i] = True
    assert looks_sorted(ro, ci, M) and mixed.sum() > M // 3
    vals = pkg.gen_dense_host(int(ci.size), seed, 2)
    B = dense(pkg, K, N, seed, 10)
    out = lone_run(ctx, dev, M, K, N, ro, ci, vals, B)
    check(oracle, ro, ci, vals, B, M, N, out)
    assert (out[lengths == 0] == 0).all()
    # sums of split products do not have the bits of a chain of multiply-adds in a row of 50 entries and 300 columns or more
    gathered = gather_run(ctx, dev, M, K, N, ro, ci, vals, B)
    assert all((out[i] != gathered[i]).any() for i in range(M) if lengths[i] and not mixed[i]), "rows not multiplied"


def test_many_tiles_per_cluster(pkg, oracle, ctx, dev):
    """More tiles for every pair of blocks than are planned ahead, of problems of different sizes, as a prepared batch
    (columns known to ascend; the one-shot call: test_many_tiles_with_columns_out_of_order)."""
    import torch

    shapes = [(17 + 53 * i % 290, 40 + 31 * i % 90, 260 + 4 * (i % 3)) for i in range(120)]
    assert sum(-(-M // 128) * -(-N // 256) for M, K, N in shapes) > 5 * 74
    ctx.set_option(pkg.OPT_TILE_MIN_DENSITY, 0)
    try:
        arr, keep = pkg.ProblemArray(len(shapes)), []
        for i, (M, K, N) in enumerate(shapes):
            ro, ci = csr_bernoulli(pkg, M, K, 0.3, i)
            vals, B = pkg.gen_dense_host(int(ci.size), i, 2), dense(pkg, K, N, i, 10)
            out = torch.full((M * N,), float("nan"), device=dev)
            arr.set(i, M, K, N, int(ci.size), to_dev(vals, dev), to_dev(ro, dev), to_dev(ci, dev), to_dev(B, dev), out)
            keep.append((ro, ci, vals, B, out))
        batch = ctx.batch_create(arr)
        assert batch.info()[1] == len(shapes)
        batch.launch()
        torch.cuda.synchronize()
        for (M, K, N), (ro, ci, vals, B, out) in zip(shapes, keep):
            check(oracle, ro, ci, vals, B, M, N, out.cpu().numpy().reshape(M, N))
        batch.close()
    finally:
        ctx.set_option(pkg.OPT_TILE_MIN_DENSITY, -1)


@pytest.mark.parametrize("where", ["infinite", "tiny", "huge", "tiny rows", "tiny columns", "zeros", "zeros, one tiny"])
def test_numbers_that_cannot_be_split(pkg, oracle, ctx, dev, where):
    """Infinities and NaN reach the rows that refer to them and no others; magnitudes at the ends of the range keep
    their precision."""
    M, K, N = 300, 200, 512
    ro, ci = csr_rowlen_normal(pkg, M, K, 0.5, 4242)
    vals = pkg.gen_dense_host(int(ci.size), 4242, 2)
    B = dense(pkg, K, N, 4242, 10).copy()
    if where == "infinite":
        used = 130
        B[used, 5], B[used, 300] = np.nan, -np.inf
        out = batch_run(pkg, ctx, dev, M, K, N, ro, ci, vals, B)
        refers = np.array([used in ci[ro[i]:ro[i + 1]] for i in range(M)])
        assert refers.any() and not refers.all()
        assert np.isfinite(out[~refers]).all()
        assert np.isnan(out[refers][:, 5]).all() and np.isinf(out[refers][:, 300]).all()
        B[used, 5] = B[used, 300] = 0
        want = oracle.spmm(vals, ro, ci, B, M, N)
        keep = np.ones(N, bool)
        keep[[5, 300]] = False
        assert np.allclose(out[:, keep], want[:, keep], rtol=1e-4, atol=1e-4)
        return
    if where.startswith("tiny "):  # seen by one block of a pair only: a row of its half, columns of its half
        B *= np.float32(1e20)
        if where == "tiny rows":
            for i in (3, 77, 140, 260, 299):
                vals[ro[i]:ro[i + 1]] *= np.float32(1e-36)
        else:
            for _ in range(2):
                B[:, [3, 140, 141, 400]] *= np.float32(1e-28)
    elif where.startswith("zeros"):  # in some columns of B, so that the lanes of a warp part, in the last rows of it too
        B[np.arange(K)[:, None] % 5 == np.arange(N) % 7] = 0
        if where == "zeros, one tiny":
            B[K - 1, 77] = np.float32(1e-35)
    elif where == "tiny":
        vals = (vals * np.float32(1e-36)).astype(np.float32)
        B *= np.float32(1e20)
    else:
        B[7, 3] = np.float32(3.4e38)  # rounds to infinity as bf16
        vals *= np.float32(1e-3)
    check(oracle, ro, ci, vals, B, M, N, batch_run(pkg, ctx, dev, M, K, N, ro, ci, vals, B))


def test_problems_beyond_32_bit_offsets_stay_on_other_kernels(pkg, ctx, dev):
    """B of 2^30 elements and more, with a density threshold of the caller's (which takes the place of the estimate):
    the tensor-core kernel does not take a B of that size."""
    import torch

    M, K, N, per_row = 64, (1 << 21) + 64, 512, 60
    gen = torch.Generator(device=dev)
    gen.manual_seed(5)
    ci = torch.randint(0, K // per_row, (M, per_row), generator=gen, device=dev, dtype=torch.int32)
    ci += torch.arange(per_row, device=dev, dtype=torch.int32) * (K // per_row)  # ascending, over the whole range
    ci[:, -1] = K - 1 - torch.arange(M, device=dev, dtype=torch.int32)           # the last rows of B among them
    ro = torch.arange(0, M * per_row + 1, per_row, dtype=torch.int32, device=dev)
    vals = torch.rand(M * per_row, generator=gen, device=dev) - 0.5
    B = torch.rand(K, N, generator=gen, device=dev) - 0.5
    C = torch.full((M, N), float("nan"), device=dev)
    arr = pkg.ProblemArray(1)
    arr.set(0, M, K, N, M * per_row, vals, ro, ci.reshape(-1), B, C)
    ctx.set_option(pkg.OPT_TILE_MIN_DENSITY, 0)
    try:
        batch = ctx.batch_create(arr)
        batch.launch()
        torch.cuda.synchronize()
        assert batch.info(check_device=True)[2] == 0
        batch.close()
    finally:
        ctx.set_option(pkg.OPT_TILE_MIN_DENSITY, -1)
    v, rows = vals.reshape(M, per_row, 1).double(), B[ci.long()].double()
    want, scale = (v * rows).sum(1), (v * rows).abs().sum(1)
    assert ((C.double() - want).abs() <= TOL * scale).all()


@pytest.mark.parametrize("what", ["permuted", "permuted everywhere", "doubled", "other columns"])
def test_a_plan_does_not_keep_the_order_of_columns(pkg, oracle, ctx, dev, what):
    """A plan made of a sorted pattern, used after the columns inside rows have changed."""
    import torch

    M, K, N = 1024, 2048, 512
    ro, ci = csr_rowlen_normal(pkg, M, K, 0.7, 11)
    vals = pkg.gen_dense_host(int(ci.size), 11, 2)
    B = dense(pkg, K, N, 11, 10)
    d_ro = to_dev(ro, dev)
    p = ctx.plan_create(M, K, int(ci.size), d_ro, to_dev(ci, dev))
    if what.startswith("permuted"):
        other = shuffle_rows_columns(ro, ci, 3)
        for i in range(M):  # every 32nd row is one that the kernel looks at first
            if i % 32 or what == "permuted everywhere":
                ci[ro[i]:ro[i + 1]] = other[ro[i]:ro[i + 1]]
    elif what == "doubled":
        for i in range(0, M, 7):
            if ro[i + 1] - ro[i] > 3:
                ci[ro[i] + 1] = ci[ro[i]]
    else:
        ci = pkg.gen_sample_columns_host(M, K, ro, 12)
    out = torch.full((M, N), float("nan"), device=dev)
    ctx.spmm_planned(p, N, to_dev(vals, dev), d_ro, to_dev(ci, dev), to_dev(B, dev), out)
    torch.cuda.synchronize()
    p.close()
    check(oracle, ro, ci, vals, B, M, N, out.cpu().numpy())
