"""GPU PageRank (fmx_pagerank) against the oracle's restatement of
fm::alg::PageRank (matrix/libmatrix-algs/PageRank.cpp:63-133).

Bar: bit-identical ranks and the same iteration count when every vertex's
in-degree row has at most EXACT_ROW_MAX entries (all sums in the reference's
order); otherwise rows above that are summed in chunks, so ranks match within
RTOL = 1e-5 relative and the iteration count may differ by one.
"""
import numpy as np
import pytest

import oracle
from flashx_b200 import _lib, create_2d_matrix
from flashx_b200.algs import PageRank
from flashx_b200.graphs import rmat_edges

pytestmark = pytest.mark.gpu

RTOL = 1e-5


def _directed(n, m, seed):
    rng = np.random.default_rng(seed)
    return rng.integers(0, n, m).astype(np.uint32), rng.integers(0, n, m).astype(np.uint32)


@pytest.mark.parametrize("iters,damping", [(30, 0.85), (5, 0.5), (200, 0.85)])
def test_pagerank_bit_exact_on_short_rows(torch_cuda, iters, damping):
    n = 6000
    src, dst = _directed(n, 50000, 11)
    m, img, timg = create_2d_matrix(src, dst, None, block_size=(1024, 1024), is_sym=False, nrows=n, ncols=n,
                                    return_images=True)
    (idx, mat), (tidx, tmat) = img.bytes(), timg.bytes()
    assert np.bincount(dst, minlength=n).max() <= _lib.EXACT_ROW_MAX
    pr, it = PageRank(m, iters, damping)
    ref, rit = oracle.pagerank(idx, mat, tidx, tmat, iters, damping, nthreads=4)
    assert it == rit
    assert np.array_equal(pr.cpu().numpy(), ref)


def test_pagerank_rmat_s16_configuration(torch_cuda):
    """The reference's CPU configuration: R-MAT scale 16, 30 iterations at
    damping 0.85 (hub rows longer than EXACT_ROW_MAX are summed in chunks)."""
    from flashx_b200 import set_deduplicate
    n = 1 << 16
    src, dst = rmat_edges(16, seed=1)
    set_deduplicate(True)
    try:
        m, img, timg = create_2d_matrix(src, dst, None, block_size=(16384, 16384), is_sym=False, nrows=n, ncols=n,
                                        return_images=True)
    finally:
        set_deduplicate(False)
    (idx, mat), (tidx, tmat) = img.bytes(), timg.bytes()
    pr, it = PageRank(m, 30, 0.85)
    ref, rit = oracle.pagerank(idx, mat, tidx, tmat, 30, 0.85, nthreads=8)
    assert abs(it - rit) <= 1
    p = pr.cpu().numpy()
    np.testing.assert_allclose(p, ref, rtol=RTOL, atol=RTOL * float(ref.max()))
    assert abs(float(p.astype(np.float64).sum()) - float(ref.astype(np.float64).sum())) < 1e-4


def test_pagerank_errors(torch_cuda):
    from flashx_b200 import FmxError, matrix_image, sparse_matrix
    rect = sparse_matrix.create(matrix_image.build([0, 1], [1, 0], None, nrows=4, ncols=2, block_size=(2, 2)), None)
    with pytest.raises(FmxError) as e:
        PageRank(rect, 10, 0.85)
    assert e.value.code == _lib.FMX_ERR_DIM


def test_pagerank_fused_matches_stepwise_loop(torch_cuda):
    """The fused iteration (update applied where the SpMV closes a row, and
    in the fixup for chunked hub rows) against a host-driven loop of plain
    SpMVs on the transpose with the update in float32 numpy (one rounding per
    operation, as PageRank.cpp:100-123): bit-identical at R-MAT scale 16,
    whose hub rows go through the fixup, for an iteration cap below, at and
    above the point of convergence."""
    torch = torch_cuda
    from flashx_b200 import set_deduplicate
    n = 1 << 16
    src, dst = rmat_edges(16, seed=2)
    set_deduplicate(True)
    try:
        m = create_2d_matrix(src, dst, None, block_size=(16384, 16384), is_sym=False, nrows=n, ncols=n)
    finally:
        set_deduplicate(False)
    mt = m.transpose()
    assert mt.schedule()[2] > 0                   # heavy rows take the fixup path
    d = np.float32(0.85)
    deg = m.multiply(torch.ones((n, 1), device="cuda")).cpu().numpy()[:, 0]
    deg = np.maximum(deg, np.float32(1))
    tele = np.float32((1.0 - float(d)) / n)     # (1 - d) / n in double from the float d
    eps = np.float32(0.001 / n)
    pr = np.full(n, np.float32(1.0 / n), dtype=np.float32)
    x = pr / deg
    pr1 = x * deg
    ref_iters, ref = [], []
    it, conv = 0, 0
    while conv < n and it < 60:
        out = mt.multiply(torch.from_numpy(x).cuda().reshape(n, 1)).cpu().numpy()[:, 0]
        p2 = out * d + tele
        conv = int(np.count_nonzero(np.abs(pr1 - p2) < eps))
        pr = p2
        x = p2 / deg
        pr1 = x * deg
        it += 1
        ref.append(pr.copy())
    for cap in (3, 17, 60):
        got, git = PageRank(m, cap, 0.85)
        assert git == min(cap, it)
        assert np.array_equal(got.cpu().numpy(), ref[git - 1])


def test_workspace_pool_release(torch_cuda):
    """The solvers' workspace pool keeps freed memory for the next call;
    release_cached hands it back, and later calls still run."""
    torch = torch_cuda
    from flashx_b200 import release_cached
    n = 6000
    src, dst = _directed(n, 50000, 11)
    m = create_2d_matrix(src, dst, None, block_size=(1024, 1024), is_sym=False, nrows=n, ncols=n)
    p1, i1 = PageRank(m, 30, 0.85)
    release_cached(0)
    p2, i2 = PageRank(m, 30, 0.85)
    assert i1 == i2 and torch.equal(p1, p2)
    release_cached(0)


@pytest.mark.parametrize("n,m", [(6000, 50000), (300000, 2000000)])
def test_pagerank_repeats_bit_exact(torch_cuda, n, m):
    """Iterations overlap their neighbours' launches; both forms (a warp per
    range; the row kernel beyond 64 ranges per SM) must read only finished
    vectors, every time."""
    src, dst = _directed(n, m, 12)
    mat, img, timg = create_2d_matrix(src, dst, None, block_size=(16384, 16384), is_sym=False, nrows=n, ncols=n,
                                      return_images=True)
    (idx, im), (tidx, tim) = img.bytes(), timg.bytes()
    assert np.bincount(dst, minlength=n).max() <= _lib.EXACT_ROW_MAX
    ref, rit = oracle.pagerank(idx, im, tidx, tim, 12, 0.85, nthreads=4)
    for _ in range(20):
        pr, it = PageRank(mat, 12, 0.85)
        assert it == rit
        assert np.array_equal(pr.cpu().numpy(), ref)


def test_pagerank_from_ending_threads(torch_cuda):
    """The loop state's pinned words belong to a thread and go with it."""
    import threading
    src, dst = _directed(3000, 20000, 13)
    m = create_2d_matrix(src, dst, None, block_size=(1024, 1024), is_sym=False, nrows=3000, ncols=3000)
    ref, rit = PageRank(m, 20, 0.85)
    ref = ref.cpu().numpy()
    got = []

    def run():
        pr, it = PageRank(m, 20, 0.85)
        got.append((pr.cpu().numpy(), it))

    for _ in range(4):
        t = threading.Thread(target=run)
        t.start()
        t.join()
    assert len(got) == 4
    for pr, it in got:
        assert it == rit and np.array_equal(pr, ref)


def _stepwise(torch, m, n, most):
    """The ranks after each iteration of a host-driven loop of plain SpMVs
    with the update in float32 numpy, until it converges (or `most`)."""
    mt = m.transpose()
    d = np.float32(0.85)
    deg = np.maximum(m.multiply(torch.ones((n, 1), device="cuda")).cpu().numpy()[:, 0], np.float32(1))
    tele, eps = np.float32((1.0 - float(d)) / n), np.float32(0.001 / n)
    x = np.full(n, np.float32(1.0 / n), dtype=np.float32) / deg
    pr1 = x * deg
    ref, conv = [], 0
    while conv < n and len(ref) < most:
        p2 = mt.multiply(torch.from_numpy(x).cuda().reshape(n, 1)).cpu().numpy()[:, 0] * d + tele
        conv = int(np.count_nonzero(np.abs(pr1 - p2) < eps))
        x = p2 / deg
        pr1 = x * deg
        ref.append(p2)
    return ref, conv == n


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("streamed", [False, True])
def test_pagerank_row_kernel_form(torch_cuda, weighted, streamed):
    """Beyond 64 ranges per SM an iteration is the row kernel, the fixup of
    chunked rows and a pass of updates, the latter two dependent launches: the
    stepwise loop's bits and counts for caps below, at and far above the point
    of convergence (iterations queued after it must change nothing), several
    times over."""
    torch = torch_cuda
    from flashx_b200 import matrix_image, sparse_matrix
    n = 1 << 18
    src, dst = rmat_edges(18, seed=5)
    w = np.random.default_rng(3).uniform(0.5, 1, len(src)).astype(np.float32) if weighted else None
    img = matrix_image.build(src, dst, w, nrows=n, ncols=n, block_size=(16384, 16384), dedup=True)
    timg = matrix_image.build(dst, src, w, nrows=n, ncols=n, block_size=(16384, 16384), dedup=True)
    m = sparse_matrix.create(img, timg)
    assert m.transpose().schedule()[2] > 0        # rows summed in chunks
    ref, ended = _stepwise(torch, m, n, 100)
    assert ended
    if streamed:
        m = sparse_matrix.create_streamed(img, timg, slice_entries=1 << 20)
    for cap in (3, len(ref), 200, 200, 17, 200):
        got, git = PageRank(m, cap, 0.85)
        assert git == min(cap, len(ref))
        assert np.array_equal(got.cpu().numpy(), ref[git - 1])


@pytest.mark.parametrize("n,m,streamed", [(100_000, 1_600_000, False), (1 << 20, 16 << 20, False), (1 << 18, 4 << 20, True)])
def test_pagerank_ends_with_convergence(torch_cuda, n, m, streamed):
    """A uniform graph converges in a few iterations: a cap far above that
    costs little more than a cap at it (the batch that is queued when the loop
    ends runs empty; a streamed matrix copies its entries in it), in all forms
    of the iteration.  Whole queued iterations would make the ratio 2 or more."""
    import time
    torch = torch_cuda
    from flashx_b200 import matrix_image, sparse_matrix
    src, dst = _directed(n, m, 14)
    if streamed:
        img = matrix_image.build(src, dst, None, nrows=n, ncols=n, block_size=(16384, 16384), dedup=True)
        timg = matrix_image.build(dst, src, None, nrows=n, ncols=n, block_size=(16384, 16384), dedup=True)
        a = sparse_matrix.create_streamed(img, timg, slice_entries=1 << 19)
    else:
        s, d = (torch.from_numpy(x.astype(np.int32)).cuda() for x in (src, dst))
        a = sparse_matrix.from_device_edges(s, d, None, nrows=n, ncols=n, dedup=True, transpose=True)
    p1, it = PageRank(a, 200, 0.85)
    assert it <= 8                                # within the first batch
    p2, it2 = PageRank(a, it, 0.85)
    assert it2 == it and torch.equal(p1, p2)

    def best(cap):
        t = []
        for _ in range(7):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            PageRank(a, cap, 0.85)
            t.append(time.perf_counter() - t0)
        return min(t)

    best(it)
    assert best(200) <= 1.5 * best(it)


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("hub", [300, 4000, 30000])
def test_pagerank_warp_form_hubs(torch_cuda, hub, weighted):
    """A warp per range: a row of 2, 16 or 118 chunks (up to 8, up to 64 and more
    are added by 2, 32 and 256 parts), finished by the warp whose chunk arrives
    last, has the bits of the product's fixup kernel, weighted or not, and so has
    the whole loop."""
    torch = torch_cuda
    from flashx_b200 import matrix_image, sparse_matrix
    n = 40000
    rng = np.random.default_rng(hub)
    src, dst = _directed(n, 150000, hub)
    for row, deg in ((7, hub), (39999, hub // 2 + 150)):
        src = np.concatenate([src, rng.choice(n, deg, replace=False).astype(np.uint32)])
        dst = np.concatenate([dst, np.full(deg, row, dtype=np.uint32)])
    # ranges: at most one run per 128 entries and the hubs' chunks
    assert (len(dst) + n) // 128 + 400 <= 64 * torch.cuda.get_device_properties(0).multi_processor_count
    w = rng.uniform(0.5, 1, len(src)).astype(np.float32) if weighted else None
    img = matrix_image.build(src, dst, w, nrows=n, ncols=n, block_size=(16384, 16384), dedup=True)
    timg = matrix_image.build(dst, src, w, nrows=n, ncols=n, block_size=(16384, 16384), dedup=True)
    m = sparse_matrix.create(img, timg)
    ref, ended = _stepwise(torch, m, n, 100)
    assert ended
    for cap in (1, 5, 200, 200):
        got, git = PageRank(m, cap, 0.85)
        assert git == min(cap, len(ref))
        assert np.array_equal(got.cpu().numpy(), ref[git - 1])
