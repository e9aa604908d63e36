"""GPU parity: libfmx's CUDA SpMM against the CPU oracle on the same image.

Bar: bit-exact for integer types and for every row summed by one lane group
(rows of <= EXACT_ROW_MAX = 256 entries are summed in the reference's ascending-column order
with separate multiply and add roundings); bit-exact for split rows when the
inputs are integer-valued (all partial sums exact); otherwise within
RTOL = 1e-5 relative (FP32) of the oracle.
"""
import numpy as np
import pytest

import oracle
from flashx_b200 import release_cached, _lib, matrix_image, sparse_matrix, create_2d_matrix
from flashx_b200.graphs import rmat_edges

pytestmark = pytest.mark.gpu

RTOL = 1e-5


def _graph(n, m, seed, heavy=()):
    rng = np.random.default_rng(seed)
    src = rng.integers(0, n, m).astype(np.uint32)
    dst = rng.integers(0, n, m).astype(np.uint32)
    extra_s, extra_d = [], []
    for row, deg in heavy:
        assert deg <= n, "a row cannot hold more distinct columns than the matrix has"
        extra_s.append(np.full(deg, row, dtype=np.uint32))
        extra_d.append(rng.choice(n, deg, replace=False).astype(np.uint32))
    if heavy:
        src = np.concatenate([src] + extra_s)
        dst = np.concatenate([dst] + extra_d)
    return src, dst


def _dense(rng, shape, dt, integer=False):
    if dt in (np.int32, np.int64) or integer:
        return rng.integers(-8, 9, shape).astype(dt)
    return rng.standard_normal(shape).astype(dt)


def _to_torch(torch, a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _gpu_spmm(torch, m, X, out_dtype=None, s_in=None, s_out=None):
    x = _to_torch(torch, X)
    y = torch.empty((m.get_num_rows(), X.shape[1]), dtype=out_dtype or x.dtype, device="cuda")
    y.fill_(float("nan") if y.dtype.is_floating_point else -7)
    si = _to_torch(torch, s_in) if s_in is not None else None
    so = _to_torch(torch, s_out) if s_out is not None else None
    assert m.multiply(x, y, si, so), _lib.last_error()
    torch.cuda.synchronize()
    return y.float().cpu().numpy() if y.dtype == torch.bfloat16 else y.cpu().numpy()


CASES = [
    # n, m, block, weighted dtype, dedup, heavy rows (row, degree)
    (1000, 6000, (64, 128), None, False, ()),
    (5000, 60000, (1024, 1024), np.float32, True, ()),
    (20000, 100000, (16384, 16384), None, True, ((7, 20000), (11, 900), (13, 600))),
    (20000, 100000, (4096, 2048), np.float32, False, ((3, 17000), (5, 5000))),
    (3000, 20000, (256, 256), np.float64, True, ((1, 2999),)),
]


@pytest.mark.parametrize("case", range(len(CASES)))
@pytest.mark.parametrize("k", [1, 2, 3, 4, 8, 10, 16, 32, 64, 130])
def test_parity_float(torch_cuda, case, k):
    torch = torch_cuda
    n, mm, block, wdt, dedup, heavy = CASES[case]
    src, dst = _graph(n, mm, 100 + case, heavy)
    rng = np.random.default_rng(case * 1000 + k)
    vals = None if wdt is None else rng.uniform(0.0, 1.0, len(src)).astype(wdt)
    idx, mat = oracle.build_image(src, dst, vals, block=block, dedup=dedup)
    img = matrix_image.from_bytes(idx, mat)
    m = sparse_matrix.create(img, None, device=0)
    dt = np.float64 if wdt is np.float64 else np.float32
    has_split = any(d > _lib.EXACT_ROW_MAX for _, d in heavy)
    for integer in (True, False):
        X = _dense(rng, (n, k), dt, integer)
        Y = _gpu_spmm(torch, m, X)
        R = oracle.spmm(idx, mat, X, nthreads=4)
        if not has_split or (integer and wdt is None):
            bad = np.argwhere(Y.view(np.uint32 if Y.dtype == np.float32 else np.uint64)
                              != R.view(np.uint32 if R.dtype == np.float32 else np.uint64))
            assert len(bad) == 0, (
                f"not bit-exact at {len(bad)} elements (first {bad[:5].tolist()}): "
                f"max diff {np.max(np.abs(Y - R))}")
        else:
            np.testing.assert_allclose(Y, R, rtol=RTOL, atol=RTOL * np.abs(R).max())


@pytest.mark.parametrize("dt", [np.int32, np.int64])
@pytest.mark.parametrize("k", [1, 4, 5, 16])
def test_parity_integer(torch_cuda, dt, k):
    torch = torch_cuda
    src, dst = _graph(30000, 150000, 7, ((2, 20000), (9, 3000)))
    rng = np.random.default_rng(k)
    vals = rng.integers(-3, 4, len(src)).astype(np.int32 if dt is np.int32 else np.int64)
    for w in (None, vals):
        idx, mat = oracle.build_image(src, dst, w, block=(2048, 2048), dedup=True)
        m = sparse_matrix.create(matrix_image.from_bytes(idx, mat), None)
        X = rng.integers(-1000, 1000, (30000, k)).astype(dt)
        assert np.array_equal(_gpu_spmm(torch, m, X), oracle.spmm(idx, mat, X))


def test_rand_mat_gen_known_answer(torch_cuda):
    """matrix/test/rand_mat_gen.cpp:178-199: a binary matrix times
    [0, 1, ..., ncol-1] equals each row's sum of column ids (duplicates kept)."""
    torch = torch_cuda
    rng = np.random.default_rng(11)
    nrow, ncol = 30000, 20000
    deg = rng.integers(0, 60, nrow)
    src = np.repeat(np.arange(nrow, dtype=np.uint32), deg)
    dst = rng.integers(0, ncol, len(src)).astype(np.uint32)
    m = create_2d_matrix(src, dst, None, block_size=(4096, 4096), nrows=nrow, ncols=ncol)
    X = np.arange(ncol, dtype=np.int64)[:, None]
    Y = _gpu_spmm(torch, m, X)[:, 0]
    keep = src != dst
    expect = np.bincount(src[keep], weights=dst[keep].astype(np.float64), minlength=nrow).astype(np.int64)
    assert np.array_equal(Y, expect)


def test_bf16_input(torch_cuda):
    torch = torch_cuda
    src, dst = _graph(8000, 80000, 3)
    idx, mat = oracle.build_image(src, dst, None, block=(4096, 4096), dedup=True)
    m = sparse_matrix.create(matrix_image.from_bytes(idx, mat), None)
    rng = np.random.default_rng(5)
    for k in (8, 16, 32, 6):
        Xf = rng.standard_normal((8000, k)).astype(np.float32)
        xb = torch.from_numpy(Xf).to(torch.bfloat16).cuda()
        Xr = xb.float().cpu().numpy()          # the bf16-rounded operand
        y = torch.empty((8000, k), dtype=torch.float32, device="cuda")
        assert m.multiply(xb, y)
        R = oracle.spmm(idx, mat, Xr)
        assert np.array_equal(y.cpu().numpy(), R)
        yb = torch.empty((8000, k), dtype=torch.bfloat16, device="cuda")
        assert m.multiply(xb, yb)
        assert torch.equal(yb.cpu(), torch.from_numpy(R).to(torch.bfloat16))


def test_row_scales(torch_cuda):
    """y = D_out A D_in x, the normalised-adjacency operator of
    matrix/test/test-eigen.cpp:88-136 (scale_rows, SpMM, scale_rows)."""
    torch = torch_cuda
    n = 30000
    src, dst = _graph(n, 200000, 9, ((4, 18000), (8, 2000)))
    idx, mat = oracle.build_image(src, dst, None, block=(8192, 8192), dedup=True)
    m = sparse_matrix.create(matrix_image.from_bytes(idx, mat), None)
    rng = np.random.default_rng(2)
    for dt in (np.float32, np.float64):
        X = rng.standard_normal((n, 16)).astype(dt)
        s_in = rng.uniform(0.1, 2.0, n).astype(dt)
        s_out = rng.uniform(0.1, 2.0, n).astype(dt)
        Y = _gpu_spmm(torch, m, X, s_in=s_in, s_out=s_out)
        R = oracle.spmm(idx, mat, (X * s_in[:, None]).astype(dt)) * s_out[:, None]
        np.testing.assert_allclose(Y, R, rtol=RTOL if dt == np.float32 else 1e-12,
                                   atol=(RTOL if dt == np.float32 else 1e-12) * np.abs(R).max())
    # BF16 in and out with both scales (the eigensolver's correction SpMMs):
    # FP32 accumulation of the BF16-rounded operand, one BF16 rounding at the end
    s_in = rng.uniform(0.1, 2.0, n).astype(np.float32)
    s_out = rng.uniform(0.1, 2.0, n).astype(np.float32)
    for k in (16, 32, 8):
        xb = torch.from_numpy(rng.standard_normal((n, k)).astype(np.float32)).to(torch.bfloat16).cuda()
        yb = torch.empty((n, k), dtype=torch.bfloat16, device="cuda")
        assert m.multiply(xb, yb, torch.from_numpy(s_in).cuda(), torch.from_numpy(s_out).cuda())
        Xr = xb.float().cpu().numpy()
        R = (oracle.spmm(idx, mat, (Xr * s_in[:, None]).astype(np.float32)) * s_out[:, None]).astype(np.float32)
        got = yb.float().cpu().numpy()
        np.testing.assert_allclose(got, R, rtol=1e-2, atol=1e-2 * np.abs(R).max())


def test_asymmetric_transpose(torch_cuda):
    torch = torch_cuda
    rng = np.random.default_rng(4)
    src = rng.integers(0, 4000, 30000).astype(np.uint32)
    dst = rng.integers(0, 4000, 30000).astype(np.uint32)
    m, img, timg = create_2d_matrix(src, dst, None, block_size=(1024, 1024), is_sym=False, return_images=True)
    assert not m.is_symmetric()
    X = rng.integers(-8, 9, (m.get_num_cols(), 8)).astype(np.float32)
    t = m.transpose()
    i, a = img.bytes()
    ti, ta = timg.bytes()
    assert np.array_equal(_gpu_spmm(torch, m, X), oracle.spmm(i, a, X))
    assert np.array_equal(_gpu_spmm(torch, t, X), oracle.spmm(ti, ta, X))


def test_rmat_s18_parity(torch_cuda):
    torch = torch_cuda
    src, dst = rmat_edges(18, seed=1)
    rng = np.random.default_rng(0)
    for weighted in (False, True):
        vals = rng.uniform(0.0, 1.0, len(src)).astype(np.float32) if weighted else None
        vals = None if vals is None else np.where(vals == 0, np.float32(1.0), vals)
        img = matrix_image.build(src, dst, vals, nrows=1 << 18, ncols=1 << 18, block_size=(16384, 16384),
                                 dedup=True)
        idx, mat = img.bytes()
        m = sparse_matrix.create(img, None)
        rows, _ = oracle.nonzeros(idx, mat)
        light = np.bincount(rows.astype(np.int64), minlength=1 << 18) <= _lib.EXACT_ROW_MAX
        assert not light.all()     # the hubs exercise the split paths
        for k in (1, 4, 16, 32):
            Xi = rng.integers(-8, 9, (1 << 18, k)).astype(np.float32)
            Y, R = _gpu_spmm(torch, m, Xi), oracle.spmm(idx, mat, Xi, nthreads=8)
            if weighted:   # split rows re-associate non-integer products
                assert np.array_equal(Y[light], R[light])
                np.testing.assert_allclose(Y, R, rtol=RTOL, atol=RTOL * np.abs(R).max())
            else:
                assert np.array_equal(Y, R)
            Xf = rng.standard_normal((1 << 18, k)).astype(np.float32)
            Y, R = _gpu_spmm(torch, m, Xf), oracle.spmm(idx, mat, Xf, nthreads=8)
            assert np.array_equal(Y[light], R[light])
            np.testing.assert_allclose(Y, R, rtol=RTOL, atol=RTOL * np.abs(R).max())


@pytest.mark.parametrize("dtype", ["float32", "float64"])
def test_spmv_kernel_matches_lane_group_kernel(torch_cuda, dtype):
    """k = 1 without row scales runs the warp-per-range SpMV kernel; with row
    scales of exactly 1 (x * 1 and y * 1 are exact) it runs the lane-group
    kernel.  Rows of up to EXACT_ROW_MAX entries have the same arithmetic in
    both and must agree bit for bit; hub rows (chunks added up in another
    association) within RTOL."""
    torch = torch_cuda
    tdt = getattr(torch, dtype)
    n = 1 << 17
    src, dst = rmat_edges(17, seed=4)
    rng = np.random.default_rng(1)
    ones = torch.ones(n, device="cuda", dtype=tdt)
    for weighted in (False, True):
        vals = rng.uniform(0.0, 1.0, len(src)).astype(np.float32) if weighted else None
        m = sparse_matrix.create(matrix_image.build(src, dst, vals, nrows=n, ncols=n, block_size=(16384, 16384),
                                                    dedup=True), None)
        assert m.schedule()[2] > 0
        light = torch.from_numpy(np.bincount(src[src != dst].astype(np.int64), minlength=n) <= _lib.EXACT_ROW_MAX)
        X = torch.randn((n, 1), device="cuda", dtype=tdt)
        Y1 = m.multiply(X)
        Ys = torch.empty_like(Y1)
        assert m.multiply(X, Ys, row_scale_in=ones, row_scale_out=ones)
        y1, ys = Y1.cpu()[:, 0], Ys.cpu()[:, 0]
        assert torch.equal(y1[light], ys[light]) and not bool(light.all())
        torch.testing.assert_close(y1, ys, rtol=RTOL, atol=RTOL * float(ys.abs().max()))
        # a strided single column (ldx = ldy = 3)
        X3 = torch.zeros((n, 3), device="cuda", dtype=tdt)
        X3[:, :1] = X
        Y3 = torch.full((n, 3), 7.0, device="cuda", dtype=tdt)
        assert m.multiply(X3[:, :1], Y3[:, :1])
        assert torch.equal(Y3[:, :1], Y1) and bool((Y3[:, 1:] == 7).all())


@pytest.mark.parametrize("dtype", ["float32", "float64", "int32", "int64", "bfloat16"])
@pytest.mark.parametrize("k", [2, 3, 5, 7, 12, 15, 24, 31, 32, 33, 40, 65])
def test_lane_widths(torch_cuda, dtype, k):
    """Every lane width and remainder of the row kernel: whole and odd panels,
    operands that start off the vector grid (a column slice of a wider
    block), rows of 0 to 256 entries, with and without row scales.  Integer
    operands and power-of-two scales keep every sum exact, so each element
    must equal the oracle's."""
    torch = torch_cuda
    tdt = getattr(torch, dtype)
    n = 3001
    src, dst = _graph(n, 15000, 40 + k, ((5, 256), (2999, 255), (77, 8), (78, 9)))
    idx, mat = oracle.build_image(src, dst, None, block=(1024, 1024), dedup=True)
    m = sparse_matrix.create(matrix_image.from_bytes(idx, mat), None, device=0)
    rng = np.random.default_rng(k)
    X = rng.integers(-8, 9, (n, k))
    R = oracle.spmm(idx, mat, X.astype(np.float64))
    scales = [(None, None)]
    if tdt.is_floating_point:
        s = np.ldexp(1.0, rng.integers(-2, 3, n))
        sdt = torch.float64 if tdt == torch.float64 else torch.float32
        sc = torch.from_numpy(s).to("cuda", sdt)
        scales += [(sc, None), (None, sc), (sc, sc)]
    for off, pad in ((0, 0), (1, 2), (4, 4)):
        Xw = torch.zeros((n, off + k + pad), dtype=tdt, device="cuda")
        Xw[:, off:off + k] = torch.from_numpy(X).to("cuda", tdt)
        for si, so in scales:
            Yw = torch.full((n, off + k + pad), 77, dtype=torch.float32 if tdt == torch.bfloat16 else tdt, device="cuda")
            assert m.multiply(Xw[:, off:off + k], Yw[:, off:off + k], si, so), _lib.last_error()
            want = R
            if si is not None:
                want = oracle.spmm(idx, mat, X * s[:, None])
            if so is not None:
                want = want * s[:, None]
            got = Yw.cpu().double().numpy()
            assert np.array_equal(got[:, off:off + k], want), (off, si is not None, so is not None)
            assert (got[:, :off] == 77).all() and (got[:, off + k:] == 77).all()


@pytest.mark.parametrize("k,dtype,wdt", [(16, np.float32, None), (16, np.float32, np.float32), (12, np.float32, None),
                                         (8, np.float64, None), (10, np.float32, None), (4, np.int64, np.int64)])
@pytest.mark.parametrize("per_group", [20, 30, 50])
def test_lane_steps(torch_cuda, per_group, k, dtype, wdt):
    """The row kernel takes 32, 16 or 8 entries a step by the entries per lane
    group of the machine (lines at 24 and 40); integer values keep every sum
    exact, so all elements equal the oracle's, in rows of 0 to 256 entries and
    in one longer row."""
    torch = torch_cuda
    lanes = k * np.dtype(dtype).itemsize // (8 if k == 10 else 16)
    mm = per_group * 148 * 24 * (32 // lanes)
    n = 20000
    src, dst = _graph(n, mm, per_group + k, ((5, 256), (19999, 255), (77, 9000)))
    vals = None if wdt is None else np.random.default_rng(k).integers(1, 5, len(src)).astype(wdt)
    idx, mat = oracle.build_image(src, dst, vals, block=(16384, 16384), dedup=True)
    m = sparse_matrix.create(matrix_image.from_bytes(idx, mat), None)
    X = _dense(np.random.default_rng(k), (n, k), dtype, integer=True)
    assert np.array_equal(_gpu_spmm(torch, m, X), oracle.spmm(idx, mat, X))


def test_host_buffers_e2e(torch_cuda):
    src, dst = _graph(5000, 40000, 21)
    idx, mat = oracle.build_image(src, dst, None, block=(1024, 1024), dedup=True)
    m = sparse_matrix.create(matrix_image.from_bytes(idx, mat), None)
    X = np.random.default_rng(1).integers(-8, 9, (5000, 16)).astype(np.float32)
    assert np.array_equal(m.multiply_host(X), oracle.spmm(idx, mat, X))


@pytest.mark.parametrize("n,k,pad,dtype", [(70001, 5, 0, "float32"), (70001, 5, 3, "float32"), (262144, 1, 0, "float64"),
                                           (33333, 33, 7, "float64"), (1 << 18, 16, 0, "float32"), (150000, 2, 1, "int32")])
def test_host_buffers_through_pinned_slots(torch_cuda, n, k, pad, dtype):
    """Pageable operands of more than 1 MB go through pinned slots on several
    threads: chunk remainders, strided rows, repeated calls, calls of two
    threads at once (the second copies directly) and after the slots were
    handed back, each equal to the device product bit for bit."""
    import threading
    torch = torch_cuda
    src, dst = _graph(n, 4 * n, 31)
    mats = [sparse_matrix.create(matrix_image.build(src, dst, None, nrows=n, ncols=n, dedup=True), None)
            for _ in range(2)]
    code = {"float32": _lib.F32, "float64": _lib.F64, "int32": _lib.I32}[dtype]
    rng = np.random.default_rng(n)
    X = _dense(rng, (n, k + pad), np.dtype(dtype).type)
    want = mats[0].multiply(torch.from_numpy(np.ascontiguousarray(X[:, :k])).cuda()).cpu().numpy()
    got = [np.full((n, k + pad), 7, dtype=dtype) for _ in range(4)]

    def call(m, y):
        rc = _lib.lib.fmx_spmm_host(m.handle, code, X.ctypes.data, k + pad, code, y.ctypes.data, k + pad, k)
        assert rc == _lib.FMX_OK, _lib.last_error()

    call(mats[0], got[0])
    release_cached(0)
    call(mats[0], got[1])
    th = [threading.Thread(target=call, args=(m, y)) for m, y in zip(mats, got[2:])]
    for t in th:
        t.start()
    for t in th:
        t.join()
    for y in got:
        assert np.array_equal(y[:, :k], want) and (y[:, k:] == 7).all()


def test_host_buffers_async_two_streams(torch_cuda):
    """fmx_spmm_host_async: six calls in flight on two streams, each with its
    own pinned X and Y, through the matrix's two staging slots; every Y equals
    the oracle's (integer-valued X, so exact), and so does a later call on a
    third stream."""
    torch = torch_cuda
    src, dst = _graph(20000, 100000, 23, ((7, 15000), (11, 900)))
    idx, mat = oracle.build_image(src, dst, None, block=(4096, 4096), dedup=True)
    m = sparse_matrix.create(matrix_image.from_bytes(idx, mat), None)
    rng = np.random.default_rng(5)
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    xs, ys, want = [], [], []
    for i in range(6):
        x = torch.from_numpy(rng.integers(-8, 9, (20000, 16)).astype(np.float32)).pin_memory()
        y = torch.full((20000, 16), float("nan")).pin_memory()
        xs.append(x)
        ys.append(y)
        want.append(oracle.spmm(idx, mat, x.numpy()))
    for i in range(6):
        m.multiply_host_async(xs[i].numpy(), ys[i].numpy(), streams[i % 2].cuda_stream)
    for s in streams:
        s.synchronize()
    for i in range(6):
        assert np.array_equal(ys[i].numpy(), want[i]), i
    del streams
    s3 = torch.cuda.Stream()
    y3 = torch.full((20000, 16), float("nan")).pin_memory()
    m.multiply_host_async(xs[0].numpy(), y3.numpy(), s3.cuda_stream)
    s3.synchronize()
    assert np.array_equal(y3.numpy(), want[0])


def test_multiply_errors(torch_cuda):
    """Dimension and type mismatches return False, like the reference."""
    torch = torch_cuda
    src, dst = _graph(1000, 5000, 1)
    m = create_2d_matrix(src, dst, None, block_size=(256, 256), nrows=1000, ncols=1000)
    x = torch.zeros((999, 4), device="cuda")
    y = torch.zeros((1000, 4), device="cuda")
    assert not m.multiply(x, y)
    x = torch.zeros((1000, 4), device="cuda")
    assert not m.multiply(x, torch.zeros((1000, 4), dtype=torch.float64, device="cuda"))
    assert m.multiply(x, y)


def test_repeated_calls_varying_k(torch_cuda):
    """Scratch reuse: one matrix multiplied repeatedly with panel widths that
    shrink and grow (k = 130 ends with a 2-column panel) stays exact."""
    torch = torch_cuda
    src, dst = _graph(3000, 30000, 17)
    idx, mat = oracle.build_image(src, dst, None, block=(512, 1024), dedup=False)
    m = sparse_matrix.create(matrix_image.from_bytes(idx, mat), None)
    rng = np.random.default_rng(9)
    for k in (130, 32, 2, 64, 130, 16, 1, 33, 16):
        X = rng.integers(-8, 9, (3000, k)).astype(np.float32)
        for _ in range(2):
            assert np.array_equal(_gpu_spmm(torch, m, X), oracle.spmm(idx, mat, X))


@pytest.mark.parametrize("n,k,dtype", [(3000, 16, "float32"), (3000, 1, "float32"), (3000, 7, "float64"),
                                       (200000, 16, "float32"), (200000, 1, "float32")])
def test_graph_capture(torch_cuda, n, k, dtype):
    """A product captured in a CUDA graph (its kernels are dependent launches
    where they are short) replays on new operands with the eager results."""
    torch = torch_cuda
    src, dst = _graph(n, 12 * n, 51, ((7, 1500), (9, 600)))
    m = sparse_matrix.create(matrix_image.build(src, dst, None, nrows=n, ncols=n, dedup=True), None)
    g = torch.Generator(device="cuda").manual_seed(k)
    x = torch.randn((n, k), generator=g, device="cuda", dtype=getattr(torch, dtype))
    y = torch.empty_like(x)
    assert m.multiply(x, y)                       # the kernels' first use: outside the capture
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        assert m.multiply(x, y)
        assert m.multiply(y, x)
    for seed in (1, 2):
        x0 = torch.randn(x.shape, generator=g, device="cuda", dtype=x.dtype)
        x.copy_(x0)
        graph.replay()
        torch.cuda.synchronize()
        y1 = m.multiply(x0)
        assert torch.equal(y, y1) and torch.equal(x, m.multiply(y1))


def test_empty_matrix(torch_cuda):
    """A matrix without edges (every block row stored as one empty tile) gives
    Y = 0, overwriting whatever Y held."""
    torch = torch_cuda
    e = np.zeros(0, dtype=np.uint32)
    idx, mat = oracle.build_image(e, e, None, nrows=64, ncols=64, block=(16, 16))
    m = sparse_matrix.create(matrix_image.from_bytes(idx, mat), None)
    assert m.get_nnz() == 0
    for k in (1, 16):
        X = np.ones((64, k), dtype=np.float32)
        Y = _gpu_spmm(torch, m, X)
        assert np.array_equal(Y, oracle.spmm(idx, mat, X)) and not Y.any()


@pytest.fixture(scope="module")
def rmat_s24():
    """The bench graph: R-MAT scale 24, edge factor 16, seed 1, deduplicated,
    self-loops removed, 16384 x 16384 tiles; unweighted and uniform(0,1]
    weighted images of the same edges."""
    src, dst = rmat_edges(24, seed=1)
    n = 1 << 24
    vals = np.random.default_rng(24).uniform(0.0, 1.0, len(src)).astype(np.float32)
    vals[vals == 0] = 1.0
    out = {}
    for name, v in (("binary", None), ("weighted", vals)):
        img = matrix_image.build(src, dst, v, nrows=n, ncols=n, block_size=(16384, 16384), dedup=True)
        out[name] = img
    del src, dst, vals
    idx, mat = out["binary"].bytes()
    rows, cols = oracle.nonzeros(idx, mat)
    out["outdeg"] = np.bincount(rows.astype(np.int64), minlength=n)
    out["indeg"] = np.bincount(cols.astype(np.int64), minlength=n)
    return out


@pytest.mark.parametrize("k", [1, 4, 16, 32])
def test_rmat_s24_properties(torch_cuda, rmat_s24, k):
    """Full-size checks on the bench graph, unweighted: A 1 = out-degrees;
    A (X + Z) = A X + A Z bit for bit (integer-valued operands keep every
    partial sum exact); the checksum of checksums 1^T (A X) = indeg^T X; and
    bit-exact agreement with the oracle on a sample of block rows."""
    torch = torch_cuda
    img = rmat_s24["binary"]
    m = sparse_matrix.create(img, None)
    n = m.get_num_rows()
    assert m.get_nnz() == int(rmat_s24["outdeg"].sum())
    assert 8 * int(rmat_s24["outdeg"].max()) < (1 << 24)
    ones = torch.ones((n, k), device="cuda")
    y = torch.empty((n, k), device="cuda")
    assert m.multiply(ones, y)
    deg = torch.from_numpy(rmat_s24["outdeg"].astype(np.float32)).cuda()
    assert torch.equal(y, deg[:, None].expand(n, k))
    g = torch.Generator(device="cuda").manual_seed(k)
    X = torch.randint(-4, 5, (n, k), generator=g, device="cuda").float()
    Z = torch.randint(-4, 5, (n, k), generator=g, device="cuda").float()
    yx, yz, ys = (torch.empty((n, k), device="cuda") for _ in range(3))
    assert m.multiply(X, yx) and m.multiply(Z, yz) and m.multiply(X + Z, ys)
    assert torch.equal(ys, yx + yz)
    indeg = torch.from_numpy(rmat_s24["indeg"].astype(np.float64)).cuda()
    assert torch.equal(yx.double().sum(0), (indeg[:, None] * X.double()).sum(0))
    idx, mat = img.bytes()
    Xh = X.cpu().numpy()
    R = oracle.spmm(idx, mat, Xh, nthreads=16, brows=(0, 4))
    assert np.array_equal(yx[: 4 * 16384].cpu().numpy(), R[: 4 * 16384])


@pytest.mark.parametrize("k", [1, 16, 32])
def test_rmat_s24_weighted(torch_cuda, rmat_s24, k):
    """Full-size weighted image with N(0,1) operands: rows of at most
    EXACT_ROW_MAX entries match the oracle bit for bit on a sample of block
    rows, every sampled row within RTOL, and A 1 equals the oracle's row
    sums of the weights within RTOL."""
    torch = torch_cuda
    img = rmat_s24["weighted"]
    m = sparse_matrix.create(img, None)
    n = m.get_num_rows()
    g = torch.Generator(device="cuda").manual_seed(100 + k)
    X = torch.randn((n, k), generator=g, device="cuda")
    y = torch.empty((n, k), device="cuda")
    assert m.multiply(X, y)
    idx, mat = img.bytes()
    R = oracle.spmm(idx, mat, X.cpu().numpy(), nthreads=16, brows=(0, 4))[: 4 * 16384]
    Y = y[: 4 * 16384].cpu().numpy()
    light = rmat_s24["outdeg"][: 4 * 16384] <= _lib.EXACT_ROW_MAX
    assert np.array_equal(Y[light], R[light])
    np.testing.assert_allclose(Y, R, rtol=RTOL, atol=RTOL * np.abs(R).max())


def _whole_runs(rows, n):
    """Ranges of the warp-per-range kernel's list for binary rows of these
    entry counts: runs of whole rows and chunks of longer ones (part.h)."""
    d = np.bincount(rows, minlength=n)
    L = np.cumsum(np.where((d >= 1) & (d <= _lib.EXACT_ROW_MAX), d, 1))
    run = int(np.clip(int(L[-1]) // (148 * 32 * 16), 128, 256)) // 8 * 8
    start = np.concatenate([[0], L[:-1]]) // run
    heavy = d[d > _lib.EXACT_ROW_MAX]
    return 1 + int(np.count_nonzero(np.diff(start))) + int(np.sum((heavy + 255) // 256))


def _blocks256(t):
    """Sums of rows of 256 terms: binary trees over blocks of 16, block b added
    to running sum b % 4, a tree over those."""
    t = t.reshape(len(t), 16, 16)
    while t.shape[2] > 1:
        t = t[:, :, 0::2] + t[:, :, 1::2]
    a = np.zeros((len(t), 4), t.dtype)
    for q in range(4):
        a = a + t[:, 4 * q:4 * q + 4, 0]
    return (a[:, 0] + a[:, 1]) + (a[:, 2] + a[:, 3])


def _strided32(t):
    """The same by 32 strided running sums and a tree over them."""
    a = np.zeros((len(t), 32), t.dtype)
    for j in range(8):
        a = a + t[:, 32 * j:32 * j + 32]
    while a.shape[1] > 1:
        h = a.shape[1] // 2
        a = a[:, :h] + a[:, h:]
    return a[:, 0]


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("extra,warps", [(100_000, True), (3_000_000, False)])
@pytest.mark.parametrize("length", [512, 437, 259])
def test_spmv_chunk_sums(torch_cuda, length, extra, warps, weighted, dtype):
    """k = 1, rows of two chunks of up to 256 entries, bit for bit: a warp per
    range (up to 64 ranges per SM) adds a chunk by 32 strided sums and a tree, a
    lane per range by blocks of 16 into four running sums, and whole chunks with
    no larger error against FP64 than the former has on the same numbers."""
    torch = torch_cuda
    n, rows = 1 << 17, 1500
    rng = np.random.default_rng(extra)
    cols = np.stack([np.sort(rng.choice(n, length, replace=False)) for _ in range(rows)])
    src = np.concatenate([np.repeat(np.arange(rows), length), rng.integers(rows, n, extra)]).astype(np.uint32)
    dst = np.concatenate([cols.reshape(-1), rng.integers(0, n, extra)]).astype(np.uint32)
    assert (_whole_runs(src, n) <= 64 * torch.cuda.get_device_properties(0).multi_processor_count) == warps
    w = rng.uniform(0.5, 1, len(src)).astype(dtype) if weighted else None
    m = sparse_matrix.create(matrix_image.build(src, dst, w, nrows=n, ncols=n, block_size=(16384, 16384),
                                                dedup=False, remove_self=False), None)
    X = rng.standard_normal((n, 1)).astype(dtype)
    got = _gpu_spmm(torch, m, X)[:rows, 0]
    t = X[cols, 0]
    if weighted:
        t = t * w[:rows * length].reshape(rows, length)
    c = np.zeros((2, rows, 256), t.dtype)
    c[0, :, :length // 2], c[1, :, :length - length // 2] = t[:, :length // 2], t[:, length // 2:]
    order = _strided32 if warps else _blocks256
    assert np.array_equal(got, order(c[0]) + order(c[1]))
    if dtype == "float32" and length == 512:
        exact = t.astype(np.float64).sum(1)
        assert np.linalg.norm(got - exact) <= np.linalg.norm(_strided32(c[0]) + _strided32(c[1]) - exact)


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("scale,warps", [(15, True), (18, False)])
def test_spmv_forms_agree(torch_cuda, scale, warps, dtype):
    """k = 1 on both sides of the line between the warp-per-range kernel and
    the row kernel, against the row kernel's scaled form with scales of exactly
    1: equal bits in rows of up to EXACT_ROW_MAX entries, hub rows (whose chunks
    are added in another order) within RTOL, weighted or not, also for a strided
    column."""
    torch = torch_cuda
    tdt = getattr(torch, dtype)
    n = 1 << scale
    src, dst = rmat_edges(scale, seed=4)
    key = np.unique(src.astype(np.int64) * n + dst)
    src, dst = (key // n).astype(np.uint32), (key % n).astype(np.uint32)
    assert (_whole_runs(src, n) <= 64 * torch.cuda.get_device_properties(0).multi_processor_count) == warps
    ones = torch.ones(n, device="cuda", dtype=tdt)
    for weighted in (False, True):
        vals = np.random.default_rng(1).uniform(0.0, 1.0, len(src)).astype(np.float32) if weighted else None
        m = sparse_matrix.create(matrix_image.build(src, dst, vals, nrows=n, ncols=n, block_size=(16384, 16384),
                                                    dedup=False, remove_self=False), None)
        light = torch.from_numpy(np.bincount(src, minlength=n) <= _lib.EXACT_ROW_MAX).cuda()
        X = torch.randn((n, 1), device="cuda", dtype=tdt)
        Y1 = m.multiply(X)
        Ys = torch.empty_like(Y1)
        assert m.multiply(X, Ys, row_scale_in=ones, row_scale_out=ones)
        assert torch.equal(Y1[light], Ys[light]) and not bool(light.all())
        torch.testing.assert_close(Y1, Ys, rtol=RTOL, atol=RTOL * float(Ys.abs().max()))
        X3 = torch.zeros((n, 3), device="cuda", dtype=tdt)
        X3[:, :1] = X
        Y3 = torch.full((n, 3), 7.0, device="cuda", dtype=tdt)
        assert m.multiply(X3[:, :1], Y3[:, :1])
        assert torch.equal(Y3[:, :1], Y1) and bool((Y3[:, 1:] == 7).all())


@pytest.mark.parametrize("ydt", ["float32", "bfloat16"])
@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("k,pad", [(9, 0), (11, 0), (13, 2), (16, 1), (21, 0), (31, 0), (33, 0), (63, 0), (65, 0), (130, 1)])
def test_bf16_rows_of_odd_width(torch_cuda, k, pad, weighted, ydt):
    """BF16 rows that are no whole vectors, on a matrix with enough entries for
    lanes of four columns G apart: remainders of 1 to 4 columns in the last
    lanes, several panels, odd strides, with and without scales.  Small integer
    values, weights and power-of-two scales keep every sum exact (BF16 results:
    its rounding), in rows of 0 to 256 entries and in two longer ones."""
    torch = torch_cuda
    n, mm = 30000, 300 * 148 * 20 * 4
    src, dst = _graph(n, mm, 60 + k, ((5, 256), (29999, 9000), (77, 300)))
    rng = np.random.default_rng(k)
    vals = rng.integers(1, 3, len(src)).astype(np.float32) if weighted else None
    idx, mat = oracle.build_image(src, dst, vals, block=(16384, 16384), dedup=True)
    m = sparse_matrix.create(matrix_image.from_bytes(idx, mat), None)
    assert m.get_nnz() >= 300 * 148 * 20 * (32 // min(k, 32))
    X = rng.integers(-2, 3, (n, k))
    s = np.ldexp(1.0, rng.integers(-2, 3, n))
    sc = torch.from_numpy(s).to("cuda", torch.float32)
    tdt = getattr(torch, ydt)
    Xw = torch.full((n, k + pad), 99, dtype=torch.bfloat16, device="cuda")
    Xw[:, :k] = torch.from_numpy(X).to("cuda", torch.bfloat16)
    R = oracle.spmm(idx, mat, X.astype(np.float64))
    Rs = oracle.spmm(idx, mat, X * s[:, None])
    for si, so, want in ((None, None, R), (sc, None, Rs), (None, sc, R * s[:, None]), (sc, sc, Rs * s[:, None])):
        Yw = torch.full((n, k + pad), 77, dtype=tdt, device="cuda")
        assert m.multiply(Xw[:, :k], Yw[:, :k], si, so), _lib.last_error()
        assert torch.equal(Yw[:, :k].cpu(), torch.from_numpy(want).to(tdt))
        assert bool((Yw[:, k:] == 77).all())


def test_bf16_odd_width_costs_no_more_than_fp32(torch_cuda):
    """D^-1/2 A D^-1/2 on 31 columns at R-MAT scale 20: BF16 rows, half the
    bytes, must not take longer than FP32 rows."""
    torch = torch_cuda
    n = 1 << 20
    s, d = rmat_edges(20, seed=1)
    s, d = (torch.from_numpy(np.concatenate(p).astype(np.int32)).cuda() for p in ((s, d), (d, s)))
    m = sparse_matrix.from_device_edges(s, d, None, nrows=n, ncols=n, dedup=True)
    sc = torch.rand(n, device="cuda") + 0.5
    best = {}
    for dt in (torch.float32, torch.bfloat16):
        x = torch.randn((n, 31), device="cuda").to(dt)
        y = torch.empty_like(x)
        ev = [torch.cuda.Event(enable_timing=True) for _ in range(9)]
        for _ in range(3):
            assert m.multiply(x, y, sc, sc)
        ev[0].record()
        for e in ev[1:]:
            assert m.multiply(x, y, sc, sc)
            e.record()
        torch.cuda.synchronize()
        best[dt] = min(a.elapsed_time(b) for a, b in zip(ev, ev[1:]))
    assert best[torch.bfloat16] <= best[torch.float32]


def _best_ms(torch, call, reps=10):
    for _ in range(3):
        assert call()
    ev = [torch.cuda.Event(enable_timing=True) for _ in range(reps + 1)]
    ev[0].record()
    for e in ev[1:]:
        assert call()
        e.record()
    torch.cuda.synchronize()
    return min(a.elapsed_time(b) for a, b in zip(ev, ev[1:]))


def _rmat_device(torch, scale):
    s, d = (torch.from_numpy(x.astype(np.int32)).cuda() for x in rmat_edges(scale, seed=1))
    return sparse_matrix.from_device_edges(s, d, None, nrows=1 << scale, ncols=1 << scale, dedup=True)


def test_wide_bf16_rows_into_fp32(torch_cuda):
    """BF16 rows of 24 columns or more into FP32 (matrices of 8M entries or more):
    the same bits whether Y's rows start on sectors or 16 bytes off, and 32
    columns with input scales cost little more than into BF16 (1.2 times when
    every entry paid for a row close)."""
    torch = torch_cuda
    n, k = 1 << 20, 32
    m = _rmat_device(torch, 20)
    x = torch.randn((n, k), device="cuda").to(torch.bfloat16)
    sc = torch.rand(n, device="cuda") + 0.5
    y, z = (torch.zeros(n * k + 8, device="cuda")[off:off + n * k].view(n, k) for off in (0, 4))
    for si, so in ((None, None), (sc, None), (None, sc), (sc, sc)):
        assert m.multiply(x, y, si, so) and m.multiply(x, z, si, so)
        assert torch.equal(y, z)
    b = torch.empty_like(x)
    assert _best_ms(torch, lambda: m.multiply(x, y, sc, None)) <= 1.12 * _best_ms(torch, lambda: m.multiply(x, b, sc, None))


def test_input_scales_cost_little(torch_cuda):
    """Input scales of FP32 rows: a warp runs one copy of a step's sums, the
    scaled one when any of its groups meets a column outside the pack.  32
    columns at R-MAT scale 21 stay near the unscaled product (1.2 times when
    each group went its own way)."""
    torch = torch_cuda
    n, k = 1 << 21, 32
    m = _rmat_device(torch, 21)
    x = torch.randn((n, k), device="cuda")
    y = torch.empty_like(x)
    sc = torch.rand(n, device="cuda") + 0.5
    assert _best_ms(torch, lambda: m.multiply(x, y, sc, None)) <= 1.14 * _best_ms(torch, lambda: m.multiply(x, y))


@pytest.mark.parametrize("k", [48, 56, 64, 128])
def test_bf16_wide_rows(torch_cuda, k):
    """BF16 rows of 96 bytes or more into BF16 in lanes of 16 columns (matrices
    of 8M entries or more): whole and aligned rows take them, others do not;
    integer values and power-of-two scales, so that every element is the exact
    sum rounded once."""
    torch = torch_cuda
    n = 30000
    src, dst = _graph(n, 9_000_000, k, ((5, 256), (29999, 9000), (77, 300)))
    idx, mat = oracle.build_image(src, dst, None, block=(16384, 16384), dedup=True)
    m = sparse_matrix.create(matrix_image.from_bytes(idx, mat), None)
    assert m.get_nnz() >= 8 << 20
    rng = np.random.default_rng(k)
    X = rng.integers(-2, 3, (n, k))
    s = np.ldexp(1.0, rng.integers(-2, 3, n))
    sc = torch.from_numpy(s).to("cuda", torch.float32)
    R = oracle.spmm(idx, mat, X.astype(np.float64))
    Rs = oracle.spmm(idx, mat, X * s[:, None])
    for pad, off in ((0, 0), (16, 0), (8, 8)):
        Xw = torch.full((n, k + pad), 99, dtype=torch.bfloat16, device="cuda")
        Xw[:, off:off + k] = torch.from_numpy(X).to("cuda", torch.bfloat16)
        for si, so, want in ((None, None, R), (sc, None, Rs), (None, sc, R * s[:, None]), (sc, sc, Rs * s[:, None])):
            Yw = torch.full((n, k + pad), 77, dtype=torch.bfloat16, device="cuda")
            assert m.multiply(Xw[:, off:off + k], Yw[:, off:off + k], si, so), _lib.last_error()
            assert torch.equal(Yw[:, off:off + k].cpu(), torch.from_numpy(want).to(torch.bfloat16))
            assert bool((Yw[:, :off] == 77).all()) and bool((Yw[:, off + k:] == 77).all())


def test_bf16_wide_rows_cost(torch_cuda):
    """64 BF16 columns with input scales at R-MAT scale 21 against 32: two lanes
    a 64-byte row, four a 128-byte row (eight of 16 bytes took 1.85 times as
    long)."""
    torch = torch_cuda
    n = 1 << 21
    m = _rmat_device(torch, 21)
    sc = torch.rand(n, device="cuda") + 0.5
    t = {}
    for k in (32, 64):
        x = torch.randn((n, k), device="cuda").to(torch.bfloat16)
        y = torch.empty_like(x)
        t[k] = _best_ms(torch, lambda: m.multiply(x, y, sc, None))
    assert t[64] <= 1.72 * t[32]


def test_packed_product_takes_one_panel(torch_cuda):
    """The product whose operand's producer left the hot pack (the library's own
    entry point, used by the eigensolver's filter) refuses operands of several
    panels, whose later panels would be multiplied with the first one's pack."""
    import ctypes as C
    torch = torch_cuda
    n = 3000
    src, dst = _graph(n, 30000, 9)
    m = sparse_matrix.create(matrix_image.build(src, dst, None, nrows=n, ncols=n, dedup=True), None)
    call = _lib.lib._ZN3fmx11spmm_packedEPK10fmx_matrixiPKvliPvllS4_S4_P11CUstream_st
    call.argtypes = [C.c_void_p, C.c_int, C.c_void_p, C.c_int64, C.c_int, C.c_void_p, C.c_int64, C.c_int64, C.c_void_p,
                     C.c_void_p, C.c_void_p]
    st = torch.cuda.current_stream().cuda_stream
    for k, rc in ((32, _lib.FMX_OK), (16, _lib.FMX_OK), (33, _lib.FMX_ERR_INVAL), (48, _lib.FMX_ERR_INVAL)):
        x = torch.randn((n, k), device="cuda")
        y = torch.empty_like(x)
        assert call(m.handle, _lib.F32, x.data_ptr(), k, _lib.F32, y.data_ptr(), k, k, None, None, st) == rc
    torch.cuda.synchronize()


@pytest.mark.parametrize("k", [16, 24, 32])
def test_scaled_rows_in_huge_operands(torch_cuda, k):
    """FP32 row scales with an operand that spans 2 GB or more (a few columns of a
    wide block): rows of less than a line go in 16-byte lanes, with the bits of
    the 32-byte lanes that take them from a small operand."""
    torch = torch_cuda
    n, ld = 1 << 15, 1 << 14
    src, dst = _graph(n, 400000, k, ((5, 256), (77, 9000)))
    m = sparse_matrix.create(matrix_image.build(src, dst, None, nrows=n, ncols=n, dedup=True), None)
    wide = torch.empty((n, ld), device="cuda")
    x = wide[:, 64:64 + k]
    x.copy_(torch.randn((n, k), device="cuda"))
    sc = torch.rand(n, device="cuda") + 0.5
    for si, so in ((sc, None), (None, sc), (sc, sc)):
        y, z = torch.empty((n, k), device="cuda"), torch.empty((n, k), device="cuda")
        assert m.multiply(x, y, si, so) and m.multiply(x.contiguous(), z, si, so)
        assert torch.equal(y, z)
