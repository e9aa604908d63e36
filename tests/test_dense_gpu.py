"""Dense eigensolver kernels against plain PyTorch FP64 references.

Tolerances (relative to the result's max magnitude):
  BF16 tensor cores      3e-2  (8-bit mantissa operands, FP32 accumulate)
  TF32x3 tensor cores    1e-5  (split operands: FP32-level accuracy)
  FP64 CUDA-core Gram    1e-12
"""
import ctypes as C

import numpy as np
import pytest

from flashx_b200 import _lib

pytestmark = pytest.mark.gpu

TOL = {_lib.DENSE_BF16: 3e-2, _lib.DENSE_TF32X3: 1e-5, _lib.DENSE_F64: 1e-12}


def _stream(torch):
    return torch.cuda.current_stream().cuda_stream


@pytest.mark.parametrize("prec", [_lib.DENSE_BF16, _lib.DENSE_TF32X3])
@pytest.mark.parametrize("n,K,N,ldx", [(1000, 16, 16, 16), (100003, 16, 16, 16), (100, 16, 16, 16), (50000, 32, 16, 32),
                                       (7777, 48, 32, 48), (300, 8, 64, 8), (130, 64, 48, 64),
                                       # K padded to the MMA step; rows wider than K
                                       (999, 12, 24, 12), (4097, 20, 16, 24), (70000, 16, 16, 20),
                                       # K % 4 != 0: the thread-staged kernel
                                       (5000, 10, 16, 10), (333, 3, 8, 7)])
def test_tc_gemm(torch_cuda, prec, n, K, N, ldx):
    torch = torch_cuda
    g = torch.Generator(device="cuda").manual_seed(n + K)
    Xf = torch.randn((n, ldx), generator=g, device="cuda")
    X = Xf[:, :K]
    B = torch.randn((K, N), generator=g, device="cuda")
    Y = torch.full((n, N), float("nan"), device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    rc = _lib.lib.fmx_dense_gemm(prec, Xf.data_ptr(), ldx, n, K, B.data_ptr(), N, N, Y.data_ptr(), N, err.data_ptr(),
                                 _stream(torch))
    assert rc == 0, _lib.last_error()
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    ref = X.double() @ B.double()
    scale = float(ref.abs().max())
    assert float((Y.double() - ref).abs().max()) <= TOL[prec] * scale


@pytest.mark.parametrize("prec", [_lib.DENSE_BF16, _lib.DENSE_TF32X3, _lib.DENSE_F64])
@pytest.mark.parametrize("n,M,N", [(1000, 16, 16), (200001, 16, 16), (100, 16, 16), (65536, 32, 32), (4097, 48, 16), (129, 64, 64),
                                   (50, 16, 48), (777, 12, 5), (3, 1, 16), (99999, 8, 8), (100003, 16, 9)])
def test_gram(torch_cuda, prec, n, M, N):
    _gram_case(torch_cuda, prec, n, M, N, M, N)


# strided rows and row lengths that are not whole 16-byte units: the
# pipelined kernel takes rows of up to 64 floats in whole units, the older
# kernels the rest
@pytest.mark.parametrize("prec", [_lib.DENSE_BF16, _lib.DENSE_TF32X3])
@pytest.mark.parametrize("n,M,N,ldx,ldw", [(70001, 16, 16, 20, 32), (5000, 10, 6, 12, 8), (3333, 7, 16, 7, 16),
                                           (40000, 24, 20, 24, 20), (1000, 16, 16, 100, 16)])
def test_gram_strided(torch_cuda, prec, n, M, N, ldx, ldw):
    _gram_case(torch_cuda, prec, n, M, N, ldx, ldw)


def _gram_case(torch_cuda, prec, n, M, N, ldx, ldw):
    torch = torch_cuda
    g = torch.Generator(device="cuda").manual_seed(n + M + N)
    Xf = torch.randn((n, ldx), generator=g, device="cuda")
    Wf = torch.randn((n, ldw), generator=g, device="cuda")
    X, W = Xf[:, :M], Wf[:, :N]
    parts = _lib.lib.fmx_dense_gram_parts(prec, n)
    dt = torch.float64 if prec == _lib.DENSE_F64 else torch.float32
    part = torch.empty(parts * M * N, dtype=dt, device="cuda")
    G = torch.full((M, N), float("nan"), dtype=dt, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    for _ in range(2):                      # deterministic: same bits twice
        rc = _lib.lib.fmx_dense_gram(prec, Xf.data_ptr(), ldx, M, Wf.data_ptr(), ldw, N, n, part.data_ptr(),
                                     G.data_ptr(), err.data_ptr(), _stream(torch))
        assert rc == 0, _lib.last_error()
        torch.cuda.synchronize()
        if _ == 0:
            first = G.clone()
    assert torch.equal(first, G)
    assert int(err.item()) == 0
    ref = X.double().T @ W.double()
    scale = float(ref.abs().max())
    assert float((G.double() - ref).abs().max()) <= TOL[prec] * scale * (1 if prec != _lib.DENSE_F64 else 10)


@pytest.mark.parametrize("n,M,N,ldx,ldw", [(1, 16, 16, 16, 16), (3, 8, 8, 8, 8), (5, 32, 32, 32, 32), (17, 9, 17, 9, 17),
                                           (33, 24, 24, 24, 24), (4099, 31, 33, 40, 36), (20001, 48, 8, 48, 8),
                                           (70003, 64, 40, 64, 64), (100001, 15, 2, 16, 3)])
def test_gram_f64_tiles(torch_cuda, n, M, N, ldx, ldw):
    """The FP64 tensor-path Gram at the edges of its tiles and trips: row
    remainders, columns that fill no lane unit, blocks shared over warps; NaN
    beyond the columns must not leak in.  One operand (the symmetric form)
    must equal the two-operand form of a copy to FP64 rounding."""
    torch = torch_cuda
    _gram_case(torch, _lib.DENSE_F64, n, M, N, ldx, ldw)
    g = torch.Generator(device="cuda").manual_seed(n)
    Xf = torch.full((n, ldx + 4), float("nan"), device="cuda")
    Xf[:, :M] = torch.randn((n, M), generator=g, device="cuda")
    Xc = Xf.clone()
    part = torch.empty(_lib.lib.fmx_dense_gram_parts(_lib.DENSE_F64, n) * M * M, dtype=torch.float64, device="cuda")
    G = [torch.full((M, M), float("nan"), dtype=torch.float64, device="cuda") for _ in range(2)]
    for W, out in ((Xf, G[0]), (Xc, G[1])):
        assert _lib.lib.fmx_dense_gram(_lib.DENSE_F64, Xf.data_ptr(), ldx + 4, M, W.data_ptr(), ldx + 4, M, n,
                                       part.data_ptr(), out.data_ptr(), None, _stream(torch)) == 0
    ref = Xf[:, :M].double().T @ Xf[:, :M].double()
    tol = 1e-12 * float(ref.abs().max())
    assert float((G[0] - ref).abs().max()) <= tol and float((G[1] - ref).abs().max()) <= tol
    assert torch.equal(G[0], G[0].T)


@pytest.mark.parametrize("b", [1, 4, 16, 33, 64])
def test_chol_inv(torch_cuda, b):
    torch = torch_cuda
    g = torch.Generator(device="cuda").manual_seed(b)
    A = torch.randn((b + 5, b), generator=g, device="cuda", dtype=torch.float64)
    G = A.T @ A + 0.1 * torch.eye(b, device="cuda", dtype=torch.float64)
    T = torch.empty((b, b), dtype=torch.float64, device="cuda")
    info = torch.full((1,), -1, dtype=torch.int32, device="cuda")
    assert _lib.lib.fmx_dense_chol_inv(G.data_ptr(), b, T.data_ptr(), info.data_ptr(), _stream(torch)) == 0
    torch.cuda.synchronize()
    assert int(info.item()) == 0
    assert torch.allclose(torch.triu(T), T)
    I = T.T @ G @ T
    assert float((I - torch.eye(b, device="cuda", dtype=torch.float64)).abs().max()) < 1e-10
    # a non-positive pivot is reported
    Gbad = G.clone()
    Gbad[b // 2, b // 2] = -1.0
    assert _lib.lib.fmx_dense_chol_inv(Gbad.data_ptr(), b, T.data_ptr(), info.data_ptr(), _stream(torch)) == 0
    torch.cuda.synchronize()
    assert int(info.item()) > 0


@pytest.mark.parametrize("b", [1, 2, 7, 16, 24, 31, 32, 33, 48, 64])
def test_sym_eig(torch_cuda, b):
    torch = torch_cuda
    g = torch.Generator(device="cuda").manual_seed(100 + b)
    A = torch.randn((b, b), generator=g, device="cuda", dtype=torch.float64)
    H = A + A.T
    w = torch.empty(b, dtype=torch.float64, device="cuda")
    V = torch.empty((b, b), dtype=torch.float64, device="cuda")
    assert _lib.lib.fmx_dense_sym_eig(H.data_ptr(), b, w.data_ptr(), V.data_ptr(), _stream(torch)) == 0
    torch.cuda.synchronize()
    ref = torch.linalg.eigvalsh(H).flip(0)
    assert float((w - ref).abs().max()) < 1e-10 * max(1.0, float(ref.abs().max()))
    assert float((V.T @ V - torch.eye(b, device="cuda", dtype=torch.float64)).abs().max()) < 1e-10
    assert float((H @ V - V * w).abs().max()) < 1e-9 * max(1.0, float(ref.abs().max()))


def test_gram_f64_of_few_rows(torch_cuda):
    """What follows the loop must not outweigh it: over 1,000 and 10,000 rows and
    both forms, 32 columns (eight row groups to add up) take no longer than 33
    (two row groups); added up in turn they took 1.2 times as long."""
    torch = torch_cuda
    part = torch.empty(_lib.lib.fmx_dense_gram_parts(_lib.DENSE_F64, 10000) * 33 * 33, dtype=torch.float64, device="cuda")
    G = torch.empty((33, 33), dtype=torch.float64, device="cuda")
    total = {32: 0.0, 33: 0.0}
    for n in (1000, 10000):
        for one_operand in (False, True):
            for b in (32, 33):
                X = torch.randn((n, b), device="cuda")
                W = X if one_operand else torch.randn((n, b), device="cuda")
                ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
                t = []
                for _ in range(8):
                    torch.cuda._sleep(200000)         # the launches queue up behind it
                    ev[0].record()
                    for _ in range(20):
                        assert _lib.lib.fmx_dense_gram(_lib.DENSE_F64, X.data_ptr(), b, b, W.data_ptr(), b, b, n,
                                                       part.data_ptr(), G.data_ptr(), None, _stream(torch)) == 0
                    ev[1].record()
                    torch.cuda.synchronize()
                    t.append(ev[0].elapsed_time(ev[1]))
                total[b] += min(t)
    assert total[32] <= 1.1 * total[33]


@pytest.mark.parametrize("b", [2, 16, 33])
@pytest.mark.parametrize("exponent", [-1030, -1000, 0, 1000])
def test_chol_inv_at_the_ends_of_the_range(torch_cuda, b, exponent):
    """G times 2^exponent, down to subnormal pivots, whose reciprocals overflow:
    T is the unscaled one times 2^(-exponent / 2).  At 2^-1030 the entries keep
    44 bits; the pivots of G = A^T A + b I are at least b and its entries at most
    about 4 b, so that their rounding of 2^-44 grows by less than b^2 * 16."""
    torch = torch_cuda
    g = torch.Generator(device="cuda").manual_seed(b)
    A = torch.randn((2 * b, b), generator=g, device="cuda", dtype=torch.float64)
    G = A.T @ A + b * torch.eye(b, device="cuda", dtype=torch.float64)
    T, S = (torch.empty((b, b), dtype=torch.float64, device="cuda") for _ in range(2))
    info = torch.full((2,), -1, dtype=torch.int32, device="cuda")
    small = torch.from_numpy(np.ldexp(G.cpu().numpy(), exponent)).cuda()
    assert _lib.lib.fmx_dense_chol_inv(G.data_ptr(), b, T.data_ptr(), info.data_ptr(), _stream(torch)) == 0
    assert _lib.lib.fmx_dense_chol_inv(small.data_ptr(), b, S.data_ptr(), info[1:].data_ptr(), _stream(torch)) == 0
    assert info.tolist() == [0, 0]
    got = np.ldexp(S.cpu().numpy(), exponent // 2)
    tol = 16 * b * b * 2.0 ** (-44 if exponent < -1022 else -52)
    assert np.abs(got - T.cpu().numpy()).max() <= tol * float(T.abs().max())
