"""The workloads that this library's speed is measured on.

listed() names them, draw() gives more of the same ranges, prepare() makes a
case's inputs on the GPU from a seed, run() is one pass through the public
entry points, work() the bytes and operations that pass cannot do without and
exact() its result in 64 bits, computed with plain torch.

Kinds:
  spmm      Y = A X or A^T X on a directed R-MAT graph (sparse_matrix.multiply)
  scaled    Y = D^-1/2 A D^-1/2 X on a symmetric graph (NA_operator and the
            eigensolver's BF16 operand)
  pagerank  PageRank, 30 iterations at damping 0.85
  block     one basis step of the block eigensolver: Gram, Cholesky, basis
            update, Rayleigh quotient and the projected eigenproblem
  gnn       one training step of the warm-start network
  eigen     a whole compute_eigen on a stochastic block model graph
  host      the multiply on host buffers, as the FlashMatrix binding calls it

Graphs: R-MAT with a/b/c/d = 0.57/0.19/0.19/0.05, vertices relabelled at
random, duplicate edges and self-loops dropped by the builder; block model
graphs of average degree 20.  Matrices are built by the device builder, which
is outside run() as it is in a program that multiplies many times.
"""
import ctypes as C
import math

import numpy as np
import torch

from flashx_b200 import _lib, sparse_matrix
from flashx_b200.algs import PageRank
from flashx_b200.eigen import NA_operator, compute_eigen, eigen_options
from flashx_b200.warmstart import warm_start_net

DEV = "cuda:0"
A, B, CQ = 0.57, 0.19, 0.19             # R-MAT quadrants (d = 0.05)
CHUNK = 1 << 26                         # edges generated at a time
DTYPES = {"f32": torch.float32, "f64": torch.float64, "i32": torch.int32, "i64": torch.int64,
          "bf16": torch.bfloat16}
BYTES = {"f32": 4, "f64": 8, "i32": 4, "i64": 8, "bf16": 2}


def listed():
    return [
        # the reference's own CPU configuration: R-MAT scale 16, FP64, k = 8
        dict(name="spmm_f64_s16_k8", kind="spmm", n=1 << 16, ef=16, k=8, dtype="f64", weighted=False, transpose=False),
        # a single vector (SpMV): degrees, power iterations, one step of an iterative method
        dict(name="spmv_f32_s22_k1", kind="spmm", n=1 << 22, ef=16, k=1, dtype="f32", weighted=False, transpose=False),
        # the headline: R-MAT scale 24, FP32, k = 16
        dict(name="spmm_f32_s24_k16", kind="spmm", n=1 << 24, ef=16, k=16, dtype="f32", weighted=False,
             transpose=False),
        # edge weights uniform in (0, 1], the widest panel of the sweep
        dict(name="spmm_w32_s22_k32", kind="spmm", n=1 << 22, ef=16, k=32, dtype="f32", weighted=True,
             transpose=False),
        # an odd vertex count and a panel that is no whole vector, through the
        # transpose (k = 10 is the reference unit test's panel)
        dict(name="spmm_t_f32_n1m_k10", kind="spmm", n=999_983, ef=16, k=10, dtype="f32", weighted=False,
             transpose=True),
        # integer counting (paths, neighbours): int64 with integer weights
        dict(name="spmm_i64_n300k_k4", kind="spmm", n=300_007, ef=16, k=4, dtype="i64", weighted=True,
             transpose=False),
        # the operator of the eigensolver's mixed-precision filter
        dict(name="scaled_bf16_s21_k16", kind="scaled", graph="rmat", n=1 << 21, ef=16, k=16, dtype="bf16"),
        # PageRank at the reference's CPU configuration
        dict(name="pagerank_s16", kind="pagerank", n=1 << 16, ef=16, iters=30),
        # the block eigensolver's dense step at n = 4.2M, 16 columns
        dict(name="block_n4m_b16", kind="block", n=1 << 22, b=16),
        # a training step of the learned warm start on a block model graph
        dict(name="gnn_sbm_n100k", kind="gnn", n=100_000, blocks=8, ratio=12.0),
        # a whole eigensolve on a block model graph, random start
        dict(name="eigen_sbm_n50k", kind="eigen", n=50_000, nev=4, precision="plain"),
        # the drop-in call on pageable host buffers
        dict(name="host_f32_s18_k16", kind="host", n=1 << 18, ef=16, k=16, dtype="f32"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["spmm"] * 8 + ["scaled"] * 3 + ["pagerank"] * 2 + ["block"] * 2 + ["gnn", "eigen", "host"])
    if kind == "spmm":
        dtype = rng.choice(["f32"] * 5 + ["f64"] * 3 + ["i32", "i64"])
        n = _log(rng, 1 << 12, 1 << 24)
        if rng.random() < 0.3:
            n = 1 << (n.bit_length() - 1)
        # panels: one column, whole vectors or any width; operands of at most 512 MB
        most = max(1, min(64, (1 << 29) // (n * BYTES[dtype])))
        k = rng.choice([1, 2, 4, 8, 16, 16, 32, rng.randint(2, 40)])
        return dict(kind=kind, n=n, ef=rng.choice([8, 16, 16]), k=min(k, most), dtype=dtype,
                    weighted=rng.random() < 0.4, transpose=rng.random() < 0.3)
    if kind == "scaled":
        graph = rng.choice(["rmat", "sbm"])
        n = _log(rng, 1 << 12, 1 << 21) if graph == "rmat" else _log(rng, 10_000, 200_000)
        return dict(kind=kind, graph=graph, n=n, ef=16 if graph == "rmat" else 10, k=rng.choice([8, 16, 16, 24, 32]),
                    dtype=rng.choice(["f32", "f32", "bf16"]))
    if kind == "pagerank":
        return dict(kind=kind, n=_log(rng, 1 << 12, 1 << 20), ef=16, iters=rng.choice([10, 20, 30, 30]))
    if kind == "block":
        b = rng.choice([8, 16, 16, 24, 32, 48])
        return dict(kind=kind, n=_log(rng, 10_000, (1 << 26) // b), b=b)
    if kind == "gnn":
        return dict(kind=kind, n=_log(rng, 10_000, 200_000), blocks=rng.randint(4, 16),
                    ratio=round(rng.uniform(5, 20), 2))
    if kind == "eigen":
        return dict(kind=kind, n=_log(rng, 10_000, 100_000), nev=4, precision="plain")
    return dict(kind="host", n=_log(rng, 1 << 12, 1 << 18), ef=16, k=rng.choice([1, 8, 16, rng.randint(2, 16)]),
                dtype=rng.choice(["f32", "f64"]))


# ---------------------------------------------------------------------------
# Graphs (plain torch, on the GPU)
# ---------------------------------------------------------------------------

def _gen(seed, salt):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 1009 + salt)


def _rmat(n, ef, seed):
    """R-MAT edges (int32 src, dst) on n vertices: the 2^scale generator with
    labels permuted, edges between the first n labels kept."""
    scale = max(1, (n - 1).bit_length())
    g = _gen(seed, 1)
    perm = torch.randperm(1 << scale, generator=g, device=DEV, dtype=torch.int32)
    src, dst = [], []
    left = ef << scale
    while left > 0:
        m = min(left, CHUNK)
        left -= m
        r = torch.zeros(m, dtype=torch.int32, device=DEV)
        c = torch.zeros(m, dtype=torch.int32, device=DEV)
        for _ in range(scale):
            u = torch.rand(m, generator=g, device=DEV)
            rb = u >= A + B
            cb = ((u >= A) & (u < A + B)) | (u >= A + B + CQ)
            r.mul_(2).add_(rb)
            c.mul_(2).add_(cb)
        r, c = perm[r], perm[c]
        if n < 1 << scale:
            keep = (r < n) & (c < n)
            r, c = r[keep], c[keep]
        src.append(r)
        dst.append(c)
    return torch.cat(src), torch.cat(dst)


def _both(src, dst):
    return torch.cat([src, dst]), torch.cat([dst, src])


def _sbm(n, p_in, sizes, seed, degree=20):
    """Block model edges, both directions, and the vertices' block labels:
    n * degree / 2 edges from uniform vertices, an edge of block b staying in
    its block with probability p_in[b], else ending anywhere."""
    g = _gen(seed, 2)
    nb = len(p_in)
    cum = torch.tensor(np.concatenate([[0], np.cumsum(sizes)]) * n / float(np.sum(sizes)), device=DEV).long()
    cum[-1] = n
    m = n * degree // 2
    u = torch.randint(0, n, (m,), generator=g, device=DEV)
    blk = torch.searchsorted(cum, u, right=True) - 1
    lo, size = cum[blk], (cum[1:] - cum[:-1])[blk]
    near = lo + (torch.rand(m, generator=g, device=DEV, dtype=torch.float64) * size).long()
    far = torch.randint(0, n, (m,), generator=g, device=DEV)
    p = torch.tensor(p_in, device=DEV)[blk]
    v = torch.where(torch.rand(m, generator=g, device=DEV) < p, near, far)
    perm = torch.randperm(n, generator=g, device=DEV)
    labels = torch.empty(n, dtype=torch.int64, device=DEV)
    labels[perm] = torch.repeat_interleave(torch.arange(nb, device=DEV), cum[1:] - cum[:-1])
    s, d = _both(perm[u].int(), perm[v].int())
    return s, d, labels


def _graph(case, seed):
    """src, dst, values or None, labels or None."""
    kind, n = case["kind"], case["n"]
    if kind == "gnn":
        nb, r = case["blocks"], case["ratio"]
        p = r / (r + nb - 1)
        # the share of in-block edges of `ratio`, part of them from the uniform draw
        s, d, lab = _sbm(n, [max(0.0, (p - 1 / nb) / (1 - 1 / nb))] * nb, [1] * nb, seed)
        return s, d, None, lab
    if kind == "eigen":
        # communities of different sizes and strengths: separate eigenvalues
        s, d, lab = _sbm(n, [0.95, 0.85, 0.75, 0.65], [3, 4, 5, 6], seed)
        return s, d, None, lab
    if kind == "scaled" and case["graph"] == "sbm":
        s, d, lab = _sbm(n, [0.6] * 8, [1] * 8, seed)
        return s, d, None, lab
    s, d = _rmat(n, case["ef"], seed)
    if kind == "scaled":
        s, d = _both(s, d)
    v = None
    if case.get("weighted"):
        g = _gen(seed, 3)
        if case["dtype"] in ("i32", "i64"):
            v = torch.randint(1, 9, (s.numel(),), generator=g, device=DEV, dtype=DTYPES[case["dtype"]])
        else:
            v = 1 - torch.rand(s.numel(), generator=g, device=DEV, dtype=DTYPES[case["dtype"]])
    return s, d, v, None


def _dense(rows, k, dtype, seed, salt=4):
    g = _gen(seed, salt)
    if dtype in ("i32", "i64"):
        return torch.randint(-8, 9, (rows, k), generator=g, device=DEV, dtype=DTYPES[dtype])
    if dtype == "f64":
        return torch.rand((rows, k), generator=g, device=DEV, dtype=torch.float64) * 2 - 1
    return torch.randn((rows, k), generator=g, device=DEV).to(DTYPES[dtype])


def _block_x(case, seed):
    """A filtered block: columns of falling size that lean on one another."""
    n, b = case["n"], case["b"]
    x = _dense(n, b, "f32", seed)
    x[:, 1:] += 0.25 * x[:, :-1].clone()
    return x * (0.9 ** torch.arange(b, device=DEV)), _dense(n, b, "f32", seed, 5)


def _nonzero(s):
    return torch.where(s > 0, s, torch.ones_like(s))


def _gnn_params(seed):
    """Glorot-uniform W1 (64 x 64), zero b1, W2 (64 x 16)."""
    r = np.random.default_rng(seed)
    a1, a2 = math.sqrt(6 / 128), math.sqrt(6 / 80)
    return np.concatenate([r.uniform(-a1, a1, 4096), np.zeros(64), r.uniform(-a2, a2, 1024)]).astype(np.float32)


# ---------------------------------------------------------------------------
# prepare, run
# ---------------------------------------------------------------------------

def prepare(case, seed):
    kind, n = case["kind"], case["n"]
    st = {"case": case}
    if kind == "block":
        b = case["b"]
        x, noise = _block_x(case, seed)
        st["x"], st["w"] = x, x + 0.1 * noise       # W = A X of a symmetric operator: near X's span
        parts = _lib.lib.fmx_dense_gram_parts(_lib.DENSE_F64, n)
        f64 = dict(dtype=torch.float64, device=DEV)
        st["part"] = torch.empty(parts * b * b, **f64)
        st["g"], st["t"], st["h"], st["v"] = (torch.empty((b, b), **f64) for _ in range(4))
        st["ev"] = torch.empty(b, **f64)
        st["y"] = torch.empty((n, b), device=DEV)
        st["info"], st["err"] = (torch.zeros(1, dtype=torch.int32, device=DEV) for _ in range(2))
        return st
    s, d, v, lab = _graph(case, seed)
    m = sparse_matrix.from_device_edges(s, d, v, nrows=n, ncols=n, dedup=True, remove_self=True,
                                        transpose=kind == "pagerank" or bool(case.get("transpose")))
    del s, d, v
    st["m"] = m
    if kind == "spmm":
        if case["transpose"]:
            st["m"] = m.transpose()
        st["x"] = _dense(n, case["k"], case["dtype"], seed)
        st["y"] = torch.empty_like(st["x"])
    elif kind == "scaled":
        st["op"] = NA_operator(m)
        st["x"] = _dense(n, case["k"], case["dtype"], seed)
        st["y"] = torch.empty_like(st["x"])
    elif kind == "gnn":
        st["op"] = NA_operator(m)
        st["net"] = warm_start_net()
        st["net"].set_params(_gnn_params(seed))
        st["z"] = _dense(n, _lib.GNN_FEATURES, "f32", seed)
        # the ideal eigenvectors: D^1/2 on each block, normalised
        u = torch.nn.functional.one_hot(lab, case["blocks"]).float() / _nonzero(st["op"].scale)[:, None]
        st["u"] = (u / u.norm(dim=0)).contiguous()
    elif kind == "eigen":
        st["op"] = NA_operator(m)
        o = eigen_options()
        o.init(case["nev"])
        o.which, o.tol, o.precision = "LA", 1e-6, case["precision"]
        st["opts"] = o
    elif kind == "host":
        st["x"] = _dense(n, case["k"], case["dtype"], seed).cpu().numpy()
        st["y"] = np.zeros_like(st["x"])
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "spmm":
        st["m"].multiply(st["x"], st["y"])
        return st["y"]
    if kind == "scaled":
        st["m"].multiply(st["x"], st["y"], st["op"].scale, st["op"].scale)
        return st["y"]
    if kind == "pagerank":
        pr, it = PageRank(st["m"], case["iters"], 0.85)
        return {"pr": pr, "iters": it}
    if kind == "block":
        return _block_step(st, case["n"], case["b"])
    if kind == "gnn":
        loss, grad = st["net"].loss_grad(st["op"], st["z"], st["u"], want_grad=True)
        return {"loss": loss, "grad": grad}
    if kind == "eigen":
        res = compute_eigen(st["op"], True, st["opts"])
        return {"vals": res.vals, "vecs": res.vecs}
    return st["m"].multiply_host(st["x"], st["y"])


def _block_step(st, n, b):
    lib, p = _lib.lib, lambda t: t.data_ptr()
    s = torch.cuda.current_stream().cuda_stream
    x, w, y = st["x"], st["w"], st["y"]
    ck = _lib.check
    # CholQR: G = X^T X, T = R^-1, Y = X T
    ck(lib.fmx_dense_gram(_lib.DENSE_F64, p(x), b, b, p(x), b, b, n, p(st["part"]), p(st["g"]), None, s))
    ck(lib.fmx_dense_chol_inv(p(st["g"]), b, p(st["t"]), p(st["info"]), s))
    tf = st["t"].float()
    ck(lib.fmx_dense_gemm(_lib.DENSE_TF32X3, p(x), b, n, b, p(tf), b, b, p(y), b, p(st["err"]), s))
    # Rayleigh quotient X^T W and the projected eigenproblem (of G, symmetric)
    ck(lib.fmx_dense_gram(_lib.DENSE_F64, p(x), b, b, p(w), b, b, n, p(st["part"]), p(st["h"]), None, s))
    ck(lib.fmx_dense_sym_eig(p(st["g"]), b, p(st["ev"]), p(st["v"]), s))
    return {"g": st["g"], "t": st["t"], "y": y, "h": st["h"], "ev": st["ev"], "v": st["v"]}


# ---------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------

def work(case):
    kind, n = case["kind"], case["n"]
    if kind == "block":
        b = case["b"]
        # X once for G and Y, W once, Y written
        return {"bytes": 3 * 4 * n * b, "flops": 6 * n * b * b}
    if kind in ("gnn", "eigen"):
        nnz = 20 * n
        if kind == "gnn":
            # features, hidden layer forward and backward, two SpMMs of 16 columns
            return {"bytes": 4 * n * (64 + 64 + 64 + 4 * 16) + 2 * 4 * nnz, "flops": 4 * n * 64 * (64 + 16 + 16) + 64 * nnz}
        # about 25 operator applications to 16 columns
        return {"bytes": 25 * (4 * nnz + 8 * n * 16), "flops": 25 * 32 * nnz}
    nnz = case["ef"] * n * (2 if kind == "scaled" else 1)
    if kind == "pagerank":
        return {"bytes": case["iters"] * (4 * nnz + 4 * 5 * n), "flops": case["iters"] * 2 * nnz}
    e = BYTES[case["dtype"]]
    per = 4 + (e if case.get("weighted") else 0)
    return {"bytes": 4 * (n + 1) + per * nnz + 2 * n * case["k"] * e, "flops": 2 * nnz * case["k"]}


# ---------------------------------------------------------------------------
# exact: the same in 64 bits
# ---------------------------------------------------------------------------

def _csr64(n, src, dst, vals):
    """Row-major CSR in FP64 of the edge list: self-loops dropped, the first
    occurrence of a duplicate kept."""
    at = torch.nonzero(src != dst).squeeze(1)
    key = src[at].long() * n + dst[at].long()
    key, order = torch.sort(key, stable=True)
    first = torch.ones_like(key, dtype=torch.bool)
    first[1:] = key[1:] != key[:-1]
    key = key[first]
    row = torch.div(key, n, rounding_mode="floor")
    col = (key - row * n).int()
    ptr = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    ptr[1:] = torch.cumsum(torch.bincount(row, minlength=n), 0)
    val = torch.ones(key.numel(), dtype=torch.float64, device=DEV) if vals is None else \
        vals[at][order][first].double()
    return torch.sparse_csr_tensor(ptr.int(), col, val, size=(n, n), check_invariants=False), ptr[1:] - ptr[:-1]


def _scale64(deg):
    """D^-1/2 as the operator holds it: rounded to FP32."""
    d = deg.double()
    return torch.where(d > 0, 1 / torch.sqrt(d.clamp(min=1)), torch.zeros_like(d)).float().double()


def exact(case, seed):
    kind, n = case["kind"], case["n"]
    if case.get("dtype") in ("i32", "i64"):
        return None                                  # whole numbers
    if kind == "block":
        return _exact_block(case, seed)
    s, d, v, lab = _graph(case, seed)
    if case.get("transpose") or kind == "pagerank":
        s, d = d, s
    m, deg = _csr64(n, s, d, v)
    if kind == "pagerank":
        out_deg = _csr64(n, d, s, v)[1].double().clamp(min=1)
        return _exact_pagerank(m, out_deg, n, case["iters"])
    del s, d, v
    if kind in ("spmm", "host"):
        y = m @ _dense(n, case["k"], case["dtype"], seed).double()
        return y.cpu().numpy() if kind == "host" else y
    sc = _scale64(deg)[:, None]
    if kind == "scaled":
        return sc * (m @ (sc * _dense(n, case["k"], case["dtype"], seed).double()))
    if kind == "gnn":
        return _exact_gnn(case, seed, m, sc, lab)
    # the eigenvalues by orthogonal iteration on (A_s + I)^8 from a wider block
    q = torch.linalg.qr(torch.randn((n, 24), generator=_gen(1, 9), device=DEV, dtype=torch.float64))[0]
    for _ in range(40):
        for _ in range(8):
            q = (q + sc * (m @ (sc * q))) / 2
        q = torch.linalg.qr(q)[0]
    h = q.T @ (sc * (m @ (sc * q)))
    return {"vals": torch.linalg.eigvalsh((h + h.T) / 2).flip(0)[:case["nev"]].cpu().numpy(), "vecs": None}


def _exact_block(case, seed):
    n, b = case["n"], case["b"]
    x, noise = _block_x(case, seed)
    w = x + 0.1 * noise
    g = torch.zeros((b, b), dtype=torch.float64, device=DEV)
    h = torch.zeros_like(g)
    for i in range(0, n, 1 << 20):
        xs = x[i:i + (1 << 20)].double()
        g += xs.T @ xs
        h += xs.T @ w[i:i + (1 << 20)].double()
    r = torch.linalg.cholesky(g).T
    t = torch.linalg.solve_triangular(r, torch.eye(b, dtype=torch.float64, device=DEV), upper=True)
    y = x.double() @ t.float().double()
    # the eigenvectors' signs are free
    return {"g": g, "t": t, "y": y, "h": h, "ev": torch.linalg.eigvalsh(g).flip(0), "v": None}


def _exact_pagerank(mt, out_deg, n, iters):
    pr = torch.full((n,), 1.0 / n, dtype=torch.float64, device=DEV)
    it = 0
    while it < iters:
        new = 0.85 * (mt @ (pr / out_deg)[:, None]).squeeze(1) + 0.15 / n
        it += 1
        done = bool(((pr - new).abs() < 0.001 / n).all())
        pr = new
        if done:
            break
    return {"pr": pr, "iters": None}


def _exact_gnn(case, seed, m, sc, lab):
    """The network and its loss with FP64 weights and products."""
    p = torch.tensor(_gnn_params(seed), dtype=torch.float64, device=DEV)
    w1, b1, w2 = p[:4096].view(64, 64), p[4096:4160], p[4160:].view(64, 16)
    z = _dense(case["n"], _lib.GNN_FEATURES, "f32", seed).double()
    u = torch.nn.functional.one_hot(lab, case["blocks"]).float() / _nonzero(sc.float())
    u = (u / u.norm(dim=0)).double()
    pre = z @ w1 + b1
    h = pre.clamp(min=0)
    y = sc * (m @ (sc * (h @ w2)))
    gi = torch.linalg.inv(y.T @ y)
    k = (u.T @ y) @ gi
    nev = case["blocks"]
    loss = 1 - float((k * (u.T @ y)).sum()) / nev
    dy = (2 / nev) * (y @ (k.T @ k) - u @ k)
    dz2 = sc * (m @ (sc * dy))                       # A_s is symmetric
    dw2 = h.T @ dz2
    dh = (dz2 @ w2.T) * (pre > 0)
    grad = torch.cat([(z.T @ dh).reshape(-1), dh.sum(0), dw2.reshape(-1)])
    return {"loss": loss, "grad": grad.cpu().numpy()}
