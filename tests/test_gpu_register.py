"""The register-gather forward kernel where its shapes change: every team size
and vector count, rows presummed ahead of the tree's waits, items whose parent
sits in the same group of a warp, empty rows, scalar columns, and X rows 2^32
bytes apart.

Every row here has at most 256 entries, so nothing is split and FP32 results
must equal the oracle's bit for bit (the same FMAs in the same order)."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _deep_structure(n=700, seed=0, near=0.45, child=0.9):
    """A forest in which a share `near` of the rows hangs from one of the three
    rows before it and a share `child` from any earlier row (most rows are below
    level 0 by default); about a tenth of the rows are 32 entries or longer."""
    rng = np.random.default_rng(seed)
    parent = np.full(n, -1)
    for v in range(1, n):
        u = rng.random()
        if u < near:
            parent[v] = v - 1 - rng.integers(0, min(v, 3))
        elif u < child:
            parent[v] = rng.integers(0, v)
    depth = np.zeros(n, dtype=int)
    for v in range(n):
        depth[v] = depth[parent[v]] + 1 if parent[v] >= 0 else 0
    lens = rng.choice([0, 1, 2, 3, 4, 5, 7, 8, 9, 16, 31], size=n)
    long_rows = rng.choice(n, n // 10, replace=False)
    lens[long_rows] = rng.choice([32, 33, 48, 63, 64, 65, 129, 256], size=long_rows.size)
    crow = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    col = np.concatenate([rng.choice(n, k, replace=False) for k in lens]).astype(np.int32)
    sign = rng.choice([-1.0, 1.0], col.size).astype(np.float32)
    kids = np.nonzero(parent >= 0)[0]
    kids = kids[np.argsort(depth[kids], kind="stable")].astype(np.int32)
    src = parent[kids].astype(np.int32)
    mult = (rng.random(n) + 0.5).astype(np.float32)
    return n, crow, col, sign, np.array([0, kids.size], np.int32), src, kids, mult


def _plan(s):
    from cbm.plan import Plan

    n, crow, col, sign, br, src, dst, mult = s
    return Plan(crow, col, sign, n, n, br, src, dst, multipliers=mult, host=True)


def _oracle(op, s, x):
    from oracle import oracle

    n, crow, col, sign, br, src, dst, mult = s
    rows = np.repeat(np.arange(n), np.diff(crow))
    val = sign
    if op in ("adx", "dadx"):
        val = val * mult[col]
    if op == "dadx":
        return oracle.spmm_fused_update(crow, col, val * mult[rows], x, br, src, dst, mult, gpu_order=True)
    return oracle.spmm_update(crow, col, val, x, br, src, dst)


@pytest.mark.parametrize("op", ["ax", "dadx"])
@pytest.mark.parametrize("dtype,cols", [(torch.float32, c) for c in (1, 3, 4, 8, 12, 31, 33, 47, 64, 100, 128, 132,
                                                                     256, 260, 512, 700)] +
                         [(torch.bfloat16, c) for c in (1, 8, 33, 40, 64, 120, 128, 250, 256, 264, 520, 1024)])
def test_deep_tree_matches_oracle(op, dtype, cols):
    s = _deep_structure()
    p = _plan(s)
    x = torch.randn(s[0], cols, device="cuda").to(dtype)
    y = torch.full((s[0], cols), float("nan"), device="cuda")
    ref = _oracle(op, s, x.float().cpu().numpy())
    for _ in range(2):  # a second product on the same flags and counters
        p.matmul(op, x, y)
        np.testing.assert_array_equal(y.cpu().numpy(), ref)
    if dtype == torch.bfloat16:
        yb = torch.empty(s[0], cols, device="cuda", dtype=dtype)
        p.matmul(op, x, yb)
        assert torch.equal(yb.cpu(), torch.from_numpy(ref).to(dtype))
    p.check_device()


@pytest.mark.parametrize("dtype,cols", [(torch.float32, 1), (torch.float32, 12), (torch.float32, 33),
                                        (torch.float32, 64), (torch.float32, 128), (torch.bfloat16, 40),
                                        (torch.bfloat16, 128)])
@pytest.mark.parametrize("near,child", [(0.1, 0.2), (0.45, 0.9)], ids=["shallow", "deep"])
def test_larger_trees_match_oracle(near, child, dtype, cols):
    """More groups than resident warps; on the shallow tree also records in
    length order inside windows (two of them in level 0)."""
    from oracle import oracle

    s = _deep_structure(n=11000, seed=6, near=near, child=child)
    n, crow, col, sign, br, src, dst, _ = s
    p = _plan(s)
    p.tune(variant="register")
    p.set_compensation(-1)
    x = torch.randn(n, cols, device="cuda").to(dtype)
    xn = x.float().cpu().numpy()
    y = torch.full((n, cols), float("nan"), device="cuda")
    p.matmul("dadx", x, y)
    ref = _oracle("dadx", s, xn)
    np.testing.assert_array_equal(y.cpu().numpy(), ref)
    p.matmul_gin(x, y, 0.25)
    np.testing.assert_array_equal(y.cpu().numpy(), oracle.spmm_update_add(crow, col, sign, xn, 0.25, br, src, dst))
    if dtype == torch.bfloat16:
        yb = torch.empty(n, cols, device="cuda", dtype=dtype)
        p.matmul("dadx", x, yb)
        assert torch.equal(yb.cpu(), torch.from_numpy(ref).to(dtype))
    p.check_device()


@pytest.mark.parametrize("cols", [64, 128, 256, 512])
@pytest.mark.parametrize("chunk", [32, 48, 256])
def test_deep_tree_same_as_staged(cols, chunk):
    """Split rows and presummed rows together: the staged kernel sums the same
    chunks in the same order."""
    s = _deep_structure(seed=1)
    p = _plan(s)
    x = torch.randn(s[0], cols, device="cuda")
    y, z = torch.empty_like(x), torch.empty_like(x)
    p.tune(variant="register", chunk_nnz=chunk)
    assert (p.stats["chunks"] > 0) == (chunk < 256)
    p.matmul("dadx", x, y)
    p.tune(variant="staged", chunk_nnz=chunk)
    p.matmul("dadx", x, z)
    assert torch.equal(y, z)
    p.tune(variant="register", chunk_nnz=chunk)
    p.set_passes("two")
    p.matmul("dadx", x, z)
    assert torch.equal(y, z)
    p.check_device()


@pytest.mark.parametrize("dtype,cols", [(torch.float32, 20), (torch.float32, 33), (torch.float32, 128),
                                        (torch.float32, 256), (torch.bfloat16, 40), (torch.bfloat16, 256)])
def test_deep_tree_gin_and_compensation(dtype, cols):
    from oracle import oracle

    s = _deep_structure(seed=2)
    n, crow, col, sign, br, src, dst, _ = s
    p = _plan(s)
    x = torch.randn(n, cols, device="cuda").to(dtype)
    y = torch.empty(n, cols, device="cuda")
    p.matmul_gin(x, y, 0.25)
    ref = oracle.spmm_update_add(crow, col, sign, x.float().cpu().numpy(), 0.25, br, src, dst)
    np.testing.assert_array_equal(y.cpu().numpy(), ref)
    if dtype == torch.bfloat16:
        # compensated rows from depth 2 on: within the bound of any summation
        # order, 2 * terms * 2^-24 of the magnitudes summed
        p.set_compensation(2)
        p.matmul("ax", x, y)
        xd = x.double().cpu().numpy()
        exact, mag = np.zeros((n, cols)), np.zeros((n, cols))
        terms = np.zeros(n)
        par = {int(v): int(u) for u, v in zip(src, dst)}
        order = [v for v in range(n) if v not in par] + [int(v) for v in dst]
        for v in order:
            e = slice(crow[v], crow[v + 1])
            exact[v] = sign[e] @ xd[col[e]]
            mag[v] = np.abs(xd[col[e]]).sum(0)
            terms[v] = crow[v + 1] - crow[v]
            if v in par:
                exact[v] += exact[par[v]]
                mag[v] += mag[par[v]]
                terms[v] += terms[par[v]] + 1
        err = np.abs(y.double().cpu().numpy() - exact)
        assert (err <= 2.0 * terms[:, None] * 2.0 ** -24 * mag + 1e-30).all()
    p.check_device()


def test_presummed_rows_need_no_workspace():
    """An FP32 product of a plan without split rows runs without a workspace."""
    from cbm import _lib

    s = _deep_structure(seed=3)
    p = _plan(s)
    assert p.stats["chunks"] == 0
    x = torch.randn(s[0], 64, device="cuda")
    y = torch.empty_like(x)
    rc = _lib.load().cbm_matmul(p._h, _lib.OP_AX, x.data_ptr(), _lib.F32, 64, y.data_ptr(), _lib.F32, 64, 64, None, 0,
                                C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == _lib.OK
    np.testing.assert_array_equal(y.cpu().numpy(), _oracle("ax", s, x.cpu().numpy()))


def test_new_multipliers_reach_the_scaled_entries():
    s = _deep_structure(seed=4)
    p = _plan(s)
    x = torch.randn(s[0], 40, device="cuda")
    y = torch.empty_like(x)
    p.matmul("adx", x, y)
    m2 = (np.random.default_rng(9).random(s[0]) + 0.25).astype(np.float32)
    p.set_multipliers(torch.from_numpy(m2).cuda())
    for chunk in (256, 128, 256):  # also after the entries are laid out again
        p.tune(chunk_nnz=chunk)
        if chunk == 256:
            p.matmul("adx", x, y)
            np.testing.assert_array_equal(y.cpu().numpy(), _oracle("adx", s[:-1] + (m2,), x.cpu().numpy()))


@pytest.mark.parametrize("cols", [5, 128])
def test_rows_of_x_4_gib_apart(cols):
    from cbm.plan import Plan

    ld = (1 << 30) + 4  # floats between the two rows of X
    store = torch.empty(ld + cols, device="cuda")
    x = store.as_strided((2, cols), (ld, 1))
    x.copy_(torch.randn(2, cols, device="cuda"))
    p = Plan(np.array([0, 2, 3], np.int32), np.array([0, 1, 1], np.int32), np.array([1, 1, -1], np.float32), 2, 2,
             np.array([0, 1], np.int32), np.array([0], np.int32), np.array([1], np.int32), host=True)
    p.tune(variant="register")
    y = torch.empty(2, cols, device="cuda")
    p.matmul("ax", x, y)
    xs = x.cpu()
    top = xs[0] + xs[1]
    assert torch.equal(y.cpu(), torch.stack([top, -xs[1] + top]))
    p.check_device()


@pytest.mark.parametrize("op", ["ax", "dadx"])
@pytest.mark.parametrize("chunk", [32, 256])
@pytest.mark.parametrize("dtype,cols", [(torch.float32, c) for c in (1, 3, 4, 8, 12, 16, 20, 33, 40, 64, 128, 132, 256,
                                                                     300, 1028)] +
                         [(torch.bfloat16, c) for c in (1, 5, 8, 16, 24, 40, 128, 136, 520, 1032)])
def test_adjoint_of_a_deep_tree(op, chunk, dtype, cols):
    """dX = M Delta^T P^T M G against FP64, within the bound of any summation
    order: 2 * terms * 2^-24 of the magnitudes summed (+ 3 scalings)."""
    s = _deep_structure(seed=5)
    n, crow, col, sign, br, src, dst, mult = s
    p = _plan(s)
    p.tune(chunk_nnz=chunk)
    g = torch.randn(n, cols, device="cuda").to(dtype)
    dx = torch.full((n, cols), float("nan"), device="cuda")
    p.adjoint(op, g, dx)
    m = mult.astype(np.float64) if op == "dadx" else np.ones(n)
    h = g.double().cpu().numpy() * m[:, None]
    mag, terms = np.abs(h), np.ones(n)
    for u, v in zip(src[::-1], dst[::-1]):  # deepest first: children into parents
        h[u] += h[v]
        mag[u] += mag[v]
        terms[u] += terms[v]
    rows = np.repeat(np.arange(n), np.diff(crow))
    exact, total, count = np.zeros((n, cols)), np.zeros((n, cols)), np.zeros(n)
    np.add.at(exact, col, sign[:, None].astype(np.float64) * h[rows])
    np.add.at(total, col, mag[rows])
    np.add.at(count, col, 1 + terms[rows])
    err = np.abs(dx.double().cpu().numpy() - exact * m[:, None])
    assert (err <= 2.0 * (count[:, None] + 3) * 2.0 ** -24 * total * m[:, None] + 1e-30).all()
    p.check_device()
