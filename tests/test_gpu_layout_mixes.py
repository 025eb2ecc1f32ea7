"""Presummed rows together with the other things a product keeps in its workspace or
reads with a stride: BF16 results and GIN with compensation, GIN with BF16 results,
leading dimensions above the width, one- and two-lane teams under compensation; new
multipliers at every chunk size."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _structure(n=900, seed=3):
    """A forest with 90 % of the rows below level 0, a tenth of them 32 entries and more."""
    rng = np.random.default_rng(seed)
    v = np.arange(n)
    parent = np.where(rng.random(n) < 0.9, (v * rng.random(n)).astype(np.int64), -1)
    parent[0] = -1
    depth = np.zeros(n, np.int64)
    for i in range(1, n):
        if parent[i] >= 0:
            depth[i] = depth[parent[i]] + 1
    lens = rng.integers(0, 20, n)
    long_rows = rng.choice(n, n // 10, replace=False)
    lens[long_rows] = rng.choice([32, 33, 64, 100, 200], long_rows.size)
    crow = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    col = np.concatenate([rng.choice(n, k, replace=False) for k in lens]).astype(np.int32)
    sign = rng.choice([-1.0, 1.0], col.size).astype(np.float32)
    kids = np.nonzero(parent >= 0)[0]
    kids = kids[np.argsort(depth[kids], kind="stable")].astype(np.int32)
    mult = (rng.random(n) + 0.5).astype(np.float32)
    return n, crow, col, sign, np.array([0, kids.size], np.int32), parent[kids].astype(np.int32), kids, mult


def _plan(s):
    from cbm.plan import Plan

    n, crow, col, sign, br, src, dst, mult = s
    return Plan(crow, col, sign, n, n, br, src, dst, multipliers=mult, host=True)


def _exact(s, x, gin):
    """A X (+ gin * X) in 64 bits, the magnitudes summed and the number of terms."""
    n, crow, col, sign, _, src, dst, _ = s
    xd = x.double().cpu().numpy()
    rows = np.repeat(np.arange(n), np.diff(crow))
    val, mag, terms = np.zeros(xd.shape), np.zeros(xd.shape), np.diff(crow).astype(float)
    np.add.at(val, rows, sign[:, None] * xd[col])
    np.add.at(mag, rows, np.abs(xd[col]))
    for u, v in zip(src, dst):
        val[v] += val[u]
        mag[v] += mag[u]
        terms[v] += terms[u] + 1
    return val + gin * xd, mag + abs(gin * xd), terms[:, None] + 1


@pytest.mark.parametrize("gin", [False, True])
@pytest.mark.parametrize("ydt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("comp", [-1, 0, 2])
@pytest.mark.parametrize("chunk", [64, 256])
@pytest.mark.parametrize("cols", [1, 2, 8, 16, 24, 40, 64, 128, 256])
def test_presummed_rows_with_state_and_residual_rows(cols, chunk, comp, ydt, gin):
    """Within the bound of any summation order, 2 * terms * 2^-24 of the magnitudes
    summed, and half a last place of a BF16 result (2^-8 of it)."""
    s = _structure()
    p = _plan(s)
    p.tune(chunk_nnz=chunk)
    assert (p.stats["chunks"] > 0) == (chunk == 64)
    p.set_compensation(comp)
    x = torch.randn(s[0], cols, device="cuda").to(torch.bfloat16)
    y = torch.full((s[0], cols), float("nan"), device="cuda", dtype=ydt)
    exact, mag, terms = _exact(s, x, 1.25 if gin else 0.0)
    bound = 2.0 * terms * 2.0 ** -24 * mag + 1e-30
    if ydt == torch.bfloat16:
        bound = bound + 2.0 ** -8 * (np.abs(exact) + bound)
    for _ in range(2):
        p.matmul_gin(x, y, 0.25) if gin else p.matmul("ax", x, y)
        assert (np.abs(y.double().cpu().numpy() - exact) <= bound).all()
    p.check_device()


@pytest.mark.parametrize("cols,ldx,ldy", [(40, 44, 48), (40, 41, 43), (33, 64, 40), (128, 132, 256), (4, 8, 12),
                                          (1, 3, 2), (256, 260, 256)])
@pytest.mark.parametrize("op", ["ax", "dadx"])
def test_presummed_rows_wait_in_a_strided_result(op, cols, ldx, ldy):
    """FP32 sums wait in Y itself: the same as with contiguous operands, and nothing
    outside the rows' columns is written."""
    s = _structure(seed=5)
    n = s[0]
    p = _plan(s)
    x = torch.randn(n, cols, device="cuda")
    want = torch.empty_like(x)
    p.matmul(op, x, want)
    xs = torch.full((n, ldx), float("nan"), device="cuda")
    xs[:, :cols] = x
    ys = torch.full((n, ldy), 7.0, device="cuda")
    p.matmul(op, xs[:, :cols], ys[:, :cols])
    assert torch.equal(ys[:, :cols], want) and (ys[:, cols:] == 7.0).all()
    p.check_device()


@pytest.mark.parametrize("chunk", [32, 128, 256])
def test_new_multipliers_at_every_chunk_size(chunk):
    s = _structure(seed=7)
    n, crow, col, sign, br, src, dst, _ = s
    p = _plan(s)
    p.tune(chunk_nnz=chunk)
    m2 = (np.random.default_rng(9).random(n) + 0.25).astype(np.float32)
    x = torch.randn(n, 40, device="cuda")
    y, z = torch.empty_like(x), torch.empty_like(x)
    p.matmul("adx", x, y)
    p.set_multipliers(torch.from_numpy(m2).cuda())
    p.matmul("adx", x, y)
    q = _plan(s[:-1] + (m2,))  # created with them
    q.tune(chunk_nnz=chunk)
    q.matmul("adx", x, z)
    assert torch.equal(y, z)
    scaled = torch.from_numpy(m2).cuda()[:, None] * x
    exact, mag, terms = _exact(s, scaled, 0.0)
    assert (np.abs(y.double().cpu().numpy() - exact) <= 2.0 * (terms + 2) * 2.0 ** -24 * mag + 1e-30).all()
    p.check_device()
