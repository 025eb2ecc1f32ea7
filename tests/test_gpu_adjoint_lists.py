"""The adjoint's gather over the lists of its columns: how finely a list is summed, and
lists and children lists long enough to be split, over every team size."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

FP32_COLS = [1, 2, 4, 5, 8, 12, 16, 31, 32, 40, 47, 64, 128, 132, 260, 520]
BF16_COLS = [1, 8, 16, 24, 33, 40, 64, 128, 136, 264, 520]


def _teams(cols):
    """Teams of a warp that FP32 rows of `cols` columns leave room for."""
    vectors = cols // 4 if cols % 4 == 0 else cols
    return 32 // min(32, 1 << (vectors - 1).bit_length())


def _plan(n, lists, src=(), dst=(), sign=None, mult=None):
    """A square plan whose column j has the rows lists[j] (ascending)."""
    from cbm.plan import Plan

    col = np.repeat(np.arange(len(lists)), [len(r) for r in lists])
    row = np.concatenate(lists)
    at = np.lexsort((col, row))
    row, col = row[at], col[at].astype(np.int32)
    crow = np.concatenate([[0], np.cumsum(np.bincount(row, minlength=n))]).astype(np.int32)
    val = np.ones(col.size, np.float32) if sign is None else sign[:col.size]
    p = Plan(crow, col, val, n, n, np.array([0, len(src)] if len(src) else [0], np.int32),
             np.array(src, np.int32), np.array(dst, np.int32), multipliers=mult, host=True)
    return p, row, col, val


@pytest.mark.parametrize("cols", FP32_COLS)
def test_a_list_is_summed_in_as_many_chains_as_a_warp_has_teams(cols):
    """One row of 1 and rows of 2^-25, a quarter of its last place: a chain of
    additions that starts at the 1 loses every one of them.  With the list's entries
    over t chains only one chain in t does, so at most ceil(L / t) are lost; the
    chains' own sums are exact and the additions that join them round off at most
    half a last place of 1 (2^-24) each."""
    n = 600
    tiny = 2.0 ** -25
    lens = [2, 4, 5, 16, 17, 33, 63, 64, 65, 66, 128, 200, 255, 256]
    rng = np.random.default_rng(0)
    lists = [np.concatenate([[0], 1 + np.sort(rng.choice(n - 1, k - 1, replace=False))]) for k in lens]
    p, *_ = _plan(n, lists)
    g = torch.full((n, cols), tiny, device="cuda")
    g[0] = 1.0
    dx = torch.full((n, cols), float("nan"), device="cuda")
    p.adjoint("ax", g, dx)
    got = dx.double().cpu().numpy()
    t = _teams(cols)
    joins = 2 + (t - 1).bit_length() + 1
    for j, k in enumerate(lens):
        exact = 1.0 + (k - 1) * tiny
        assert np.abs(got[j] - exact).max() <= -(-k // t) * tiny + joins * 2.0 ** -24, k
    assert (got[len(lens):] == 0).all()
    p.check_device()


@pytest.mark.parametrize("op", ["ax", "dadx"])
@pytest.mark.parametrize("chunk", [32, 100, 256])
@pytest.mark.parametrize("dtype,cols", [(torch.float32, c) for c in FP32_COLS] +
                         [(torch.bfloat16, c) for c in BF16_COLS])
def test_split_lists_match_fp64(op, chunk, dtype, cols):
    """dX = M Delta^T P^T M G, within the bound of any summation order: 2 * terms *
    2^-24 of the magnitudes summed (+ 3 scalings)."""
    n = 1300
    rng = np.random.default_rng(3)
    # node 0 has 150 children, node 1 (one of them) 70; a few deeper chains
    src, dst = [0] * 150, list(range(1, 151))
    src, dst = src + [1] * 70, dst + list(range(200, 270))
    for v in range(270, 420):
        src.append(int(rng.integers(200, v)))
        dst.append(v)
    lens = rng.choice([0, 1, 2, 5, 17, 33, 60, 64, 65, 66, 90], n)
    lens[:8] = [500, 257, 256, 255, 130, 1000, 101, 100]
    lists = [np.sort(rng.choice(n, k, replace=False)) for k in lens]
    sign = rng.choice([-1.0, 1.0], int(lens.sum())).astype(np.float32)
    mult = (rng.random(n) + 0.5).astype(np.float32)
    p, row, col, val = _plan(n, lists, src, dst, sign, mult)
    p.tune(chunk_nnz=chunk)
    # the long lists of columns and of children are split
    assert lens.max() > chunk and np.bincount(src).max() > 64
    g = torch.randn(n, cols, device="cuda").to(dtype)
    dx = torch.full((n, cols), float("nan"), device="cuda")
    m = mult.astype(np.float64) if op == "dadx" else np.ones(n)
    h = g.double().cpu().numpy() * m[:, None]
    mag, terms = np.abs(h), np.ones(n)
    for u, v in zip(src[::-1], dst[::-1]):  # deepest first: children into parents
        h[u] += h[v]
        mag[u] += mag[v]
        terms[u] += terms[v]
    exact, total, count = np.zeros((n, cols)), np.zeros((n, cols)), np.zeros(n)
    np.add.at(exact, col, val[:, None].astype(np.float64) * h[row])
    np.add.at(total, col, mag[row])
    np.add.at(count, col, 1 + terms[row])
    bound = 2.0 * (count[:, None] + 3) * 2.0 ** -24 * total * m[:, None] + 1e-30
    for _ in range(2):  # a second product on the same flags and counters
        p.adjoint(op, g, dx)
        assert (np.abs(dx.double().cpu().numpy() - exact * m[:, None]) <= bound).all()
    if dtype == torch.bfloat16:
        db = torch.empty(n, cols, device="cuda", dtype=dtype)
        p.adjoint(op, g, db)
        assert torch.equal(db, dx.to(dtype))
    p.check_device()
