"""The register-gather kernel on both sides of its rule for small plans: one group of
rows claimed at a time, with more gathers in flight for teams of 8 lanes and more, and
two groups claimed ahead on larger plans; levels narrower than a warp, whose rows share
it with their parents.  No row is split, so FP32 results equal the oracle's bit for bit."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _structure(n, near, child, seed=0, top=40):
    """Rows of up to `top` entries; a share `near` of them hangs from one of the three
    rows before it, a share `child` from any earlier one."""
    rng = np.random.default_rng(seed)
    v = np.arange(n)
    u = rng.random(n)
    parent = np.where(u < near, v - 1 - rng.integers(0, 3, n), (v * rng.random(n)).astype(np.int64))
    parent = np.where((u < child) & (v > 0), np.maximum(parent, 0), -1)
    depth = np.zeros(n, np.int64)
    for i in range(n):
        if parent[i] >= 0:
            depth[i] = depth[parent[i]] + 1
    lens = rng.integers(0, top, n)
    crow = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    col = rng.integers(0, n, crow[-1]).astype(np.int32)
    sign = rng.choice([-1.0, 1.0], col.size).astype(np.float32)
    kids = np.nonzero(parent >= 0)[0]
    kids = kids[np.argsort(depth[kids], kind="stable")].astype(np.int32)
    mult = (rng.random(n) + 0.5).astype(np.float32)
    return n, crow, col, sign, np.array([0, kids.size], np.int32), parent[kids].astype(np.int32), kids, mult


def _check(s, cols, dtype):
    from cbm.plan import Plan
    from oracle import oracle

    n, crow, col, sign, br, src, dst, mult = s
    p = Plan(crow, col, sign, n, n, br, src, dst, multipliers=mult, host=True)
    p.tune(variant="register")
    p.set_compensation(-1)
    x = torch.randn(n, cols, device="cuda").to(dtype)
    xn = x.float().cpu().numpy()
    y = torch.full((n, cols), float("nan"), device="cuda")
    rows = np.repeat(np.arange(n), np.diff(crow))
    ref = oracle.spmm_fused_update(crow, col, sign * mult[col] * mult[rows], xn, br, src, dst, mult, gpu_order=True)
    for _ in range(2):  # a second product on the same flags and counters
        p.matmul("dadx", x, y)
        np.testing.assert_array_equal(y.cpu().numpy(), ref)
    p.matmul_gin(x, y, 0.25)
    np.testing.assert_array_equal(y.cpu().numpy(), oracle.spmm_update_add(crow, col, sign, xn, 0.25, br, src, dst))
    if dtype == torch.bfloat16:
        yb = torch.empty(n, cols, device="cuda", dtype=dtype)
        p.matmul("dadx", x, yb)
        assert torch.equal(yb.cpu(), torch.from_numpy(ref).to(dtype))
    p.check_device()


# rows on either side of the rule, by lanes per row (32 * 148 * 24 * 8 lanes in all on B200)
@pytest.mark.parametrize("near,child", [(0.1, 0.2), (0.45, 0.9)], ids=["shallow", "deep"])
@pytest.mark.parametrize("n,cols,dtype", [
    (29_000, 128, torch.float32), (29_000, 256, torch.float32), (29_000, 47, torch.float32),
    (29_000, 256, torch.bfloat16), (58_000, 64, torch.float32), (58_000, 128, torch.float32),
    (58_000, 120, torch.bfloat16), (115_000, 32, torch.float32), (115_000, 40, torch.bfloat16),
    (28_300, 128, torch.float32), (28_300, 260, torch.float32), (56_000, 12, torch.bfloat16),
    (230_000, 16, torch.float32), (230_000, 4, torch.float32), (920_000, 1, torch.float32),
    (460_000, 8, torch.float32), (920_000, 8, torch.bfloat16)])
def test_both_sides_of_the_small_plan_rule(n, cols, dtype, near, child):
    _check(_structure(n, near, child, top=6 if n > 100_000 else 40), cols, dtype)


@pytest.mark.parametrize("cols,dtype", [(c, torch.float32) for c in (1, 2, 4, 8, 16, 20, 32, 47, 64, 128, 192)] +
                         [(c, torch.bfloat16) for c in (1, 8, 16, 24, 40, 64, 128, 256)])
@pytest.mark.parametrize("n", [1, 2, 31, 33, 257, 1500])
def test_levels_narrower_than_a_warp(n, cols, dtype):
    """Chains: nearly every row waits on one of the three before it."""
    _check(_structure(n, 0.97, 0.98, seed=n), cols, dtype)
