"""Which forward kernel AUTO takes, told by the grid it launches, and that its results
are that kernel's."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _plan(n, deep):
    from cbm.plan import Plan

    rng = np.random.default_rng(1)
    lens = rng.integers(0, 12, n)
    crow = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    col = rng.integers(0, n, crow[-1]).astype(np.int32)
    val = rng.choice([-1.0, 1.0], col.size).astype(np.float32)
    kids = np.arange(n - int(n * (0.8 if deep else 0.1)), n, dtype=np.int32)
    src = (rng.random(kids.size) * (n - kids.size)).astype(np.int32)
    return Plan(crow, col, val, n, n, np.array([0, kids.size], np.int32), src, kids, host=True)


@pytest.mark.parametrize("n,deep,cols,dtype,kernel", [
    (30_000, False, 128, torch.float32, "register"), (30_000, False, 132, torch.float32, "staged"),
    (30_000, False, 192, torch.bfloat16, "register"), (30_000, False, 200, torch.bfloat16, "staged"),
    (30_000, False, 256, torch.bfloat16, "staged"), (30_000, False, 264, torch.bfloat16, "staged"),
    (8_000, False, 256, torch.bfloat16, "register"), (8_000, False, 264, torch.bfloat16, "staged"),
    (30_000, True, 256, torch.bfloat16, "register"), (8_000, True, 512, torch.float32, "register"),
    (30_000, True, 516, torch.float32, "staged"), (8_000, True, 1024, torch.float32, "staged"),
    (8_000, True, 1024, torch.bfloat16, "register")])
def test_auto_takes(n, deep, cols, dtype, kernel):
    p = _plan(n, deep)
    x = torch.randn(n, cols, device="cuda").to(dtype)
    out, grid = {}, {}
    for variant in ("register", "staged", "auto"):
        p.tune(variant=variant)
        out[variant] = torch.empty(n, cols, device="cuda")
        p.matmul("ax", x, out[variant])
        grid[variant] = p.stats["grid"]
    p.check_device()
    assert torch.equal(out["auto"], out["staged"]) and torch.equal(out["auto"], out["register"])
    assert grid["staged"] == grid["register"] or grid["auto"] == grid[kernel]
