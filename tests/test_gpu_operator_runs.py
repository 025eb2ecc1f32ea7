"""The reference operators' row product on few rows: a block takes fewer rows than it
has teams, down to one warp's share.  One FMA per entry in order, so the oracle's result
bit for bit."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cols", [1, 3, 4, 8, 12, 16, 33, 64, 128, 256])
@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 592, 600, 2215, 9473, 20_000])
def test_few_rows_match_the_oracle(n, cols):
    from cbm import cbm_mkl_cpp as ops
    from oracle import oracle

    rng = np.random.default_rng(n)
    lens = rng.integers(0, 20, n)
    lens[rng.integers(0, n, max(1, n // 50))] = rng.choice([17, 65, 90, 300], max(1, n // 50))
    crow = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    col = rng.integers(0, n, crow[-1]).astype(np.int32)
    val = rng.standard_normal(col.size).astype(np.float32)
    kids = np.arange(n - n // 3, n, dtype=np.int32)
    src = (rng.random(kids.size) * (n - kids.size)).astype(np.int32)
    br = np.array([0, kids.size], np.int32)
    t = lambda a: torch.from_numpy(a).cuda()  # noqa: E731
    x = torch.randn(n, cols, device="cuda")
    y = torch.full((n, cols), float("nan"), device="cuda")
    head = (t(crow[:-1].copy()), t(crow[1:].copy()), t(col), t(val), x)
    ops.s_spmm_csr_int32(*head, y)
    none = np.zeros(0, np.int32)
    xn = x.cpu().numpy()
    np.testing.assert_array_equal(y.cpu().numpy(),
                                  oracle.spmm_update(crow, col, val, xn, np.zeros(1, np.int32), none, none))
    y.fill_(float("nan"))
    ops.s_spmm_update_csr_int32(*head, t(br), t(src), t(kids), y)
    np.testing.assert_array_equal(y.cpu().numpy(), oracle.spmm_update(crow, col, val, xn, br, src, kids))
    ops.check_device()
