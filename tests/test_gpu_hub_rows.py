"""The reference operators on rows long enough to be summed by column slices
(csrc/direct.cu): lengths around the thresholds, the rings' groups of 4 and 8 and the
entry batches of 32, whole and partial slices of 32 columns, scalar columns.
One FMA per entry in order, so the oracle's result bit for bit."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _csr(n, seed=0):
    rng = np.random.default_rng(seed)
    lens = rng.integers(0, 12, n)
    special = [15, 16, 17, 20, 21, 31, 33, 63, 64, 65, 100, 128, 129, 160, 161, 255, 256, 257, 264, 289, 511, 512, 513, n]
    lens[rng.choice(n, len(special), replace=False)] = special
    crow = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    col = np.concatenate([rng.choice(n, k, replace=False) for k in lens]).astype(np.int32)
    val = rng.standard_normal(col.size).astype(np.float32)
    return crow, col, val


def _run(crow, col, val, x, y, eps=None):
    from cbm import cbm_mkl_cpp as ops

    t = lambda a: torch.from_numpy(a).cuda()  # noqa: E731
    args = (t(crow[:-1].copy()), t(crow[1:].copy()), t(col), t(val), x)
    if eps is None:
        ops.s_spmm_csr_int32(*args, y)
    else:
        ops.s_spmm_add_csr_int32(*args, eps, y)


@pytest.mark.parametrize("cols", [1, 3, 4, 8, 16, 20, 31, 32, 33, 36, 64, 100, 128, 250, 256, 300])
def test_long_rows_match_the_oracle(cols):
    from cbm import cbm_mkl_cpp as ops
    from oracle import oracle

    n = 900
    crow, col, val = _csr(n)
    x = torch.randn(n, cols, device="cuda")
    y = torch.full((n, cols), float("nan"), device="cuda")
    _run(crow, col, val, x, y)
    none = np.zeros(0, np.int32)
    ref = oracle.spmm_update(crow, col, val, x.cpu().numpy(), np.zeros(1, np.int32), none, none)
    np.testing.assert_array_equal(y.cpu().numpy(), ref)
    _run(crow, col, val, x, y, 0.5)
    gin = oracle.spmm_update_add(crow, col, val, x.cpu().numpy(), 0.5, np.zeros(1, np.int32), none, none)
    np.testing.assert_array_equal(y.cpu().numpy(), gin)
    ops.check_device()


@pytest.mark.parametrize("cols", [33, 256])
def test_bad_column_in_a_long_row_is_recorded_and_skipped(cols):
    from cbm import _lib
    from cbm import cbm_mkl_cpp as ops
    from oracle import oracle

    n = 900
    crow, col, val = _csr(n, seed=1)
    row = int(np.argmax(np.diff(crow)))
    at = crow[row] + 70
    x = torch.randn(n, cols, device="cuda")
    y = torch.empty_like(x)
    bad = col.copy()
    bad[at] = n + 5
    _run(crow, bad, val, x, y)
    status, info = ops.device_status()
    assert status == _lib.ERR_INDEX and info == at
    kept = val.copy()
    kept[at] = 0.0  # what the entry adds where it is left out
    none = np.zeros(0, np.int32)
    ref = oracle.spmm_update(crow, col, kept, x.cpu().numpy(), np.zeros(1, np.int32), none, none)
    np.testing.assert_array_equal(y.cpu().numpy(), ref)
