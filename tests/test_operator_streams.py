"""The reference operators' workspaces: one per stream (CPU, no product runs), and tree
products on several streams at once (GPU)."""
import numpy as np
import pytest
import torch


@pytest.fixture
def ops(monkeypatch):
    from cbm import cbm_mkl_cpp

    monkeypatch.setattr(cbm_mkl_cpp, "_WORKSPACE", {})
    return cbm_mkl_cpp


def test_every_stream_has_its_own_workspace(ops, monkeypatch):
    monkeypatch.setattr(ops, "_capturing", lambda: False)
    cpu = torch.device("cpu")
    a, b = ops._workspace(cpu, 100, 1), ops._workspace(cpu, 100, 2)
    assert a.data_ptr() != b.data_ptr() and not a.any() and not b.any()
    assert ops._workspace(cpu, 50, 1) is a
    a[0], a[300] = 7, 9
    grown = ops._workspace(cpu, 10_000, 1)
    assert grown.numel() >= 256 + 8 * 10_000 and grown[0] == 7 and not grown[256:].any()
    assert ops._workspace(cpu, 100, 2) is b


def test_workspaces_are_bounded_and_their_status_kept(ops, monkeypatch):
    monkeypatch.setattr(ops, "_capturing", lambda: False)
    monkeypatch.setattr(ops, "_CARRIED", {})
    monkeypatch.setattr(torch.cuda, "synchronize", lambda device=None: None)
    monkeypatch.setattr(ops, "_status", lambda ws, stream: (int(ws[0]), 5))
    cpu = torch.device("cpu")
    ops._workspace(cpu, 1, 100)[0] = 2
    for stream in range(ops._MAX_STREAMS + 3):
        ops._workspace(cpu, 1, stream)
    assert len(ops._WORKSPACE) == ops._MAX_STREAMS and (None, 100) not in ops._WORKSPACE
    assert ops._CARRIED == {None: (2, 5)}


def test_a_capture_takes_a_workspace_that_is_there_and_keeps_it(ops, monkeypatch):
    cpu = torch.device("cpu")
    monkeypatch.setattr(ops, "_capturing", lambda: False)
    a = ops._workspace(cpu, 100, 1)
    monkeypatch.setattr(ops, "_capturing", lambda: True)
    assert ops._workspace(cpu, 100, 2) is a
    own = ops._workspace(cpu, 10_000, 2)  # none is large enough
    assert own is not a and not own.any()
    monkeypatch.setattr(ops, "_capturing", lambda: False)
    assert ops._workspace(cpu, 9_000, 2) is not own
    ops._workspace(cpu, 20_000, 1)  # stream 1's workspace is replaced, the graphs keep theirs
    assert any(w is a for w in ops._WORKSPACE.values()) and any(w is own for w in ops._WORKSPACE.values())


@pytest.mark.gpu
def test_tree_products_on_several_streams_at_once():
    from cbm import cbm_mkl_cpp
    from cbm.cbm4dad import cbm4dad
    from cbm import synthetic

    rng = np.random.Generator(np.random.PCG64(0))
    n = 20_000
    ei = synthetic.near_duplicates(synthetic.community_graph(n, 32, 10, 2, rng=rng), n, 0.3, 0.1, rng=rng)
    op = cbm4dad(torch.from_numpy(ei), torch.ones(ei.shape[1]), alpha=0)
    crow = op.deltas.crow_indices()
    head = (crow[:-1].contiguous(), crow[1:].contiguous(), op.deltas.col_indices(), op.deltas.values())
    tail = (op.mca_offset, op.mca_src_idx, op.mca_dst_idx, op.D)
    xs = [torch.randn(n, 64, device="cuda") for _ in range(4)]
    want = [torch.empty_like(x) for x in xs]
    for x, y in zip(xs, want):
        cbm_mkl_cpp.s_spmm_fused_update_csr_int32(*head, x, *tail, y)
    cbm_mkl_cpp.check_device()
    streams = [torch.cuda.Stream() for _ in xs]
    got = [torch.full_like(x, float("nan")) for x in xs]
    torch.cuda.synchronize()
    for _ in range(20):
        for s, x, y in zip(streams, xs, got):
            with torch.cuda.stream(s):
                cbm_mkl_cpp.s_spmm_fused_update_csr_int32(*head, x, *tail, y)
    cbm_mkl_cpp.check_device()
    for y, w in zip(got, want):
        assert torch.equal(y, w)
