"""Buffers the wrappers keep per stream and replace when a call needs more: the old one stays allocated (a graph captured
before holds its address), and what is superseded stays below what is in use.  Host code only."""
import weakref

import pytest
import torch


@pytest.mark.parametrize("which", ["workspace", "plain_scratch", "row_max"])
def test_superseded_buffers_stay_allocated(monkeypatch, which):
    import fused_fp8_gemm as f
    import rwkvq_abi as abi
    monkeypatch.setattr(abi, "stream_ptr", lambda: 12345)
    monkeypatch.setattr(abi, "_superseded", [])
    monkeypatch.setattr(abi, "_workspaces", {})
    monkeypatch.setattr(abi, "_plain", {})
    monkeypatch.setattr(f, "_row_max", {})
    dev = torch.device("cpu")
    sizes = [1 << 20, (1 << 20) + 1, 3 << 20, (3 << 20) + 5, 20 << 20, 1 << 20]
    if which == "workspace":
        monkeypatch.setattr(abi, "_ws_need", {(i, 1, 1, 1): s for i, s in enumerate(sizes)})
        get = lambda i: abi.workspace(i, 1, 1, 1, dev)  # noqa: E731
    elif which == "plain_scratch":
        get = lambda i: abi.plain_scratch(sizes[i], dev)  # noqa: E731
    else:
        get = lambda i: f._row_max_scratch(dev, sizes[i])  # noqa: E731
    refs, ptrs = [], set()
    for i, s in enumerate(sizes):
        buf = get(i)
        assert buf.numel() >= s and buf.data_ptr() == get(i).data_ptr()
        if which != "plain_scratch":
            assert not bool(buf.any())
        if buf.data_ptr() not in ptrs:
            ptrs.add(buf.data_ptr())
            refs.append(weakref.ref(buf))
        del buf
    assert len(refs) > 2 and all(r() is not None for r in refs)
    assert sum(b.numel() for b in abi._superseded) <= get(0).numel()


def test_weight_only_workspace_is_asked_once_per_shape_and_device(monkeypatch):
    """The plan behind the size depends on the device's SM count: two unlike devices in one process each get their own."""
    import torch
    import rwkvq_abi as abi

    class Lib:
        asked = 0

        def rwkvq_tc_gemm_wa16_workspace_bytes(self, m, n, k, bits):
            Lib.asked += 1
            return 1000 + Lib.asked
    monkeypatch.setattr(abi, "lib", Lib)
    monkeypatch.setattr(abi, "_wa16_need", {})
    d0, d1 = torch.device("cuda", 0), torch.device("cuda", 1)
    assert [abi.wa16_workspace_bytes(100, 4096, 4096, 4, d) for d in (d0, d1, d0, d1)] == [1001, 1002, 1001, 1002]
    assert abi.wa16_workspace_bytes(100, 4096, 4096, 8, d0) == 1003
