"""Host side of paged decode, with no launch: what the kernel reads as 16-byte vectors starts on 16 bytes."""
import ctypes
from types import SimpleNamespace

import pytest
import torch

from inquant import _native as N
from inquant.batched import DecodeBatch, PagedSequenceState
from inquant.triton_attention import SharedDecodeWorkspace
from inquant_vllm import kernels
from inquant_vllm.layout import PageLayout

HEADS, Q_HEADS, BLOCK = 2, 8, 16


def _off(x, elements):
    """The same tensor, contiguous, ``elements`` into a buffer that starts on 16 bytes."""
    buffer = torch.empty(x.numel() + 16, dtype=x.dtype)
    assert buffer.data_ptr() % 16 == 0
    view = buffer[elements:elements + x.numel()].view(x.shape)
    view.copy_(x)
    return view


@pytest.fixture
def launches(monkeypatch):
    """The argument structures that would be launched, with the values at their addresses."""
    seen, library = [], N.library()

    def decode(args, _stream):
        seq = args._obj.seq_host[0]
        rows = {name: getattr(seq, name) for name in ("query", "pool", "sink_key", "sink_value", "tail_key", "tail_value")}
        assert all(address % 16 == 0 for address in rows.values()), rows
        seen.append({name: ctypes.string_at(rows[name], 256) for name in ("query", "sink_key", "sink_value", "tail_key", "tail_value")})
        return N.OK
    monkeypatch.setattr(N, "library", lambda: SimpleNamespace(
        inq_decode_attention=decode, inq_decode_units=library.inq_decode_units, inq_decode_workspace_floats=library.inq_decode_workspace_floats))
    monkeypatch.setattr(N, "require_cuda", lambda *_: None)
    monkeypatch.setattr(N, "stream_handle", lambda _device: 0)
    monkeypatch.setattr(N, "stream_identity", lambda _device: (0, 0))
    return seen


def _inputs():
    layout, gen = PageLayout(BLOCK, HEADS), torch.Generator().manual_seed(1)
    query, dense = (torch.randn(s, generator=gen).to(torch.bfloat16) for s in ((1, Q_HEADS, 128), (2, HEADS, BLOCK + 4, 128)))
    return layout, query, dense, torch.zeros((3, layout.page_bytes), dtype=torch.uint8), torch.zeros(2, dtype=torch.int32)


def test_unaligned_query_and_dense_rows_are_copied(launches):
    layout, query, dense, pool, ids = _inputs()

    def run(query, dense):
        kernels.paged_decode(query, pool, ids, dense, 2, 5, 4, layout, SharedDecodeWorkspace(), 0.1)
    run(query, dense)
    for elements in (1, 4):
        run(_off(query, elements), dense)
        run(query, _off(dense, elements))
    assert len(launches) == 5 and all(rows == launches[0] for rows in launches)


def test_unaligned_pages_are_refused(launches):
    layout, query, dense, pool, ids = _inputs()
    with pytest.raises(ValueError, match="start on 16 bytes"):
        kernels.paged_decode(query, _off(pool, 1), ids, dense, 2, 5, 4, layout, SharedDecodeWorkspace(), 0.1)
    assert not launches


@pytest.mark.parametrize("what", ["dense", "pool"])
def test_a_batch_refuses_unaligned_rows_and_pages(what):
    layout, _, dense, pool, ids = _inputs()
    given = {"dense": dense, "pool": pool}
    given[what] = _off(given[what], 1)
    sequence = PagedSequenceState(given["pool"], ids, 2, given["dense"], 5, 4, layout)
    with pytest.raises(ValueError, match="start on 16 bytes"):
        DecodeBatch([sequence], Q_HEADS, torch.bfloat16)
