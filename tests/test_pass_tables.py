"""The index tables of a ragged prefill pass against their definitions, on the CPU."""

import pytest
import torch

from b200serve.models.qwen36 import PackedBatch
from b200serve.ops import cuda_ops


@pytest.mark.parametrize("lens", [[1], [64], [65, 1, 200], [3, 0, 130], [7, 64, 63, 128]])
def test_batch_and_span_tables(lens):
    n, dev = len(lens), torch.device("cpu")
    toks = [list(range(10 * i, 10 * i + m)) for i, m in enumerate(lens)]
    pos0 = [64 * i for i in range(n)]
    table = torch.arange(n * 5, dtype=torch.int32).view(n, 5)
    for tokens in (toks, [tuple(t) for t in toks]):
        b = PackedBatch.prefill(tokens, [i + 3 for i in range(n)], pos0, table, "cpu")
        assert b.tokens.dtype == b.positions.dtype == torch.int64 and b.seq_of_row.dtype == b.slots.dtype == torch.int32
        assert b.tokens.tolist() == [t for ts in toks for t in ts]
        assert b.positions.tolist() == [p + j for p, m in zip(pos0, lens) for j in range(m)]
        assert b.seq_of_row.tolist() == [i for i, m in enumerate(lens) for _ in range(m)]
        assert b.slots.tolist() == [i + 3 for i in range(n)] and torch.equal(b.block_tables, table) and b.G == 0
    assert torch.equal(PackedBatch.prefill(toks, [0] * n, pos0, table.long(), "cpu").block_tables, table.long())
    starts = b.seg_starts
    T = starts[-1]
    n_chunks, chunks, per_seg, seq, st, slots = cuda_ops._gdn_prefill_meta(starts, b.seg_slots, T, dev)
    ref = [[i, r, min(64, starts[i + 1] - r), int(r == starts[i])] for i in range(n) for r in range(starts[i], starts[i + 1], 64)]
    assert n_chunks == len(ref) and chunks.view(-1, 4).tolist() == ref
    assert per_seg.view(-1, 2).tolist() == [[sum(-(-m // 64) for m in lens[:i]), -(-lens[i] // 64)] for i in range(n)]
    assert seq.tolist() == b.seq_of_row.tolist() and st.tolist() == starts and slots.tolist() == b.seg_slots


def test_batch_from_other_kinds_of_sequences():
    """Tokens and slots in any container of whole numbers, bytes among them: one token per byte."""
    table = torch.zeros(2, 4, dtype=torch.int32)
    for toks in ([b"abcdefgh", bytearray(b"xyz")], [torch.arange(97, 105), (120, 121, 122)], [range(97, 105), [120, 121, 122]]):
        for slots in ([4, 9], (4, 9), torch.tensor([4, 9])):
            b = PackedBatch.prefill(toks, slots, [0, 64], table, "cpu")
            assert b.tokens.tolist() == list(range(97, 105)) + [120, 121, 122] and b.slots.tolist() == [4, 9]


def test_span_tables_are_made_for_every_call():
    """Two calls with the same spans: what becomes of the first one's tables is nothing to the second."""
    dev = torch.device("cpu")
    for t in cuda_ops._gdn_prefill_meta([0, 70, 75], [2, 5], 75, dev)[1:]:
        t.fill_(-1)
    n, chunks, per_seg, seq, starts, slots = cuda_ops._gdn_prefill_meta([0, 70, 75], [2, 5], 75, dev)
    assert n == 3 and chunks.view(-1, 4).tolist() == [[0, 0, 64, 1], [0, 64, 6, 0], [1, 70, 5, 1]]
    assert per_seg.tolist() == [0, 2, 2, 1] and seq.tolist() == [0] * 70 + [1] * 5
    assert starts.tolist() == [0, 70, 75] and slots.tolist() == [2, 5]


@pytest.mark.parametrize("lens", [[], [1], [64], [65, 1, 200], [3, 0, 130], [0, 0], [7, 64, 63, 128], [0, 5, 0, 70, 1, 64, 129, 33, 16, 17, 0]])
@pytest.mark.parametrize("rows", [16, 32, 64, 128, None])
@pytest.mark.parametrize("few", [0, 8, 100])  # whole arrays, the rule, a loop over the spans
def test_tables_of_a_pass_against_their_definitions(lens, rows, few, monkeypatch):
    from b200serve.ops import spans

    monkeypatch.setattr(spans, "FEW", few)
    n, starts = len(lens), [sum(lens[:i]) for i in range(len(lens) + 1)]
    slots, pos0 = [3 + i for i in range(n)], [64 * i for i in range(n)]
    t = spans.span_tables(starts, slots, pos0, rows, torch.device("cpu"))
    nseg, n_chunks, chunks, per_span, seq, st, sl = t.gdn
    ref = [[i, r, min(64, starts[i + 1] - r), int(r == starts[i])] for i in range(n) for r in range(starts[i], starts[i + 1], 64)]
    assert nseg == n and n_chunks == len(ref) and chunks.view(-1, 4).tolist() == ref
    assert per_span.view(-1, 2).tolist() == [[sum(-(-m // 64) for m in lens[:i]), -(-m // 64)] for i, m in enumerate(lens)]
    assert seq.tolist() == [i for i, m in enumerate(lens) for _ in range(m)] and st.tolist() == starts and sl.tolist() == slots
    if rows is None:
        assert t.flash is None
    else:
        ref = [[i, p, starts[i], m] for i, m in enumerate(lens) for p in range(0, m, rows)]
        assert t.flash[:2] == (rows, len(ref)) and t.flash[2].view(-1, 4).tolist() == ref and t.flash[3].tolist() == pos0
        assert (t.flash[2].data_ptr() - chunks.data_ptr()) % 16 == 0 and (per_span.data_ptr() - chunks.data_ptr()) % 16 == 0
    assert t.of(list(starts), list(slots), list(pos0), rows) and not t.of(starts, [s + 1 for s in slots] + [0], pos0, rows)
