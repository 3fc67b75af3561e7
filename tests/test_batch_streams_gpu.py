"""The tensors and span tables of a prefill pass, used on another stream than the one they were made on, and under capture."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _batch(seed, lens=(65, 1, 200)):
    from b200serve.models.qwen36 import PackedBatch

    g = torch.Generator().manual_seed(seed)
    toks = [torch.randint(0, 1 << 40, (n,), generator=g).tolist() for n in lens]
    pos0 = [64 * (seed + i) for i in range(len(lens))]
    table = torch.randint(0, 1 << 20, (len(lens), 9), generator=g).int()
    slots = [seed + 3 * i for i in range(len(lens))]
    return PackedBatch.prefill(toks, slots, pos0, table, "cuda"), toks, slots, pos0, table


def test_batch_is_on_the_device_for_every_stream():
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(a):
        _batch(1)  # the memory that the next batch takes holds this one's numbers
        torch.cuda.synchronize()
        torch.cuda._sleep(200_000_000)  # about 0.1 s: what the stream is busy with when the batch is made
        batch, toks, slots, pos0, table = _batch(2)
    with torch.cuda.stream(b):
        got = [t.clone() for t in (batch.tokens, batch.positions, batch.seq_of_row, batch.slots, batch.block_tables)]
    b.synchronize()
    assert got[0].tolist() == [t for ts in toks for t in ts]
    assert got[1].tolist() == [p + j for p, ts in zip(pos0, toks) for j in range(len(ts))]
    assert got[2].tolist() == [i for i, ts in enumerate(toks) for _ in ts]
    assert got[3].tolist() == slots and torch.equal(got[4].cpu(), table)
    torch.cuda.synchronize()


def test_span_tables_are_on_the_device_for_every_stream():
    from b200serve.ops import cuda_ops

    dev = torch.device("cuda", 0)
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(a):
        cuda_ops._gdn_prefill_meta([0, 65, 66, 266], [4, 5, 6], 266, dev)
        torch.cuda.synchronize()
        torch.cuda._sleep(200_000_000)
        cuda_ops._gdn_prefill_meta([0, 200, 201, 266], [7, 8, 9], 266, dev)
    with torch.cuda.stream(b):
        n, chunks, per_seg, seq, starts, slots = cuda_ops._gdn_prefill_meta([0, 200, 201, 266], [7, 8, 9], 266, dev)
        got = [t.clone() for t in (per_seg, seq, starts, slots)]
    b.synchronize()
    assert got[0].tolist() == [0, 4, 4, 1, 5, 2] and got[1].tolist() == [0] * 200 + [1] + [2] * 65
    assert got[2].tolist() == [0, 200, 201, 266] and got[3].tolist() == [7, 8, 9]
    torch.cuda.synchronize()


def test_batch_under_capture_is_refused():
    _batch(1)
    x = torch.zeros(4, device="cuda")
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        x.add_(1.0)
        with pytest.raises(RuntimeError, match="captur"):
            _batch(2)
    graph.replay()
    assert x.tolist() == [1.0] * 4


@pytest.mark.parametrize("heads", [8, 4])  # query heads of the one key head: the batch's own tile table, and one built on demand
def test_captured_pass_keeps_its_tables_while_other_passes_run(heads):
    from b200serve.config import ModelConfig
    from b200serve.models.checkpoint import random_weights
    from b200serve.models.qwen36 import Model, PackedBatch
    from b200serve.ops import cuda_ops

    cfg = ModelConfig.tiny(num_attention_heads=heads, head_dim=64)
    model = Model(random_weights(cfg, seed=0, device="cuda", dtype=torch.bfloat16, std=0.05), 40, 6, ops=cuda_ops)
    toks = torch.randint(0, cfg.vocab_size, (400,), generator=torch.Generator().manual_seed(3)).tolist()
    table = torch.arange(1, 29, dtype=torch.int32).view(4, 7)

    def run(spans, batch=None):
        model.conv_state.zero_()
        model.rec_state.zero_()
        model.kv.zero_()
        batch = batch or PackedBatch.prefill([toks[a:b] for a, b in spans], list(range(1, len(spans) + 1)), [0] * len(spans),
                                             table[: len(spans)], "cuda")
        return model.forward(batch), batch

    spans, others = [(0, 70), (10, 11), (5, 135)], [[(0, 300)], [(0, 20), (20, 150)], [(3, 9), (9, 100), (0, 1), (7, 77)]]
    want, batch = run(spans)
    want = want.clone()
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        got, _ = run(spans, batch)
    alone = [run(s)[0].clone() for s in others]
    graph.replay()
    assert torch.equal(got, want)
    for s, h in zip(others, alone):  # and two passes in turn on two streams
        a = torch.cuda.Stream()
        a.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(a):
            again, _ = run(s)
        torch.cuda.current_stream().wait_stream(a)
        assert torch.equal(again, h)
    graph.replay()
    assert torch.equal(got, want)
    cuda_ops.check_errors(got.device)
