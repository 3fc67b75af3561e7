"""Kernels that start while the one before them still runs read its results only behind their dependency wait."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [1, 32, 128, 2048])
def test_combine_right_behind_the_kernel_that_writes_its_weights_and_positions(T):
    from b200serve.ops import cuda_ops as C

    E, k, H, dev = 64, 8, 256, "cuda"
    P = k + 1
    g = torch.Generator(device=dev).manual_seed(T)
    pairs = torch.randn(T * P, H, device=dev, generator=g).bfloat16()
    res = torch.randn(T, H, device=dev, generator=g).bfloat16()
    norm_w = torch.randn(H, device=dev, generator=g).bfloat16() * 0.1
    logits = torch.randn(8, T, E + 1, device=dev, generator=g)
    wts = torch.zeros(T, P, device=dev)
    idx, perm, inv, src = (torch.zeros(T * P, dtype=torch.int32, device=dev) for _ in range(4))
    offsets = torch.zeros(E + 2, dtype=torch.int32, device=dev)
    max_tiles = min(E + 1, T * P) + T * P // 16 + 1
    tiles, n = torch.zeros(max_tiles, 4, dtype=torch.int32, device=dev), torch.zeros(1, dtype=torch.int32, device=dev)
    new, y = torch.empty_like(res), torch.empty_like(res)
    err, ticket = C.err_word(res.device), C._ticket(res.device)

    def route(lg):
        return C.lib().b200_moe_route_plan(
            lg.data_ptr(), E + 1, T, E, k, 1, wts.data_ptr(), idx.data_ptr(), None, E + 1, 16, offsets.data_ptr(),
            tiles.data_ptr(), n.data_ptr(), max_tiles, perm.data_ptr(), inv.data_ptr(), err.data_ptr(), src.data_ptr(),
            ticket.data_ptr(), C._stream())

    def combine():
        return C.lib().b200_moe_combine_norm(pairs.data_ptr(), wts.data_ptr(), inv.data_ptr(), T, P, H, res.data_ptr(),
                                             norm_w.data_ptr(), new.data_ptr(), y.data_ptr(), 1e-6, C._stream())

    for i in range(32):
        assert route(logits[i % 8]) == 0 and combine() == 0  # nothing between the two launches
        got = y.clone()
        torch.cuda.synchronize()
        assert combine() == 0
        assert torch.equal(got, y), i
        # what the next pass must not see: zero weights, every pair at row 0
        wts.zero_()
        inv.zero_()
    C.check_errors(res.device)


@pytest.mark.parametrize("B", [1, 70])
@pytest.mark.parametrize("writer", ["reset_slot", "fill", "ring_commit", "prefill", "int64 slots", "projection"])
def test_decode_right_behind_a_kernel_that_writes_its_states_or_slots(B, writer):
    """The outcome is that of the same calls with the GPU waited for between them."""
    from b200serve.ops import cuda_ops as C

    n_k, n_v, d, dev = 4, 8, 128, "cuda"
    ch, g = 2 * n_k * d + n_v * d, torch.Generator(device="cuda").manual_seed(B)

    def rnd(*shape, scale=1.0):
        return torch.randn(*shape, device=dev, generator=g) * scale

    width = ch + n_v * d + 2 * n_v
    x, w = rnd(B, 64).bfloat16(), rnd(width, 64, scale=0.2).bfloat16()
    mixed = C.linear(x, w)
    args = (rnd(ch, 4, scale=0.3).bfloat16(), rnd(n_v, scale=0.1), rnd(n_v, scale=0.1), rnd(d, scale=0.1).bfloat16(), n_k, n_v, d, d, 1e-6)
    conv0, rec0 = rnd(1, B + 1, ch, 3).bfloat16(), rnd(1, B + 1, n_v, d, d)
    ring = rnd(1, B, 2, ch, 3).bfloat16(), rnd(1, B, 2, n_v, d, d)
    slots = torch.arange(1, B + 1, dtype=torch.int32, device=dev)
    keep = torch.zeros(B, dtype=torch.int64, device=dev)
    rows = rnd(70, width).bfloat16()

    def run(wait):
        conv, rec = conv0.clone(), rec0.clone()
        sl, m, last = slots, mixed, {}
        torch.cuda.synchronize()
        if writer == "reset_slot":
            for s in range(1, B + 1):
                C.reset_slot(conv, rec, s)
        elif writer == "fill":
            rec.zero_()
            conv.zero_()
        elif writer == "ring_commit":
            C.ring_commit(conv, rec, ring, slots, keep)
        elif writer == "prefill":
            C.gdn_prefill(rows, [0, 70], [1], conv[0], rec[0], *args)
        elif writer == "int64 slots":
            sl = slots.long()
        else:
            C.reset_slot(conv, rec, 1)
            m, last = C.linear(x, w), {"behind_projection": True}
        if wait:
            torch.cuda.synchronize()
        out = C.gdn_decode(m, sl, conv[0], rec[0], *args, **last)
        return out, conv, rec

    want = run(True)
    for i in range(20):
        assert all(torch.equal(a, b) for a, b in zip(run(False), want)), i
    C.check_errors(mixed.device)
