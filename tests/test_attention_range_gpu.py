"""Attention over the whole range of its numbers: far probabilities beside large values, sums of partials in one chain."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def C():
    from b200serve.ops import cuda_ops

    cuda_ops.lib()
    return cuda_ops


@pytest.mark.parametrize("decode", [False, True])
@pytest.mark.parametrize("D", [64, 128, 256])
def test_probability_below_the_normal_range_beside_a_large_value(C, D, decode):
    """Key 0 has log-2 score 130 above the others, and four of them have values of 2^127: each adds about 2^-130 * 2^127 to
    an output of 1."""
    n_q, n_kv, n = 8, 1, 100  # two pages
    q = torch.zeros(n, n_q, D, dtype=torch.bfloat16, device="cuda")
    kv = torch.zeros(3, 2, n_kv, 64, D, dtype=torch.bfloat16, device="cuda")
    q[:, :, 0] = 32.0
    kv[1, 0, 0, 0, 0] = torch.tensor(90.0 * D ** 0.5 / 32.0).bfloat16()
    kv[1, 1, 0, 0] = 1.0
    kv[1, 1, 0, 3:7] = 2.0 ** 127
    gate = torch.full((n, n_q * D), 30.0, dtype=torch.bfloat16, device="cuda")  # sigmoid rounds to 1
    table = torch.tensor([[1, 2]], dtype=torch.int32, device="cuda")
    if decode:
        got = C.flash_decode(q[-1:].contiguous(), gate[-1:].contiguous(), kv, table, torch.tensor([n - 1], device="cuda"), 1)
    else:
        got = C.flash_prefill(q, gate, kv, table, [0, n], [0])[-1:]
    C.check_errors(q.device)
    score = 32.0 * kv[1, 0, 0, 0, 0].double().item() * D ** -0.5
    p = torch.exp(torch.tensor(-score, dtype=torch.float64)).item()
    far = p * 4 * 2.0 ** 127
    assert 0.2 < far < 1.0
    # a probability of 2^-130 is a multiple of 2^-133 as bf16: off by a sixteenth at most; the sum is rounded to bf16
    assert ((got.double() - (1.0 + far)).abs() <= far / 16 + 2.0 ** -7).all()


@pytest.mark.parametrize("D", [64, 128, 256])
@pytest.mark.parametrize("Z", [4, 16, 17, 64, 512])
def test_partials_of_up_to_16_splits_are_added_in_one_fused_chain(C, D, Z):
    """Partials -4 s, 3 s and s with s = e^-x: 3 s is not a float, but a chain of fused multiply-adds never forms it (-4 s, -s,
    0). Products that are rounded before they are added leave a remainder."""
    rows, n_q = 64, 2
    acc = torch.full((rows, n_q, Z, D), float("nan"), device="cuda")
    ml = torch.zeros(rows, n_q, Z, 2, device="cuda")
    ml[..., 0] = float("-inf")
    acc[:, :, 0], ml[:, :, 0, 0], ml[:, :, 0, 1] = 0.0, 0.0, 1.0
    x = torch.linspace(0.01, 5.0, rows, device="cuda")[:, None]
    for z, v in ((1, -4.0), (2, 3.0), (3, 1.0)):
        acc[:, :, z], ml[:, :, z, 0], ml[:, :, z, 1] = v, -x, 1.0
    gate = torch.full((rows, n_q * D), 30.0, dtype=torch.bfloat16, device="cuda")
    out = torch.empty(rows, n_q * D, dtype=torch.bfloat16, device="cuda")
    C._check(C.lib().b200_attn_combine(acc.data_ptr(), ml.data_ptr(), gate.data_ptr(), out.data_ptr(), rows, n_q, D, Z, C._stream()),
             "attn_combine")
    assert (out == 0).all()


@pytest.mark.parametrize("width", [64, 200])
@pytest.mark.parametrize("n_q,n_kv,D", [(16, 2, 256), (4, 1, 64)])
def test_gate_that_starts_at_an_odd_element(C, width, n_q, n_kv, D):
    g = torch.Generator(device="cuda").manual_seed(D + width)
    pos = torch.tensor([700, 63, 1500], device="cuda")
    kv = torch.randn(60, 2, n_kv, 64, D, device="cuda", generator=g).bfloat16()
    table = torch.randint(1, 60, (3, width), device="cuda", generator=g).int()
    q = torch.randn(3, n_q, D, device="cuda", generator=g).bfloat16()
    flat = torch.randn(3 * n_q * D + 8, device="cuda", generator=g).bfloat16()
    for off in (1, 2, 3):
        gate = flat[off:off + 3 * n_q * D].view(3, n_q * D)
        got = C.flash_decode(q, gate, kv, table, pos, 1)
        C.check_errors(q.device)
        assert torch.equal(got, C.flash_decode(q, gate.clone(), kv, table, pos, 1))


@pytest.mark.parametrize("D,n_q,n_kv", [(256, 16, 2), (128, 4, 1), (64, 8, 8), (128, 6, 3)])
@pytest.mark.parametrize("B,longest", [(1, 1), (1, 64), (2, 513), (5, 5000), (150, 1100), (1030, 130)])
def test_decode_walk_over_the_runs_gives_the_bits_of_a_cta_per_run(D, n_q, n_kv, B, longest, monkeypatch):
    """Contexts of one key to many runs, more runs than CTAs, more sequences than one launch takes, a table wider than any of them."""
    from b200serve.ops import cuda_ops as C

    g = torch.Generator().manual_seed(B + D)
    lens = torch.randint(1, longest + 1, (B,), generator=g)
    lens[0] = longest
    pages = [(int(n) + 63) // 64 for n in lens]
    kv = torch.randn(sum(pages) + 1, 2, n_kv, 64, D, device="cuda").bfloat16()
    table = torch.zeros(B, max(pages) + 9, dtype=torch.int32)
    at = 1
    for b, k in enumerate(pages):
        table[b, :k] = torch.arange(at, at + k)
        at += k
    table, pos = table.cuda(), (lens - 1).cuda()
    q, gate = torch.randn(B, n_q, D, device="cuda").bfloat16(), torch.randn(B, n_q * D, device="cuda").bfloat16()
    got = C.flash_decode(q, gate, kv, table, pos, 1)
    monkeypatch.setattr(C, "DECODE_ATTN_SMALL_TILES", False)
    assert torch.equal(got, C.flash_decode(q, gate, kv, table, pos, 1))
    C.check_errors(q.device)


@pytest.mark.parametrize("G", [1, 2])
def test_decode_with_rows_of_the_page_table_at_any_distance(G):
    """One table for all sequences (distance 0), rows closer together than they are wide, a view of a wider table."""
    from b200serve.ops import cuda_ops as C

    n_q, n_kv, D, B, W = 8, 2, 128, 3, 20
    kv = torch.randn(W + 3, 2, n_kv, 64, D, device="cuda").bfloat16()
    row = torch.arange(W + 2, dtype=torch.int32, device="cuda") + 1
    wide = torch.zeros(B, W + 12, dtype=torch.int32, device="cuda")
    wide[:, :W] = row[:W]
    pos = torch.tensor([[64 * W - G, 700, 40][b] + j for b in range(B) for j in range(G)], device="cuda")
    q, gate = torch.randn(B * G, n_q, D, device="cuda").bfloat16(), torch.randn(B * G, n_q * D, device="cuda").bfloat16()
    for table in (row[None, :W].expand(B, W), row.as_strided((B, W), (1, 1)), wide[:, :W], wide[:1, :W].expand(B, W)):
        want = C.flash_decode(q, gate, kv, table.contiguous(), pos, G)
        assert torch.equal(C.flash_decode(q, gate, kv, table, pos, G), want) and torch.isfinite(want.float()).all()
    C.check_errors(q.device)
