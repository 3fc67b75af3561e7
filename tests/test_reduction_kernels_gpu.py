"""The kernels that merge partial results: attention partials of a split context, expert outputs of a row."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def C():
    from b200serve.ops import cuda_ops

    cuda_ops.lib()
    return cuda_ops


def _combine(C, acc, ml, gate):
    rows, n_q, Z, D = acc.shape
    out = torch.empty(rows, n_q * D, dtype=torch.bfloat16, device="cuda")
    C._check(C.lib().b200_attn_combine(acc.data_ptr(), ml.data_ptr(), gate.data_ptr(), out.data_ptr(), rows, n_q, D, Z,
                                       C._stream()), "attn_combine")
    return out


@pytest.mark.parametrize("D", [64, 128, 256])
@pytest.mark.parametrize("valid,Z", [(1, 1), (1, 8), (15, 15), (13, 16), (16, 17), (33, 63), (7, 64), (64, 64), (177, 512), (512, 512)])
def test_attention_partials_against_64_bits(C, D, valid, Z):
    g = torch.Generator(device="cuda").manual_seed(valid * 1000 + Z)
    rows, n_q = 3, 2
    acc = torch.randn(rows, n_q, Z, D, device="cuda", generator=g)
    ml = torch.stack([torch.randn(rows, n_q, Z, device="cuda", generator=g) * 4,
                      torch.rand(rows, n_q, Z, device="cuda", generator=g) * 30 + 1], -1).contiguous()
    acc[:, :, valid:] = float("nan")  # a split without keys writes only its (-inf, 0) pair
    ml[:, :, valid:, 0], ml[:, :, valid:, 1] = float("-inf"), 0.0
    gate = torch.randn(rows, n_q * D, device="cuda", generator=g).bfloat16()
    got = _combine(C, acc, ml, gate)
    w = torch.exp(ml[..., 0].double() - ml[..., 0].double().amax(-1, keepdim=True))
    o = (w[..., :valid, None] * acc[:, :, :valid].double()).sum(2) / (w * ml[..., 1].double()).sum(-1)[..., None]
    ref = o.reshape(rows, -1) * torch.sigmoid(gate.double())
    # two roundings to bf16 (8 significant bits: at most 2^-8 each) and fp32 sums of at most 512 terms
    assert ((got.double() - ref).abs() <= 2.0 ** -7 * 1.01 * ref.abs() + 1e-5).all()
    # the order of the sums follows the partials that hold keys, not the width of the table behind them
    wide = torch.full((rows, n_q, 520, D), float("nan"), device="cuda")
    wide_ml = torch.zeros(rows, n_q, 520, 2, device="cuda")
    wide_ml[..., 0] = float("-inf")
    wide[:, :, :valid], wide_ml[:, :, :valid] = acc[:, :, :valid], ml[:, :, :valid]
    assert torch.equal(_combine(C, wide, wide_ml, gate), got)


@pytest.mark.parametrize("T,P,H", [(1, 1, 8), (3, 9, 2048), (5, 10, 2056), (130, 8, 128), (2, 33, 4096)])
def test_expert_outputs_of_a_row(C, T, P, H):
    g = torch.Generator(device="cuda").manual_seed(T + P)
    pairs = torch.randn(T * P, H, device="cuda", generator=g).bfloat16()
    wts = torch.rand(T, P, device="cuda", generator=g).bfloat16().float()
    inv = torch.randperm(T * P, device="cuda", generator=g).int().view(T, P)
    inv[torch.rand(T, P, device="cuda", generator=g) < 0.2] = -1  # pairs that another rank serves
    src = pairs.double()[inv.clamp(min=0).long()] * (wts * (inv >= 0)).double()[..., None]
    ref = src.sum(1)
    out = torch.empty(T, H, device="cuda", dtype=torch.float32)
    C._check(C.lib().b200_moe_combine(pairs.data_ptr(), wts.data_ptr(), inv.data_ptr(), T, P, H, None, out.data_ptr(),
                                      C._stream()), "moe_combine")
    assert ((out.double() - ref).abs() <= 1e-6 * P * src.abs().sum(1) + 1e-12).all()
    res = torch.randn(T, H, device="cuda", generator=g).bfloat16()
    norm_w = torch.randn(H, device="cuda", generator=g).bfloat16() * 0.1
    new, y = torch.empty_like(res), torch.empty_like(res)
    C._check(C.lib().b200_moe_combine_norm(pairs.data_ptr(), wts.data_ptr(), inv.data_ptr(), T, P, H, res.data_ptr(),
                                           norm_w.data_ptr(), new.data_ptr(), y.data_ptr(), 1e-6, C._stream()), "combine_norm")
    ref_new, ref_y = C.add_rmsnorm(out.bfloat16(), res, norm_w, 1e-6)
    assert torch.equal(new, ref_new) and torch.equal(y, ref_y)


@pytest.mark.parametrize("T,V", [(1, 128), (2, 1000), (17, 129), (64, 4096), (200, 777), (256, 1280), (300, 2500), (3, 70001), (150, 70001)])
def test_greedy_head_takes_the_lowest_id_among_equal_logits(C, T, V):
    """Small whole numbers: every logit is exact, and a row has many columns with the same largest one."""
    g = torch.Generator(device="cuda").manual_seed(T * 7 + V)
    x = torch.randint(-2, 3, (T, 64), device="cuda", generator=g).bfloat16()
    w = torch.randint(-1, 2, (V, 64), device="cuda", generator=g).bfloat16()
    w[V // 2:] = w[: V - V // 2].clone()  # every logit appears twice
    logits = x.double() @ w.double().t()
    top = logits.amax(1, keepdim=True)
    first = torch.where(logits == top, torch.arange(V, device="cuda"), V).amin(1)
    idx, val = C.lm_head_argmax(x, w, return_value=True)
    assert torch.equal(idx, first) and torch.equal(val.double(), top[:, 0])


@pytest.mark.parametrize("n_q,n_kv,D,rot", [(16, 2, 256, 64), (8, 1, 64, 16), (4, 2, 128, 128), (4, 1, 32, 8), (32, 4, 64, 20)])
def test_attention_prep_heads_and_rotary_dims(C, n_q, n_kv, D, rot):
    """More heads than warps of a CTA, rotary dims that end inside a lane's run, every row in a page of its own."""
    from b200serve.ops import torch_ops as O

    T, dev = 37, "cuda"
    g = torch.Generator(device=dev).manual_seed(D + rot)
    qkv = torch.randn(T, (2 * n_q + 2 * n_kv) * D + 8, device=dev, generator=g).bfloat16()[:, :-8]
    qn, kn = (torch.randn(D, device=dev, generator=g).bfloat16() * 0.1 for _ in range(2))
    positions = torch.randint(0, 4096, (T,), device=dev, generator=g)
    tables = torch.zeros(T, 64, dtype=torch.int32, device=dev)
    tables[torch.arange(T), positions // 64] = torch.arange(1, T + 1, dtype=torch.int32, device=dev)
    seq = torch.arange(T, dtype=torch.int32, device=dev)
    kv = torch.zeros(T + 1, 2, n_kv, 64, D, device=dev, dtype=torch.bfloat16)
    q = torch.empty(T, n_q, D, device=dev, dtype=torch.bfloat16)
    gate = torch.empty(T, n_q * D, device=dev, dtype=torch.bfloat16)
    rc = C.lib().b200_attn_prep(qkv.data_ptr(), qkv.stride(0), positions.data_ptr(), tables.data_ptr(), 64, seq.data_ptr(),
                                qn.data_ptr(), kn.data_ptr(), q.data_ptr(), gate.data_ptr(), kv.data_ptr(), T, n_q, n_kv, D,
                                rot, 1e7, 1e-6, T + 1, C.err_word(qkv.device).data_ptr(), C._stream())
    assert rc == 0
    C.check_errors(qkv.device)
    rq, rg, rk, rv = O.attn_prep(qkv.float(), positions, qn.float(), kn.float(), n_q, n_kv, D, rot, 1e7, 1e-6)
    rows = torch.arange(T, device=dev)
    assert torch.equal(gate, rg.bfloat16()) and torch.equal(kv[rows + 1, 1, :, positions % 64], rv.bfloat16())
    for got, ref in ((q, rq), (kv[rows + 1, 0, :, positions % 64], rk)):
        size = ref.abs().clone()  # a rotated pair mixes two dims: four roundings to bf16 (2^-8 each) of up to their norm
        half = rot // 2
        pair = (ref[..., :half] ** 2 + ref[..., half:2 * half] ** 2).sqrt()
        size[..., :half], size[..., half:2 * half] = pair, pair
        assert ((got.float() - ref).abs() <= 2.0 ** -6 * size * 1.5 + 1e-3).all()


@pytest.mark.parametrize("n_q,n_kv,D", [(16, 2, 256), (4, 1, 128), (2, 2, 64)])
@pytest.mark.parametrize("pos0,n", [(0, 1), (0, 64), (63, 2), (64, 65), (130, 40), (256, 193), (510, 300)])
def test_flash_pages_of_growing_scores(C, n_q, n_kv, D, pos0, n):
    """Even and odd page counts; scores that grow along the context, so that the running maximum of a row, which two groups
    of threads pass to and fro, keeps moving and the output is rescaled on many pages."""
    from b200serve.ops import torch_ops as O

    g = torch.Generator(device="cuda").manual_seed(n + pos0)
    pages = (pos0 + n + 63) // 64
    kv = torch.randn(pages + 1, 2, n_kv, 64, D, device="cuda", generator=g)
    table = (torch.randperm(pages, device="cuda", generator=g) + 1).int().view(1, -1)
    for i, pg in enumerate(table[0].tolist()):
        kv[pg, 0] *= 1.0 + 1.5 * i  # log2 of a row's largest score grows by about 8 per page
    kv = kv.bfloat16()
    q = torch.randn(n, n_q, D, device="cuda", generator=g).bfloat16()
    gate = torch.randn(n, n_q * D, device="cuda", generator=g).bfloat16()
    got = C.flash_prefill(q, gate, kv, table, [0, n], [pos0])
    C.check_errors(q.device)
    ref = O.paged_attention(q.float(), gate.float(), kv.float(), table, [0, n], [pos0])
    # probabilities, output and gated output are rounded to bf16 (2^-8 each), on values of up to about four
    assert (got.float() - ref).abs().max().item() <= 3 * 2.0 ** -8 * 5


@pytest.mark.parametrize("T", [1, 16, 17, 130, 256])
@pytest.mark.parametrize("V", [200, 1000, 66000])
def test_greedy_head_with_infinite_and_undefined_logits(C, T, V):
    """Rows whose largest logit is infinite, rows of minus infinity but for one id, and rows of NaN beside ordinary ones."""
    w = _whole(V, 64, seed=V)
    w[:, 0] = 0.0
    high = torch.tensor([5, 127, 128, V - 1], device="cuda") % V
    w[high, 0] = float("inf")
    x = _whole(T, 64, seed=T)
    x[:, 0] = torch.tensor([1.0, -1.0, 2.0], device="cuda").repeat(T // 3 + 1)[:T]  # +inf or -inf at `high`
    if T > 2:
        x[T // 2] = float("nan")
    logits = x.double() @ w.double().t()
    top = logits.amax(1, keepdim=True)
    first = torch.where(logits == top, torch.arange(V, device="cuda"), V).amin(1)
    idx, val = C.lm_head_argmax(x, w, return_value=True)
    ok = ~torch.isnan(x).any(1)
    assert torch.equal(idx[ok], first[ok]) and torch.equal(val[ok].double(), top[ok, 0])
    assert (idx[~ok] >= V).all()  # no id: the embedding of such a row sets the error word
    w[:, 0] = float("inf")  # every logit minus infinity: the lowest id
    x[:, 0] = -1.0
    assert (C.lm_head_argmax(x[: max(1, T // 2)], w) == 0).all()


def _whole(rows, cols, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randint(-2, 3, (rows, cols), device="cuda", generator=g).bfloat16()


@pytest.mark.parametrize("H", [64, 2048, 2056])
def test_embedding_with_the_first_norm_is_the_two_ops(H):
    from b200serve.ops import cuda_ops as C

    g = torch.Generator(device="cuda").manual_seed(H)
    table = torch.randn(50, H, device="cuda", generator=g).bfloat16()
    w = (torch.randn(H, device="cuda", generator=g) * 0.1).bfloat16()
    tokens = torch.tensor([0, 49, 7, 7, -1, 50, 31], device="cuda")  # two outside the table
    x, y = C.embed_rmsnorm(tokens, table, w, 1e-6)
    want = C.embed(tokens, table)
    assert torch.equal(x, want) and torch.equal(y, C.add_rmsnorm(want, None, w, 1e-6)[1])


@pytest.mark.parametrize("slot", [0, 3, -1])
def test_reset_slot_zeroes_one_slot_of_every_layer(slot):
    from b200serve.ops import cuda_ops as C

    conv = torch.randn(3, 5, 264, 3, device="cuda").bfloat16()
    rec = torch.randn(3, 5, 2, 32, 33, device="cuda")[:, :, :, :, :32].contiguous()
    want_c, want_r = conv.clone(), rec.clone()
    want_c[:, slot], want_r[:, slot] = 0.0, 0.0
    C.reset_slot(conv, rec, slot)
    assert torch.equal(conv, want_c) and torch.equal(rec, want_r)
    with pytest.raises(IndexError):
        C.reset_slot(conv, rec, 5)


@pytest.mark.parametrize("form", ["layers apart", "slots apart", "rows of 8 bytes", "odd start", "no layers", "fewer conv slots"])
def test_reset_slot_of_states_that_the_kernel_does_not_take(form):
    from b200serve.ops import cuda_ops as C

    conv, rec = torch.randn(6, 5, 264, 3, device="cuda").bfloat16(), torch.randn(6, 5, 2, 32, 32, device="cuda")
    if form == "layers apart":
        conv, rec = conv[::2], rec[::2]
    elif form == "slots apart":
        conv, rec = conv[:, 1:4], rec[:, 1:4]
    elif form == "rows of 8 bytes":
        conv = torch.randn(6, 5, 4, 1, device="cuda").bfloat16()
    elif form == "odd start":
        rec = torch.randn(6 * 5 * 2048 + 1, device="cuda")[1:].view(6, 5, 2, 32, 32)
    elif form == "no layers":
        conv, rec = conv[:0], rec[:0]
    else:
        conv = conv[:, :3].contiguous()
    want_c, want_r = conv.clone(), rec.clone()
    want_c[:, 2], want_r[:, 2] = 0.0, 0.0
    C.reset_slot(conv, rec, 2)
    assert torch.equal(conv, want_c) and torch.equal(rec, want_r)
