"""The forms that the GEMM launchers pick by size: thin weight tiles, several k-blocks per stage, wide expert tiles."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def C():
    from b200serve.ops import cuda_ops

    cuda_ops.lib()
    return cuda_ops


def _bf(*shape, scale=1.0, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(*shape, device="cuda", generator=g) * scale).to(torch.bfloat16)


@pytest.mark.parametrize("N,K", [(257, 2048), (2048, 4096), (100, 256), (1000, 128), (9216, 2048), (12352, 2048), (4096, 320),
                                 (130, 64)])
def test_dense_forms_give_the_bits_of_the_plain_tile(C, N, K):
    w = _bf(N, K, scale=0.05, seed=1)
    packed = C.pack_weight(w.clone())
    for T in (1, 2, 15, 16, 17, 32, 33, 48, 49, 64, 65, 96, 128, 129, 160, 256, 257):
        x = _bf(T, K + 64, seed=T)[:, 32:32 + K]  # rows further apart than K, not at the start of the allocation
        for dt in (None, torch.float32):
            got = C.linear(x, packed, out_dtype=dt)[:, :N]
            # an explicit token tile is the plain form: 128 weight rows, one k-block per stage
            plain = C.linear(x, w, out_dtype=dt, bt=16)
            assert torch.equal(got, plain), (T, dt)
        ref = x.double() @ w.double().t()
        # fp32 sums of K products of bf16 numbers
        assert ((plain.double() - ref).abs() <= 2e-6 * K ** 0.5 * (x.double().norm(dim=1)[:, None] * w.double().norm(dim=1))).all()
    C.check_errors(x.device)


@pytest.mark.parametrize("T", [1, 2, 3, 4, 5, 8, 9, 40])
@pytest.mark.parametrize("inter,H", [(512, 2048), (128, 256), (256, 192)])
def test_expert_block_of_a_few_rows_with_packed_weights(C, T, inter, H):
    E, k = 24, 4
    x = _bf(T, H, seed=T)
    router, gu, dn = _bf(E + 1, H, scale=0.1, seed=2), _bf(E + 1, 2 * inter, H, scale=0.05, seed=3), _bf(E + 1, H, inter, scale=0.05, seed=4)
    plain = C.moe_block(x, router, gu, dn, E, k, True)
    got = C.moe_block(x, router, C.pack_weight(gu.clone(), gate_up=True), C.pack_weight(dn.clone()), E, k, True)
    C.check_errors(x.device)
    assert torch.equal(got, plain)


@pytest.mark.parametrize("T,E,k,H,I", [(600, 16, 4, 256, 128), (1100, 32, 8, 2048, 512), (515, 8, 2, 512, 192)])
@pytest.mark.parametrize("packed", [False, True])
def test_wide_expert_tiles_give_the_bits_of_the_64_row_tiles(C, T, E, k, H, I, packed):
    """Experts of every size around the tile: full tiles, last tiles of few rows, an expert without rows."""
    x = _bf(T, H, seed=T)
    router = _bf(E + 1, H, scale=0.3, seed=34)
    router[3] = -4.0 * x.float().mean(0).bfloat16()  # rarely picked
    wgu, wd = _bf(E + 1, 2 * I, H, scale=0.05, seed=35), _bf(E + 1, H, I, scale=0.05, seed=36)
    if packed:
        wgu, wd = C.pack_weight(wgu, gate_up=True), C.pack_weight(wd)
    keep = C.GATHER_MAX_BT, C.WIDE_MIN_ROWS
    try:
        C.WIDE_MIN_ROWS = 1
        wide = C.moe_block(x, router, wgu, wd, E, k, True)
        C.GATHER_MAX_BT = 64
        narrow = C.moe_block(x, router, wgu, wd, E, k, True)
    finally:
        C.GATHER_MAX_BT, C.WIDE_MIN_ROWS = keep
    C.check_errors(x.device)
    assert torch.equal(wide, narrow)


@pytest.mark.parametrize("T,E,k", [(1, 256, 8), (31, 64, 32), (32, 64, 32), (33, 64, 32), (32, 300, 7), (700, 40, 3)])
def test_routing_and_plan_of_tied_rows(C, T, E, k):
    """Quantised logits, so that ties are everywhere; the largest table that stays in shared memory, and one beyond it."""
    g = torch.Generator(device="cuda").manual_seed(T + E)
    logits = (torch.randn(T, E + 1, device="cuda", generator=g) * 3).round() / 2
    P, dev = k + 1, "cuda"
    wts = torch.empty(T, P, device=dev)
    idx, perm, inv, src = (torch.full((T * P,), -7, dtype=torch.int32, device=dev) for _ in range(4))
    offsets = torch.empty(E + 2, dtype=torch.int32, device=dev)
    max_tiles = min(E + 1, T * P) + T * P // 16 + 1
    tiles, n = torch.empty(max_tiles, 4, dtype=torch.int32, device=dev), torch.empty(1, dtype=torch.int32, device=dev)
    err = C.err_word(logits.device)
    rc = C.lib().b200_moe_route_plan(logits.data_ptr(), E + 1, T, E, k, 1, wts.data_ptr(), idx.data_ptr(), None, E + 1, 16,
                                     offsets.data_ptr(), tiles.data_ptr(), n.data_ptr(), max_tiles, perm.data_ptr(), inv.data_ptr(),
                                     err.data_ptr(), src.data_ptr(), C._ticket(logits.device).data_ptr(), C._stream())
    assert rc == 0
    C.check_errors(logits.device)
    # equal logits have equal probabilities: the lower expert id first
    order = torch.sort(logits[:, :E], dim=1, descending=True, stable=True).indices[:, :k]
    table = idx.view(T, P).long()
    assert torch.equal(table[:, :k], order) and (table[:, k] == E).all()
    pr = torch.softmax(logits[:, :E].double(), 1).gather(1, order)
    assert torch.allclose(wts[:, :k].double(), pr / pr.sum(1, keepdim=True), rtol=2.0 ** -8 * 1.01, atol=1e-7)  # bf16 weights
    assert torch.equal(offsets.long(), torch.nn.functional.pad(table.flatten().bincount(minlength=E + 1).cumsum(0), (1, 0)))
    assert torch.equal(perm.long().sort().values, torch.arange(T * P, device=dev)) and torch.equal(perm[inv.long()].long(), torch.arange(T * P, device=dev))
    assert torch.equal(table.flatten()[perm.long()], table.flatten().sort().values) and torch.equal(src, perm // P)


@pytest.mark.parametrize("T", [5, 300, 700])
def test_expert_block_of_rows_that_are_further_apart(C, T):
    """Row strides and starts that the in-GEMM row fetch does not take: the same rows, copied first."""
    E, k, H, I = 16, 4, 256, 128
    router, gu, dn = _bf(E + 1, H, scale=0.3, seed=2), _bf(E + 1, 2 * I, H, scale=0.05, seed=3), _bf(E + 1, H, I, scale=0.05, seed=4)
    wide = _bf(T * (H + 16) + 8, seed=T)
    for stride, start in ((H, 0), (H + 8, 0), (H + 4, 0), (H + 1, 0), (H + 8, 1), (H, 3)):
        x = wide[start:].as_strided((T, H), (stride, 1))
        rows = x.clone(memory_format=torch.contiguous_format)
        want, logits = C.moe_block(rows, router, gu, dn, E, k, True), C.linear(rows, router, out_dtype=torch.float32)
        assert torch.equal(C.moe_block(x, router, gu, dn, E, k, True, logits=logits), want), (stride, start)
    C.check_errors(wide.device)


@pytest.mark.parametrize("T,E,k,H,I", [(600, 16, 4, 256, 128), (515, 8, 2, 512, 192), (3, 8, 2, 512, 128)])
@pytest.mark.parametrize("packed", [False, True])
def test_wide_expert_tiles_through_the_tensor_map(C, T, E, k, H, I, packed, monkeypatch):
    """128-row tiles whose rows come from the expert-sorted copy (the second row-fetching warp has nothing to do)."""
    x = _bf(T, H, seed=T)
    router = _bf(E + 1, H, scale=0.3, seed=34)
    wgu, wd = _bf(E + 1, 2 * I, H, scale=0.05, seed=35), _bf(E + 1, H, I, scale=0.05, seed=36)
    if packed:
        wgu, wd = C.pack_weight(wgu, gate_up=True), C.pack_weight(wd)
    want = C.moe_block(x, router, wgu, wd, E, k, True)
    monkeypatch.setattr(C, "_MOE_BT_FIXED", 128)
    assert torch.equal(C.moe_block(x, router, wgu, wd, E, k, True), want)  # rows by index
    monkeypatch.setattr(C, "GATHER_MAX_BT", 64)
    assert torch.equal(C.moe_block(x, router, wgu, wd, E, k, True), want)
    C.check_errors(x.device)


@pytest.mark.parametrize("N,K", [(256, 64), (392, 448), (2048, 4096), (1160, 128)])
@pytest.mark.parametrize("packed", [False, True])
def test_two_sm_tiles_give_the_bits_of_the_plain_tile(C, N, K, packed):
    """Fewer k-blocks than stages, a last tile without a second half or with part of one, token tiles of every width."""
    w = _bf(N, K, scale=0.05, seed=1)
    ww = C.pack_weight(w.clone()) if packed else w
    for T in (1, 31, 32, 33, 255, 257, 300, 1000, 2500):
        x = _bf(T, K + 64, seed=T)[:, 32:32 + K]
        want = C.linear(x, w, bt=16)
        assert torch.equal(C.linear(x, ww, bt=C.PAIR_FORM)[:, :N], want), T
        assert torch.equal(C.linear(x, ww)[:, :N], want), T
    C.check_errors(x.device)


@pytest.mark.parametrize("T,E,k,H,I", [(600, 16, 4, 256, 128), (1100, 32, 8, 2048, 512), (515, 8, 2, 512, 256), (3, 8, 2, 512, 128),
                                       (4103, 12, 2, 256, 384)])
def test_two_sm_expert_tiles_give_the_bits_of_the_64_row_tiles(C, T, E, k, H, I, monkeypatch):
    """Experts with none, one and several tiles, tiles of 1 to 256 rows; the shared expert has T rows."""
    x = _bf(T, H + 8, seed=T)[:, :H]
    router = _bf(E + 1, H, scale=0.3, seed=34)
    router[3] = -4.0 * x.float().mean(0).bfloat16()  # rarely picked
    wgu = C.pack_weight(_bf(E + 1, 2 * I, H, scale=0.05, seed=35), gate_up=True)
    wd = C.pack_weight(_bf(E + 1, H, I, scale=0.05, seed=36))
    monkeypatch.setattr(C, "PAIR_MIN_ROWS", 1 << 30)
    want = C.moe_block(x, router, wgu, wd, E, k, True)
    monkeypatch.setattr(C, "PAIR_MIN_ROWS", 0)
    monkeypatch.setattr(C, "moe_bt", lambda *a: 64)
    assert torch.equal(C.moe_block(x, router, wgu, wd, E, k, True), want)
    C.check_errors(x.device)


@pytest.mark.parametrize("T,E,k,H,I", [(300, 32, 8, 2048, 512), (430, 64, 8, 768, 256), (200, 16, 6, 1024, 384), (206, 16, 8, 512, 256)])
def test_two_sm_expert_tiles_of_128_rows_give_the_bits_of_the_64_row_tiles(C, T, E, k, H, I, monkeypatch):
    """50 to 107 rows per expert: eight stages that are used again, several tiles per pair of SMs, both halves of a tile."""
    assert C.PAIR_MIN_ROWS * E <= T * k < C.PAIR_256_MIN_ROWS * E
    x = _bf(T, H + 8, seed=T)[:, :H]
    router = _bf(E + 1, H, scale=0.3, seed=34)
    router[3] = -4.0 * x.float().mean(0).bfloat16()  # rarely picked
    wgu = C.pack_weight(_bf(E + 1, 2 * I, H, scale=0.05, seed=35), gate_up=True)
    wd = C.pack_weight(_bf(E + 1, H, I, scale=0.05, seed=36))
    got = C.moe_block(x, router, wgu, wd, E, k, True)
    monkeypatch.setattr(C, "PAIR_MIN_ROWS", 1 << 30)
    assert torch.equal(C.moe_block(x, router, wgu, wd, E, k, True), got)
    C.check_errors(x.device)


@pytest.mark.parametrize("T,E,k,H,I", [(600, 16, 4, 256, 128), (1100, 32, 8, 2048, 512)])
def test_wide_expert_tiles_of_packed_weights_on_one_sm(C, T, E, k, H, I, monkeypatch):
    """128-row tiles of one SM against its 64-row tiles, at sizes that otherwise take two SMs per tile."""
    monkeypatch.setattr(C, "PAIR_MIN_ROWS", 1 << 30)
    test_wide_expert_tiles_give_the_bits_of_the_64_row_tiles(C, T, E, k, H, I, True)


@pytest.mark.parametrize("T,E,k", [(465, 40, 10), (466, 40, 10), (512, 300, 12)])
def test_routing_and_plan_of_more_pairs_than_threads_keep(C, T, E, k):
    """As many pairs as the last CTA's threads keep between counting and placing, and more."""
    test_routing_and_plan_of_tied_rows(C, T, E, k)


def test_plan_of_many_pairs_by_one_cta(C, monkeypatch):
    """Routing and plan as two launches: a single CTA plans more pairs than its threads keep."""
    T, E, k, H, I = 700, 16, 8, 256, 128
    x, router = _bf(T, H, seed=T), _bf(E + 1, H, scale=0.3, seed=34)
    wgu, wd = _bf(E + 1, 2 * I, H, scale=0.05, seed=35), _bf(E + 1, H, I, scale=0.05, seed=36)
    want = C.moe_block(x, router, wgu, wd, E, k, True)
    monkeypatch.setattr(C, "ROUTE_PLAN_SPLIT", True)
    assert torch.equal(C.moe_block(x, router, wgu, wd, E, k, True), want)
    C.check_errors(x.device)


@pytest.mark.parametrize("T", [257, 1531, 1600, 3000, 4100, 6400])
def test_forms_of_few_weight_tiles_and_many_rows(C, T):
    w, x = _bf(257, 256, scale=0.05, seed=1), _bf(T, 256, seed=T)
    assert torch.equal(C.linear(x, C.pack_weight(w.clone()), out_dtype=torch.float32)[:, :257], C.linear(x, w, out_dtype=torch.float32, bt=256))
    C.check_errors(x.device)


@pytest.mark.parametrize("N,K", [(4352, 64), (4163, 256), (9000, 448)])
@pytest.mark.parametrize("packed", [False, True])
def test_two_sm_head_gives_the_logits_and_picks_of_the_plain_tile(C, N, K, packed):
    """fp32 and argmax epilogues beyond 128 rows: a last pair without a second half, ties, more than one token tile."""
    w = _bf(N, K, scale=0.05, seed=1)
    w[N // 2:N // 2 + 300] = w[:300]  # equal rows: the first one is picked
    ww = C.pack_weight(w.clone()) if packed else w
    for T in (129, 160, 255, 257, 600):
        x = _bf(T, K, seed=T)
        want = C.linear(x, w, out_dtype=torch.float32, bt=16)
        assert torch.equal(C.linear(x, ww, out_dtype=torch.float32)[:, :N], want), T
        if packed and N % 128:
            continue  # (a packed head has zero rows behind its vocabulary)
        picks, val = C.lm_head_argmax(x, ww, return_value=True)
        top = want.max(1, keepdim=True).values
        assert torch.equal(val, top[:, 0]) and torch.equal(picks, (want == top).int().argmax(1)), T
    C.check_errors(x.device)


@pytest.mark.parametrize("T", [128, 129, 300])
@pytest.mark.parametrize("I,K", [(4096, 128), (4104, 128), (8192, 192), (4160, 320)])
def test_dense_gate_up_of_many_rows_and_outputs(C, T, I, K):
    """Beyond the sizes from which other epilogues take two SMs per tile, which this one does not have."""
    x, w = _bf(T, K, seed=T), _bf(2 * I, K, scale=0.05, seed=I)
    got = C.linear_silu_mul(x, w)

    def tile(bt):
        out = torch.full((T, I), 7.0, dtype=torch.bfloat16, device="cuda")
        rc = C.lib().b200_gemm_dense(x.data_ptr(), w.data_ptr(), out.data_ptr(), T, I, K, K, K, I, C.EPI_SILU_MUL, I, bt, None, None,
                                     C.err_word(x.device).data_ptr(), 1, 0, C._stream())
        return rc, out

    rc, plain = tile(16)
    assert rc == 0 and torch.equal(got, plain)
    # the rounded halves are the unfused ops'; then silu and the product are rounded to bf16 (2^-8 each), silu from fp32
    gate, up = C.linear(x, w[:I], bt=16).double(), C.linear(x, w[I:], bt=16).double()
    ref = gate * torch.sigmoid(gate) * up
    assert ((got.double() - ref).abs() <= 2.01 * 2.0 ** -8 * ref.abs() + 1e-30).all()
    rc, out = tile(C.PAIR_FORM)
    torch.cuda.synchronize()
    assert rc == -7 and (out == 7.0).all()
    C.check_errors(x.device)


@pytest.mark.parametrize("T", [300, 600])
def test_two_sm_expert_tiles_read_the_rows_of_their_own_pass(C, T):
    """Two inputs in turn: rows of the pass before, which the same stages held, would show in either CTA's half."""
    E, k, H, I = 32, 8, 2048, 512
    wgu = C.pack_weight(_bf(E + 1, 2 * I, H, scale=0.05, seed=35), gate_up=True)
    wd = C.pack_weight(_bf(E + 1, H, I, scale=0.05, seed=36))
    router, xs = _bf(E + 1, H, scale=0.3, seed=34), (_bf(T, H, seed=1), _bf(T, H, seed=2))
    assert C.PAIR_MIN_ROWS * E <= T * k
    want = [C.moe_block(x, router, wgu, wd, E, k, True) for x in xs]
    for x, w in zip(xs, want):
        halves = torch.cat([C.moe_block(x[i:i + 100], router, wgu, wd, E, k, True) for i in range(0, T, 100)])  # one SM per tile
        assert torch.equal(w, halves)
    got = [C.moe_block(xs[i % 2], router, wgu, wd, E, k, True) for i in range(64)]
    assert all(torch.equal(g, want[i % 2]) for i, g in enumerate(got))
    C.check_errors(xs[0].device)


def test_grouped_launches_refuse_token_tiles_that_no_kernel_has(C):
    E, H, I = 2, 128, 128
    wgu, x = C.pack_weight(_bf(E, 2 * I, H, seed=1), gate_up=True), _bf(24, H, seed=2)
    out = torch.full((24, I), 7.0, dtype=torch.bfloat16, device="cuda")
    tiles = torch.tensor([[0, 0, 24, 0]], dtype=torch.int32, device="cuda")
    n = torch.ones(1, dtype=torch.int32, device="cuda")
    for bt in (24, 8, 1, 0, -1, 48):
        assert C.lib().b200_gemm_grouped(x.data_ptr(), wgu.data_ptr(), out.data_ptr(), 24, E, I, 2 * I, H, I, C.EPI_SILU_MUL, I, bt,
                                         tiles.data_ptr(), n.data_ptr(), 1, C.err_word(x.device).data_ptr(), 1, 1, None, 0,
                                         C._stream()) != 0, bt
    torch.cuda.synchronize()
    assert (out == 7.0).all()
    C.check_errors(x.device)


@pytest.mark.parametrize("N,K", [(257, 384), (1024, 1152), (2048, 1152), (2048, 896), (4096, 1408)])
def test_thin_forms_of_an_odd_number_of_stages(C, N, K):
    """K a multiple of 128 but not of 256: two k-blocks per stage."""
    w = _bf(N, K, scale=0.05, seed=1)
    packed = C.pack_weight(w.clone())
    for T in (16, 17, 48, 64, 100, 129, 200, 256):
        x = _bf(T, K + 64, seed=T)[:, 32:32 + K]
        for dt in (None, torch.float32):
            assert torch.equal(C.linear(x, packed, out_dtype=dt)[:, :N], C.linear(x, w, out_dtype=dt, bt=16)), (T, dt)
    C.check_errors(w.device)


@pytest.mark.parametrize("T", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("inter,H", [(256, 1152), (128, 384), (128, 128)])
def test_expert_block_of_a_few_rows_and_an_odd_number_of_stages(C, T, inter, H):
    """Tiles of 32 gate and 32 up rows with two k-blocks per stage."""
    test_expert_block_of_a_few_rows_with_packed_weights(C, T, inter, H)


@pytest.mark.parametrize("packed", [False, True])
@pytest.mark.parametrize("N", [4352, 9216, 16384])
def test_many_outputs_of_a_few_k_blocks(C, N, packed):
    """Either side of the number of k-blocks from which two SMs share a tile."""
    for K in (64, 320, 384, 448, 576, 640):
        w = _bf(N, K, scale=0.05, seed=1)
        weights = C.pack_weight(w.clone()) if packed else w
        for T in (17, 32, 33, 48, 49, 64, 65, 128, 129):
            x = _bf(T, K, seed=T)
            for dt in (None, torch.float32):
                assert torch.equal(C.linear(x, weights, out_dtype=dt), C.linear(x, w, out_dtype=dt, bt=16)), (K, T, dt)
    C.check_errors(w.device)
