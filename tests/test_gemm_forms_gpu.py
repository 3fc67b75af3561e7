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
