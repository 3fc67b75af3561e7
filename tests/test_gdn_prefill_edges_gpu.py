"""The Gated-DeltaNet prefill kernels at their edges: far SiLU arguments and the rounding of the decode step."""

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


def _params(n_k, n_v, d):
    ch = 2 * n_k * d + n_v * d
    return (_bf(ch, 4, scale=0.4, seed=1), torch.zeros(n_v, device="cuda"), torch.zeros(n_v, device="cuda"),
            1.0 + _bf(d, scale=0.1, seed=2))


def _i32(v):
    return torch.tensor(v, dtype=torch.int32, device="cuda")


def _prefill(C, mixed, starts, par, n_k, n_v, d, conv_state, seg_start=None):
    """Conv output and gated-norm input and output of one pass over spans ``starts``, in slots 1, 2, ..."""
    T, ch, nseg = mixed.shape[0], 2 * n_k * d + n_v * d, len(starts) - 1
    n_chunks, chunks, per_seg, seq, st, slots = C._gdn_prefill_meta(starts, list(range(1, nseg + 1)), T, mixed.device)
    if seg_start is not None:
        st = seg_start
    rec = torch.zeros(nseg + 1, n_v, d, d, device="cuda")
    work = torch.empty(n_chunks * n_v * C.lib().b200_gdn_prefill_work_stride(d), device="cuda")
    conv_out = torch.full((T, ch), float("nan"), dtype=torch.bfloat16, device="cuda")
    o, out = (torch.empty(T, n_v * d, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    C._check(C.lib().b200_gdn_prefill(
        mixed.data_ptr(), mixed.stride(0), seq.data_ptr(), st.data_ptr(), slots.data_ptr(), conv_state.data_ptr(), rec.data_ptr(),
        par[0].data_ptr(), par[1].data_ptr(), par[2].data_ptr(), par[3].data_ptr(), conv_out.data_ptr(), chunks.data_ptr(),
        n_chunks, per_seg.data_ptr(), nseg, work.data_ptr(), o.data_ptr(), out.data_ptr(), T, n_k, n_v, d, d, 1e-6, 1,
        C.err_word(mixed.device).data_ptr(), C._stream()), "gdn_prefill")
    C.check_errors(mixed.device)
    return conv_out, o, out


def _decode_conv(C, mixed, par, n_k, n_v, d, conv_state):
    """Conv output of the decode kernels for the same rows, all in slot 1."""
    T, ch = mixed.shape[0], 2 * n_k * d + n_v * d
    conv_out = torch.empty(T, ch, dtype=torch.bfloat16, device="cuda")
    out = torch.empty(T, n_v * d, dtype=torch.bfloat16, device="cuda")
    rec, slots = torch.zeros(2, n_v, d, d, device="cuda"), _i32([1])
    C._check(C.lib().b200_gdn_decode(
        mixed.data_ptr(), mixed.stride(0), slots.data_ptr(), conv_state.data_ptr(), rec.data_ptr(), par[0].data_ptr(),
        par[1].data_ptr(), par[2].data_ptr(), par[3].data_ptr(), conv_out.data_ptr(), out.data_ptr(), None, None, 1, T, n_k, n_v,
        d, d, 4, 1e-6, C.err_word(mixed.device).data_ptr(), C._stream()), "gdn_decode")
    C.check_errors(mixed.device)
    return conv_out


@pytest.mark.parametrize("n_k,n_v,d", [(2, 4, 32), (2, 4, 64), (2, 4, 128), (16, 32, 128)])
def test_conv_of_prefill_has_the_bits_of_the_decode_step(C, n_k, n_v, d):
    par, ch = _params(n_k, n_v, d), 2 * n_k * d + n_v * d
    mixed = _bf(700, ch + n_v * d + 2 * n_v, scale=6.0, seed=3)
    state = _bf(2, ch, 3, seed=4)
    got, _, _ = _prefill(C, mixed, [0, 700], par, n_k, n_v, d, state.clone())
    assert torch.equal(got, _decode_conv(C, mixed, par, n_k, n_v, d, state.clone()))


@pytest.mark.parametrize("d", [32, 64, 128])
def test_silu_of_far_negative_arguments(C, d):
    """Between -88.7 and -87.4 the denominator of x / (1 + e^-x) is near the top of the float range and the quotient is still
    a normal number."""
    n_k, n_v, T = 2, 4, 64
    par, ch = _params(n_k, n_v, d), 2 * n_k * d + n_v * d
    par[0][:] = torch.tensor([0.0, 0.0, 0.0, 1.0])  # the conv hands its input on
    x = torch.linspace(-88.5, -87.5, T, device="cuda").bfloat16()
    mixed = _bf(T, ch + n_v * d + 2 * n_v, seed=5)
    state = torch.zeros(2, ch, 3, dtype=torch.bfloat16, device="cuda")
    silu = x.double() * torch.sigmoid(x.double())
    # __expf(88) is off by at most 105 units in the last place (below 2^-16), rounding to bf16 adds 2^-8
    tol = (2.0 ** -8 + 2.0 ** -16) * 1.01
    far = mixed.clone()
    far[:, :ch] = x[:, None]
    conv, _, _ = _prefill(C, far, [0, T], par, n_k, n_v, d, state.clone())
    assert ((conv.double() - silu[:, None]).abs() <= tol * silu.abs()[:, None]).all()
    far = mixed.clone()
    far[:, ch:ch + n_v * d] = x[:, None]  # the gate of the norm
    _, o, out = _prefill(C, far, [0, T], par, n_k, n_v, d, state.clone())
    of = o.double().view(T, n_v, d)
    normed = (of * torch.rsqrt(of.pow(2).mean(-1, keepdim=True) + 1e-6)).bfloat16().double()
    ref = par[3].double() * normed * silu[:, None, None]
    # the normed value may round to its other bf16 neighbour (2^-7); below 2^-126 a result has an absolute step of 2^-133
    assert ((out.double().view(T, n_v, d) - ref).abs() <= (2.0 ** -7 + tol) * 1.01 * ref.abs() + 2.0 ** -133).all()


@pytest.mark.parametrize("T,end", [(24, 16), (40, 3), (700, 699), (4100, 4090)])
def test_rows_behind_the_end_that_the_table_gives_their_span(C, T, end):
    """The conv of such a row still takes the rows above it: nothing is left unwritten."""
    n_k, n_v, d = 2, 4, 32
    par, ch = _params(n_k, n_v, d), 2 * n_k * d + n_v * d
    mixed, state = _bf(T, ch + n_v * d + 2 * n_v, seed=6), _bf(2, ch, 3, seed=7)
    whole, _, _ = _prefill(C, mixed, [0, T], par, n_k, n_v, d, state.clone())
    got, _, _ = _prefill(C, mixed, [0, T], par, n_k, n_v, d, state.clone(), seg_start=_i32([0, end]))
    assert torch.equal(got, whole)


@pytest.mark.parametrize("d", [32, 64, 128])
def test_norm_weights_that_start_at_any_element(C, d):
    n_k, n_v, T = 2, 4, 70
    par, ch = _params(n_k, n_v, d), 2 * n_k * d + n_v * d
    mixed, state = _bf(T, ch + n_v * d + 2 * n_v, seed=8), torch.zeros(2, ch, 3, dtype=torch.bfloat16, device="cuda")
    want = _prefill(C, mixed, [0, T], par, n_k, n_v, d, state.clone())[2]
    for off in (1, 2, 4, 8):
        flat = torch.zeros(d + 8, dtype=torch.bfloat16, device="cuda")
        flat[off:off + d] = par[3]
        assert torch.equal(_prefill(C, mixed, [0, T], (*par[:3], flat[off:off + d]), n_k, n_v, d, state.clone())[2], want)


@pytest.mark.parametrize("d", [32, 128])
def test_conv_of_large_passes_has_the_bits_of_small_ones(C, d):
    """From 4096 rows on the conv runs over 16 rows, below over 8: spans that start and end inside such a run, a last run that
    is not full, a span that leaves a state of its own rows and one that is shorter than the window."""
    n_k, n_v, lens = 2, 4, [1, 3, 17, 2, 4070, 5, 64, 9]
    par, ch = _params(n_k, n_v, d), 2 * n_k * d + n_v * d
    starts = [sum(lens[:i]) for i in range(len(lens) + 1)]
    T = starts[-1]
    assert T > 4096 and T % 16
    mixed, state = _bf(T, ch + n_v * d + 2 * n_v, seed=9), _bf(len(lens) + 1, ch, 3, seed=10)
    whole_state = state.clone()
    whole, _, _ = _prefill(C, mixed, starts, par, n_k, n_v, d, whole_state)
    for i, (a, b) in enumerate(zip(starts, starts[1:])):
        own = torch.stack([state[0], state[1 + i]])
        part, _, _ = _prefill(C, mixed[a:b].clone(), [0, b - a], par, n_k, n_v, d, own)
        assert torch.equal(whole[a:b], part), i
        assert torch.equal(whole_state[1 + i], own[1]), i
