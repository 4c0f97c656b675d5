"""The row kernels that take 16 bytes of several tokens per thread: the convolutions of four taps in tiles of tokens and the sum over a
token's experts.  Against the kernels that take an element at a time (which a view one entry off the 16-byte boundary still
reaches): the same sums in the same order, so the same bits; those are compared with float64 elsewhere, and here once: a convolution is
four products, 1e-6 of the norm in float32 and 2^-9 for a result rounded to bfloat16."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
LENS = [1, 2, 3, 4, 5, 1201, 7, 8, 9, 30, 1, 400, 3]  # portions that start anywhere in a tile, end in one, fill none
LONG = [1, 2, 3, 4, 5, 3201, 7, 8, 9, 30, 1, 2800, 3]  # the same, long enough for tiles at 2,056 bfloat16 channels


def portions(dtype, C, pad, seed, lens=LENS):
    """Rows of a step with `pad` padded lanes behind them, on a 16-byte boundary and one entry off it, with kept inputs."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    n, T = len(lens), sum(lens) + pad
    wide = torch.randn(T, C + 16, generator=g, device=DEV).to(dtype)
    off = torch.empty(T, C + 16, device=DEV, dtype=dtype)
    off[:, 1:1 + C] = wide[:, :C]
    cu = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), dtype=torch.int32, device=DEV)
    seq = torch.repeat_interleave(torch.arange(n, device=DEV), torch.tensor(lens, device=DEV)).int()
    seq = torch.cat([seq, torch.full((pad,), -1, device=DEV, dtype=torch.int32)])
    state = torch.randn(n + 2, 3 * C, generator=g, device=DEV)
    slots = torch.randperm(n + 2, generator=g, device=DEV)[:n].int()
    return g, wide[:, :C], off[:, 1:1 + C], cu, seq, state, slots


@pytest.mark.parametrize("in_dtype,out_dtype", [(torch.float32, torch.float32), (torch.bfloat16, torch.float32), (torch.bfloat16, torch.bfloat16)])
@pytest.mark.parametrize("C,pad,add_input,biased", [(8, 3, True, False), (1032, 0, False, True), (2048, 5, False, True)])
def test_causal_convolution(C, pad, add_input, biased, in_dtype, out_dtype):
    from tokensprint_b200 import ops

    g, x, x_off, cu, seq, state, slots = portions(in_dtype, C, pad, C + pad)
    taps = torch.randn(4, C, generator=g, device=DEV)
    bias, in_bias = (torch.randn(2, C, generator=g, device=DEV).unbind(0) if biased else (None, None))
    bias, in_bias = (None, None) if bias is None else (bias.contiguous(), in_bias.contiguous())
    got = []
    for rows in (x, x_off):
        out, kept = torch.full((x.shape[0], C), float("nan"), device=DEV, dtype=out_dtype), state.clone()
        ops.causal_conv(rows, taps, bias, kept, slots, cu, seq, len(LENS), out, activation=None if add_input else "silu", add_input=add_input, in_bias=in_bias)
        got.append((out, kept))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
    b = LENS.index(1201)  # and one portion in float64
    a = int(cu[b])
    h = torch.cat([state[slots[b]].view(3, C).double(), x[a:a + 1201].double() + (in_bias.double() if biased else 0.0)])
    want = sum(h[j:j + 1201] * taps[j].double() for j in range(4)) + (bias.double() if biased else 0.0)
    want = want + h[3:] if add_input else want * torch.sigmoid(want)
    err = float((got[0][0][a:a + 1201].double() - want).norm() / want.norm())
    assert err < (1e-6 if out_dtype == torch.float32 else 2 ** -8)


@pytest.mark.parametrize("in_dtype,out_dtype", [(torch.float32, torch.float32), (torch.bfloat16, torch.float32), (torch.bfloat16, torch.bfloat16)])
@pytest.mark.parametrize("pad,add_input,biased", [(3, True, False), (0, False, True)])
def test_causal_convolution_in_tiles(pad, add_input, biased, in_dtype, out_dtype):
    from tokensprint_b200 import ops

    C = 2056  # the last block of columns nearly empty
    g, x, x_off, cu, seq, state, slots = portions(in_dtype, C, pad, 7 + pad, LONG)
    narrow = in_dtype == torch.bfloat16
    assert ops._fn("ts_causal_conv_tile_tokens")(1 if narrow else 0, x.shape[0], len(LONG), C) == (8 if narrow else 4)
    taps = torch.randn(4, C, generator=g, device=DEV)
    bias, in_bias = torch.randn(2, C, generator=g, device=DEV).unbind(0) if biased else (None, None)
    got = []
    for rows in (x, x_off):
        out, kept = torch.full((x.shape[0], C), float("nan"), device=DEV, dtype=out_dtype), state.clone()
        ops.causal_conv(rows, taps, bias, kept, slots, cu, seq, len(LONG), out, activation=None if add_input else "silu", add_input=add_input, in_bias=in_bias)
        got.append((out, kept))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])


@pytest.mark.parametrize("T,n,C,narrow", [(128, 128, 10240, True), (512, 512, 10240, True), (512, 512, 10240, False), (320, 320, 4096, True),
                                          (1424, 26, 4096, True), (2304, 257, 8192, True), (1024, 128, 10240, True), (512, 128, 10240, False),
                                          (2048, 1, 8, True), (576, 65, 4096, False), (64, 64, 10240, False)])
def test_steps_of_many_portions_take_no_tiles_of_tokens(T, n, C, narrow):
    """Decode batches, and prompts beside so many requests that a tile's chain of single tokens would be the step."""
    from tokensprint_b200 import ops

    assert ops._fn("ts_causal_conv_tile_tokens")(1 if narrow else 0, T, n, C) == 1


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("C,H,pad", [(8, 1, 4), (1288, 130, 0)])
def test_state_space_convolution(C, H, pad, dtype):
    from tokensprint_b200 import ops

    g, x, x_off, cu, seq, state, slots = portions(dtype, C, pad, C + H)
    taps, bias = torch.randn(C, 4, generator=g, device=DEV), torch.randn(C, generator=g, device=DEV)
    dt_raw = torch.randn(x.shape[0], H, generator=g, device=DEV)
    dt_bias, a_log = torch.randn(2, H, generator=g, device=DEV).unbind(0)
    got = []
    for rows in (x, x_off):
        kept = state.clone()
        got.append((*ops.ssm_conv(rows, taps, bias, kept, slots, cu, seq, len(LENS), dt_raw, dt_bias.contiguous(), a_log.contiguous()), kept))
    for a, b in zip(*got):
        assert torch.equal(a, b)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,pad", [(1, 4), (130, 0)])
def test_state_space_convolution_in_tiles(dtype, H, pad):
    from tokensprint_b200 import ops

    C = 2056
    g, x, x_off, cu, seq, state, slots = portions(dtype, C, pad, C + H)
    assert ops._fn("ts_ssm_conv_in_tiles")(x.shape[0], len(LENS), C)
    taps, bias = torch.randn(C, 4, generator=g, device=DEV), torch.randn(C, generator=g, device=DEV)
    dt_raw = torch.randn(x.shape[0], H, generator=g, device=DEV)
    dt_bias, a_log = torch.randn(2, H, generator=g, device=DEV).unbind(0)
    got = []
    for rows in (x, x_off):
        kept = state.clone()
        got.append((*ops.ssm_conv(rows, taps, bias, kept, slots, cu, seq, len(LENS), dt_raw, dt_bias.contiguous(), a_log.contiguous()), kept))
    for a, b in zip(*got):
        assert torch.equal(a, b)


@pytest.mark.parametrize("T,n,C", [(128, 128, 4352), (256, 256, 8448), (512, 512, 4352), (512, 128, 2304), (768, 64, 2304), (2048, 1, 256), (1424, 26, 256)])
def test_small_steps_of_the_state_space_convolution_take_no_tiles(T, n, C):
    from tokensprint_b200 import ops

    assert not ops._fn("ts_ssm_conv_in_tiles")(T, n, C)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("T,N,top,shared,identity", [(1, 8, 1, False, False), (5, 2048, 4, True, True), (700, 1032, 2, False, True), (3, 1000, 7, True, False)])
def test_sum_over_experts(T, N, top, shared, identity, dtype):
    from tokensprint_b200 import ops

    g = torch.Generator(device=DEV).manual_seed(T + N)
    normal = lambda *s: torch.randn(*s, generator=g, device=DEV).to(dtype)  # noqa: E731
    pairs, x, sh = normal(T * top, N), normal(T, N), normal(T, N) if shared else None
    weight = torch.rand(T * top, generator=g, device=DEV)
    ids = torch.randint(0, 6, (T, top), generator=g, device=DEV, dtype=torch.int32) if identity else None
    out = torch.full((T, N), float("nan"), device=DEV, dtype=dtype)
    ops.moe_combine(pairs, sh, out, top, weight, ids=ids, num_experts=4, x=x if identity else None)
    v = pairs.double().view(T, top, N)
    if identity:
        v = torch.where((ids >= 4)[:, :, None], x.double()[:, None, :], v)
    want = (v * weight.double().view(T, top, 1)).sum(1) + (sh.double() if shared else 0.0)
    assert float((out.double() - want).norm() / want.norm()) < (1e-6 if dtype == torch.float32 else 2 ** -8)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("T,N,top,shared,identity", [(800, 256, 8, True, False), (200, 1032, 3, False, True), (33, 7168, 1, True, True), (66000, 256, 2, False, False)])
def test_sum_over_experts_in_pieces(T, N, top, shared, identity, dtype):
    """16 bytes a thread against an element a thread (rows off the 16-byte boundary, 66,000 tokens): the same bits."""
    from tokensprint_b200 import ops

    assert ops._fn("ts_moe_combine_in_pieces")(T, N)
    g = torch.Generator(device=DEV).manual_seed(T + N)

    def rows(n):  # the same values on a 16-byte boundary and one entry off it
        v = torch.randn(n, N, generator=g, device=DEV).to(dtype)
        off = torch.empty(n * N + 1, device=DEV, dtype=dtype)[1:].view(n, N)
        return v, off.copy_(v)

    pairs, x, sh = rows(T * top), rows(T), rows(T)
    weight = torch.rand(T * top, generator=g, device=DEV)
    ids = torch.randint(0, 6, (T, top), generator=g, device=DEV, dtype=torch.int32) if identity else None
    got = []
    for k in range(2):
        out = torch.full((T * N + 1,), float("nan"), device=DEV, dtype=dtype)[k : k + T * N].view(T, N)
        ops.moe_combine(pairs[k], sh[k] if shared else None, out, top, weight, ids=ids, num_experts=4, x=x[k] if identity else None)
        got.append(out)
    assert torch.equal(*got)


@pytest.mark.parametrize("T,N", [(1, 2048), (5, 2048), (64, 2048), (200, 512), (8192, 64), (40000, 128), (2048, 248)])
def test_small_sums_over_experts_take_an_element_a_thread(T, N):
    from tokensprint_b200 import ops

    assert not ops._fn("ts_moe_combine_in_pieces")(T, N)
