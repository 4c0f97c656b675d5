"""The few-row products that read their weights straight into their warps' rings (csrc/gemm_rows.cu): ragged N, fewer tasks than CTAs
and many more, warps with unequal shares of K, M at the edges of the halves of eight, the longest K.  Against float64;
tolerances: float32 sums of up to 12,288 products of standard normal x 0.05 stay below 1e-6 of the result's norm (1e-5
asserted), one rounding to bfloat16 is 2^-9 (1e-2)."""

import math

import pytest
import torch

from tests.plain import qwen3_plain as plain

pytestmark = pytest.mark.gpu
DEV = "cuda"
SHAPES = [(1, 137, 1024), (8, 1000, 1088), (16, 4096, 1024), (9, 8200, 1984), (2, 4104, 4096), (2, 520, 12288), (16, 2056, 2048), (5, 8200, 5632),
          (8, 100, 4096), (3, 24576, 1024)]  # M, N, K


def rel(a, b):
    return float((a.double().cpu() - b.double().cpu()).norm() / b.double().norm().cpu())


def make(M, N, K):
    g = torch.Generator(device=DEV).manual_seed(M + 3 * N + K)
    normal = lambda *s: torch.randn(*s, generator=g, device=DEV)  # noqa: E731
    return normal, normal(M, K).bfloat16(), (normal(N, K) * 0.05).bfloat16()


@pytest.mark.parametrize("M,N,K", SHAPES)
def test_plain_and_residual_epilogues(M, N, K):
    from tokensprint_b200 import ops

    normal, x, w = make(M, N, K)
    assert ops._rows_takes(M, ops._facts(w)) > 0, "the shape does not reach this kernel"
    want = x.double() @ w.double().T
    for dtype, tol in ((torch.float32, 1e-5), (torch.bfloat16, 1e-2)):
        out = torch.full((M, N), float("nan"), device=DEV, dtype=dtype)
        ops.gemm_skinny_bf16(x, w, out, direct=True)
        again = torch.empty_like(out)
        ops.gemm_skinny_bf16(x, w, again, prefetch=w, direct=True)
        assert rel(out, want) < tol and torch.equal(out, again)
    hidden0, norm_w = normal(M, N), 1 + 0.1 * normal(N)
    hidden, xprime = hidden0.clone(), torch.full((M, N), float("nan"), device=DEV, dtype=torch.bfloat16)
    ssq = torch.full((ops.gemm_ssq_tiles(M, w), M), float("nan"), device=DEV)
    ops.gemm_skinny_fused(x, w, mode=ops.GEMM_EPILOGUE_RESIDUAL_NORM, hidden=hidden, norm_weight=norm_w, xprime=xprime, ssq_out=ssq,
                          branch_scale=0.7, direct=True)
    want_h = hidden0.double() + 0.7 * want
    assert rel(hidden, want_h) < 1e-5 and rel(xprime, want_h * norm_w.double()) < 1e-2 and rel(ssq.sum(0), (want_h**2).sum(1)) < 1e-5
    # and a product that takes the row sums as its scale
    w2, x2 = (normal(136, 1024) * 0.05).bfloat16(), normal(M, 1024).bfloat16()
    out = torch.empty((M, 136), device=DEV, dtype=torch.float32)
    ops.gemm_skinny_fused(x2, w2, out=out, scale_ssq=ssq, scale_width=N, scale_eps=1e-5, direct=True)
    assert rel(out, (x2.double() @ w2.double().T) * torch.rsqrt(ssq.double().sum(0) / N + 1e-5)[:, None]) < 1e-5


@pytest.mark.parametrize("activation", ["silu", "gelu_tanh"])
@pytest.mark.parametrize("M,I,K", [(1, 64, 1024), (16, 3072, 1024), (2, 5632, 2048), (8, 1088, 4096), (4, 320, 6144)])
def test_gated_epilogue(M, I, K, activation):
    from tokensprint_b200 import ops

    normal, x, gate = make(M, I, K)
    up = (normal(I, K) * 0.05).bfloat16()
    stacked = torch.stack([gate.view(I // 64, 64, K), up.view(I // 64, 64, K)], dim=1).reshape(2 * I, K).contiguous()
    assert ops._rows_takes(M, ops._facts(stacked)) > 0
    ssq = torch.rand(37, M, device=DEV) + 0.1
    out = torch.full((M, I), float("nan"), device=DEV, dtype=torch.bfloat16)
    ops.gemm_skinny_fused(x, stacked, out=out, mode=ops.GEMM_EPILOGUE_SWIGLU, scale_ssq=ssq, scale_width=K, scale_eps=1e-6, activation=activation,
                          direct=True)
    r = torch.rsqrt(ssq.double().sum(0) / K + 1e-6)[:, None]
    a, b = (x.double() @ gate.double().T) * r, (x.double() @ up.double().T) * r
    act = torch.nn.functional.silu(a) if activation == "silu" else torch.nn.functional.gelu(a, approximate="tanh")
    assert rel(out, act * b) < 1e-2


@pytest.mark.parametrize("M,nq,nkv,K,rope,norm", [(1, 16, 8, 1024, True, True), (16, 16, 8, 1024, True, False), (5, 16, 4, 2048, False, True),
                                                  (2, 8, 8, 2048, True, True), (4, 32, 8, 4096, True, True), (3, 32, 4, 4096, True, False),
                                                  (1, 30, 5, 1088, True, True), (9, 16, 8, 1024, True, True), (15, 16, 8, 1024, True, True),
                                                  (11, 32, 8, 1024, True, False), (13, 18, 8, 1024, False, True)])
def test_heads_with_norm_rotation_and_store(M, nq, nkv, K, rope, norm):
    from tokensprint_b200 import ops

    d = 128
    normal, x, w = make(M, (nq + 2 * nkv) * d, K)
    assert ops._rows_takes(M, ops._facts(w), nq + 2 * nkv) > 0
    qw, kw = (1 + 0.2 * normal(d), 1 + 0.2 * normal(d)) if norm else (None, None)
    inv_freq = (1.0 / (1e4 ** (torch.arange(0, d, 2).float() / d))).to(DEV) if rope else None
    positions = torch.randint(0, 3000, (M,)).to(DEV, torch.int32)
    slots = torch.randperm(M + 7)[:M].to(DEV, torch.int32)
    if M > 1:
        slots[M // 2] = -1  # a row whose key and value are not stored
    ssq = torch.rand(300, M, device=DEV) + 0.1
    heads = ((x.double() @ w.double().T) * torch.rsqrt(ssq.double().sum(0) / K + 1e-6)[:, None]).cpu().view(M, nq + 2 * nkv, d)
    qh, kh, vh = heads[:, :nq], heads[:, nq:nq + nkv], heads[:, nq + nkv:]
    if norm:
        qh, kh = plain.rms_norm(qh, qw.double().cpu(), 1e-5), plain.rms_norm(kh, kw.double().cpu(), 1e-5)
    if rope:
        ang = plain.rope_angles(positions.tolist(), d, 1e4)
        qh, kh = plain.apply_rope(qh, ang), plain.apply_rope(kh, ang)
    for table in ([None, ops.rope_cos_sin(positions, inv_freq, M)] if rope else [None]):
        q = torch.full((M, nq * d), float("nan"), device=DEV, dtype=torch.bfloat16)
        kc, vc = (torch.full((M + 7, nkv, d), 7.0, device=DEV, dtype=torch.bfloat16) for _ in range(2))
        ops.gemm_qk_rope_store(x, w, q, kc, vc, slots, positions, qw, kw, 1e-5, inv_freq, nq, nkv, scale_ssq=ssq, scale_width=K, scale_eps=1e-6,
                               cos_sin=table, direct=True)
        assert rel(q.view(M, nq, d), qh) < 1e-2
        used = {s for s in slots.tolist() if s >= 0}
        for m, s in enumerate(slots.tolist()):
            if s >= 0:
                assert rel(kc[s], kh[m]) < 1e-2 and rel(vc[s], vh[m]) < 1e-2
        for s in set(range(M + 7)) - used:
            assert bool((kc[s] == 7.0).all()) and bool((vc[s] == 7.0).all()), "a slot nobody owns was written"


@pytest.mark.parametrize("M,heads,K,warps", [(1, 32, 1024, 16), (2, 33, 2048, 16), (4, 32, 1024, 8), (15, 32, 1024, 8), (11, 48, 1024, 8), (16, 32, 1024, 16),
                                             (1, 34, 4096, 8), (4, 56, 5120, 8), (4, 66, 5120, 8), (1, 67, 1024, 0), (4, 80, 5120, 0), (8, 48, 4096, 0)])
def test_heads_are_taken_only_where_their_clusters_stand_at_once(M, heads, K, warps):
    """33 clusters of four CTAs of 16 warps, 66 of 8 warps (two CTAs an SM)."""
    from tokensprint_b200 import ops

    assert ops._fn("ts_gemm_rows_takes_heads")(M, heads, K) == warps


@pytest.mark.parametrize("M,N,K,taken", [(8, 151936, 1024, True), (9, 151936, 1024, False), (16, 24576, 1024, False), (16, 6144, 1024, True),
                                         (16, 9472, 1024, True), (9, 9473, 1536, False), (16, 32768, 2048, True), (8, 24576, 4096, True),
                                         (9, 24576, 4096, False)])
def test_many_short_tasks_of_more_than_eight_rows_stay_with_the_other_kernel(M, N, K, taken):
    from tokensprint_b200 import ops

    assert (ops._fn("ts_gemm_rows_ssq_tiles")(M, N, K) > 0) == taken


@pytest.mark.parametrize("nq,nkv,K", [(16, 8, 1024), (8, 4, 1088), (4, 2, 1984)])
def test_a_head_has_the_same_bits_whatever_the_rows_beside_it(nq, nkv, K):
    """Steps of 1 to 16 rows share a head among 16 or among 8 warps a CTA: the same sums in the same order."""
    from tokensprint_b200 import ops

    d, most = 128, 16
    normal, x, w = make(most, (nq + 2 * nkv) * d, K)
    forms = {ops._fn("ts_gemm_rows_takes_heads")(M, nq + 2 * nkv, K) for M in range(1, most + 1)}
    assert forms == {8, 16}
    qw, kw = 1 + 0.2 * normal(d), 1 + 0.2 * normal(d)
    inv_freq = (1.0 / (1e4 ** (torch.arange(0, d, 2).float() / d))).to(DEV)
    positions = torch.randint(0, 3000, (most,)).to(DEV, torch.int32)
    slots = torch.randperm(most).to(DEV, torch.int32)
    ssq = torch.rand(64, most, device=DEV) + 0.1

    def run(first, last):
        q = torch.full((last - first, nq * d), float("nan"), device=DEV, dtype=torch.bfloat16)
        kc, vc = (torch.full((most, nkv, d), 7.0, device=DEV, dtype=torch.bfloat16) for _ in range(2))
        ops.gemm_qk_rope_store(x[first:last].contiguous(), w, q, kc, vc, slots[first:last].contiguous(), positions[first:last].contiguous(), qw, kw, 1e-5,
                               inv_freq, nq, nkv, scale_ssq=ssq[:, first:last].contiguous(), scale_width=K, scale_eps=1e-6, direct=True)
        at = slots[first:last].long()
        return q, kc[at], vc[at]

    whole = run(0, most)
    for first, last in ((0, 1), (15, 16), (3, 5), (0, 3), (7, 15), (1, 16), (0, 9), (4, 12)):
        for a, b in zip(run(first, last), whole):
            assert torch.equal(a, b[first:last])


@pytest.mark.parametrize("N,K", [(1000, 1024), (2056, 1984), (4104, 2048)])
def test_a_row_has_the_same_bits_whatever_the_rows_beside_it(N, K):
    """Plain, gated and residual products sum over 16 warps at every number of rows."""
    from tokensprint_b200 import ops

    normal, x, w = make(16, N, K)
    gate_up = (normal(256, K) * 0.05).bfloat16()
    hidden0, norm_w = normal(16, N), 1 + 0.1 * normal(N)

    def run(first, last):
        M, rows = last - first, x[first:last].contiguous()
        assert ops._rows_takes(M, ops._facts(w)) > 0 and ops._rows_takes(M, ops._facts(gate_up)) > 0
        plain = torch.empty(M, N, device=DEV)
        ops.gemm_skinny_bf16(rows, w, plain, direct=True)
        gated = torch.empty(M, 128, device=DEV, dtype=torch.bfloat16)
        ops.gemm_skinny_fused(rows, gate_up, out=gated, mode=ops.GEMM_EPILOGUE_SWIGLU, direct=True)
        hidden, xprime = hidden0[first:last].clone(), torch.empty(M, N, device=DEV, dtype=torch.bfloat16)
        ssq = torch.empty(ops.gemm_ssq_tiles(M, w), M, device=DEV)
        ops.gemm_skinny_fused(rows, w, mode=ops.GEMM_EPILOGUE_RESIDUAL_NORM, hidden=hidden, norm_weight=norm_w, xprime=xprime, ssq_out=ssq, direct=True)
        return plain, gated, hidden, xprime, ssq.T

    whole = run(0, 16)
    for first, last in ((0, 1), (15, 16), (3, 5), (0, 8), (0, 9), (5, 14)):
        for a, b in zip(run(first, last), whole):
            assert torch.equal(a, b[first:last])


@pytest.mark.parametrize("M", [1, 5, 17])
@pytest.mark.parametrize("off", ["table", "q", "k"])
def test_buffers_off_their_boundaries_are_refused(off, M):
    """A table of cosines and sines, query rows or a cache that do not start where the kernels read and write them: refused on the host,
    whichever kernel takes the step."""
    from tokensprint_b200 import ops

    nq, nkv, K, d = 16, 8, 1024, 128
    _, x, w = make(M, (nq + 2 * nkv) * d, K)
    inv_freq = (1.0 / (1e4 ** (torch.arange(0, d, 2).float() / d))).to(DEV)
    positions, slots = (torch.arange(M, device=DEV, dtype=torch.int32) for _ in range(2))
    rows = lambda shape, shift: torch.zeros(math.prod(shape) + 1, device=DEV, dtype=torch.bfloat16)[int(shift):][:math.prod(shape)].view(shape)
    table = ops.rope_cos_sin(positions, inv_freq, M).flatten()
    if off == "table":
        table = torch.cat([table[:1], table])[1:]
    q, kc, vc = rows((M, nq * d), off == "q"), rows((M, nkv, d), off == "k"), rows((M, nkv, d), False)
    with pytest.raises(ops.KernelError):
        ops.gemm_qk_rope_store(x, w, q, kc, vc, slots, positions, None, None, 1e-5, inv_freq, nq, nkv, cos_sin=table, direct=True)


def test_what_it_does_not_take_runs_on_the_other_kernel():
    """17 rows, rows that are not whole chunks, short rows, rows that do not start on 32 bytes, an input that leaves no room for
    the rings: the same call, the tcgen05 kernel's bits."""
    from tokensprint_b200 import ops

    for M, N, K, ld in ((17, 256, 1024, 1024), (4, 256, 1000, 1000), (4, 256, 960, 960), (4, 256, 1024, 1032), (8, 256, 12288, 12288)):
        _, x, w = make(M, N, ld)
        w, x = w[:, :K], x[:, :K].contiguous()
        a, b = (torch.empty((M, N), device=DEV, dtype=torch.float32) for _ in range(2))
        ops.gemm_skinny_bf16(x, w, a, direct=True)
        ops.gemm_skinny_bf16(x, w, b)
        assert torch.equal(a, b)
