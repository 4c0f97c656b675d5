"""Fegetar's mechanisms one by one on the GPU, each against the plain implementation (or a few
float64 lines in the test), with inputs made so that a fault shows: a far key that one score
singles out, keys on both sides of a page's edge and of a window's edge, the key just behind a
query, the first tokens, state that crosses a portion's edge and slots that are used again."""

import math

import pytest
import torch

from tests.fegetar_configs import FEG, fegetar_weights
from tests.plain import fegetar_plain as plain

pytestmark = pytest.mark.gpu

DTYPES = [torch.float32, torch.bfloat16]
TOL = {torch.float32: 2e-5, torch.bfloat16: 2e-2}


def _dev(x, dtype=None):
    return x.to("cuda", dtype) if dtype is not None else x.to("cuda")


def _i32(values):
    return torch.tensor(list(values), dtype=torch.int32, device="cuda")


def _rel(got, want):
    return float((got.double().cpu() - want.double().cpu()).abs().max() / want.double().abs().max().clamp_min(1e-30))


# ---------------------------------------------------------------------------
# embedding: the pair table and the token kept between portions


def test_pair_hash_embedding_over_portions_and_reused_slots():
    from tokensprint_b200 import ops

    V, W, buckets, mp, mc = 50, 24, 13, 7, 3
    g = torch.Generator().manual_seed(0)
    embed, table = torch.randn(V, W, generator=g), torch.randn(buckets + 1, W, generator=g)
    weights = {"embed": embed, "bigram": table}
    cfg = {"embedding": {"bigram": {"buckets": buckets, "mul_prev": mp, "mul_cur": mc}}}
    seqs = {0: torch.randint(0, V, (11,), generator=g).tolist(), 1: torch.randint(0, V, (7,), generator=g).tolist(),
            2: torch.randint(0, V, (5,), generator=g).tolist()}
    want = {k: plain.embed(v, weights, cfg) for k, v in seqs.items()}
    last = torch.full((2,), 77, dtype=torch.int32, device="cuda")  # two slots; stale content must not matter
    # steps: (sequence, first, count, slot); sequence 2 takes over slot 0 after sequence 0 has ended
    steps = [[(0, 0, 4, 0), (1, 0, 1, 1)], [(1, 1, 2, 1), (0, 4, 1, 0)], [(0, 5, 6, 0), (1, 3, 4, 1)], [(2, 0, 2, 0)], [(2, 2, 3, 0)]]
    for step in steps:
        ids, pos, sidx, cu, slots = [], [], [], [0], []
        for b, (s, first, count, slot) in enumerate(step):
            ids += seqs[s][first : first + count]
            pos += list(range(first, first + count))
            sidx += [b] * count
            cu.append(len(ids))
            slots.append(slot)
        ids_d = _i32(ids)
        hidden = torch.empty((len(ids), W), device="cuda", dtype=torch.float32)
        ops.embed_gather(hidden, _dev(embed), ids_d)
        ops.pair_hash_embed(hidden, _dev(table), ids_d, _i32(pos), _i32(sidx), _i32(cu), _i32(slots), last, buckets, mp, mc, V)
        row = 0
        for s, first, count, _ in step:
            assert torch.allclose(hidden[row : row + count].cpu().double(), want[s][first : first + count], atol=1e-6), (s, first)
            row += count


def test_pair_hash_embedding_takes_large_multipliers():
    from tokensprint_b200 import ops

    V, W, buckets, mp, mc = 200000, 8, 99991, 2147483629, 2147483587
    table = torch.arange(buckets + 1, dtype=torch.float32)[:, None].repeat(1, W)
    ids = [199999, 123456, 7]
    hidden = torch.zeros((3, W), device="cuda")
    ops.pair_hash_embed(hidden, _dev(table), _i32(ids), _i32([0, 1, 2]), _i32([0, 0, 0]), _i32([0, 3]), _i32([0]),
                        torch.zeros(1, dtype=torch.int32, device="cuda"), buckets, mp, mc, V)
    assert hidden[:, 0].tolist() == [float(r) for r in plain.pair_rows(ids, mp, mc, buckets)]


# ---------------------------------------------------------------------------
# norms and small element-wise kernels


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("width", [70, 72, 256, 1000, 4100])
def test_norm_on_the_branch(dtype, width):
    from tokensprint_b200 import ops

    g = torch.Generator().manual_seed(width)
    hidden, branch, w = torch.randn(5, width, generator=g), torch.randn(5, width, generator=g) * 3, torch.randn(width, generator=g) * 0.1
    branch = branch.to(dtype)
    want = hidden.double() + plain.norm_around_zero(branch.double(), w.double(), 1e-5)
    h, rounded = _dev(hidden.clone()), torch.empty((5, width), device="cuda", dtype=dtype)
    ops.rmsnorm_add(_dev(branch), _dev(1.0 + w), h, 1e-5, rounded)
    assert _rel(h, want) < 1e-6
    assert torch.equal(rounded, h.to(dtype))


@pytest.mark.parametrize("dtype", DTYPES)
def test_activations(dtype):
    from tokensprint_b200 import ops

    g = torch.Generator().manual_seed(3)
    x = (torch.randn(7, 50, generator=g) * 3).to(dtype)
    out = torch.empty_like(x, device="cuda")
    ops.gelu_tanh(_dev(x), out)
    assert _rel(out, plain.gelu_tanh(x.double())) < TOL[dtype]
    gu = (torch.randn(7, 2 * 30, generator=g) * 3).to(dtype)
    act = torch.empty((7, 30), device="cuda", dtype=dtype)
    ops.capped_glu(_dev(gu), act, 1.5, 1.702)
    a, b = gu[:, :30].double().clamp(max=1.5), gu[:, 30:].double().clamp(-1.5, 1.5)
    assert _rel(act, a * torch.sigmoid(1.702 * a) * (b + 1)) < TOL[dtype]
    table, ids = torch.randn(9, 40, generator=g).to(dtype), [8, 0, 3, 3, 5, 1, 2]
    y = _dev(x[:, :12].contiguous())
    ops.gelu_gate_rows(y, _dev(table), _i32(ids), 24)
    assert _rel(y, plain.gelu_tanh(x[:, :12].double()) * table[ids][:, 24:36].double()) < TOL[dtype]


# ---------------------------------------------------------------------------
# latent attention: the kernels on made-up rows


def _paged(rows: torch.Tensor, page: int, dtype, seed: int, spare: int = 3):
    """Puts a sequence's cache rows [N, D] into pages in a shuffled order; returns pool and table."""
    N, D = rows.shape
    n_pages = -(-N // page)
    g = torch.Generator().manual_seed(seed)
    order = torch.randperm(n_pages + spare, generator=g)[:n_pages]
    pool = torch.full(((n_pages + spare), page, D), float("nan"), dtype=dtype)
    for j in range(N):
        pool[order[j // page], j % page] = rows[j].to(dtype)
    return pool, order.tolist()


def _attention_reference(q, rows, positions, rank, scale, window, gates):
    out = torch.zeros(q.shape[0], q.shape[1], rank, dtype=torch.float64)
    for t, p in enumerate(positions):
        lo = max(0, p - window + 1) if window else 0
        K = rows[lo : p + 1].double()
        w = torch.softmax(q[t].double() @ K.T * scale, -1)
        out[t] = (w @ K[:, :rank]) * gates[t].double()[:, None]
    return out


ATTENTION_CASES = [
    # rank, rot, heads, page, context, queries (the step's tokens are the last `queries` positions), window
    (40, 16, 3, 16, 700, 1, 0),
    (40, 16, 3, 16, 700, 5, 0),
    (18, 6, 1, 8, 130, 33, 0),
    (32, 16, 8, 16, 257, 64, 0),
    (64, 32, 4, 16, 300, 2, 0),
    (40, 16, 3, 16, 200, 7, 37),
    (26, 10, 5, 32, 96, 96, 0),
    (48, 16, 6, 16, 333, 40, 0),
    (128, 32, 16, 32, 520, 3, 0),
    (64, 16, 2, 64, 400, 1, 100),
    (512, 64, 4, 16, 200, 9, 0),
]


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("rank, rot, H, page, N, Q, window", ATTENTION_CASES)
def test_latent_attention_finds_the_one_key(dtype, rank, rot, H, page, N, Q, window):
    """All rows are small noise except one whose score stands out for one (query, head): the output
    there must be that row's latent.  The one key sits far away, on both sides of page edges, among
    the first tokens, at the query's own place, just behind the query (not to be seen), and on
    both sides of the window's edge."""
    from tokensprint_b200 import ops

    D = rank + rot
    g = torch.Generator().manual_seed(N + Q)
    first = N - Q
    positions = list(range(first, N))
    special = sorted({0, 1, page - 1, page, page + 1, 2 * page - 1, N // 2, first - 1, first, N - 2, N - 1} & set(range(N)))
    if window:
        special = sorted(set(special) | {max(0, N - 1 - window), max(0, N - window), max(0, N - window + 1)})
    for j_star in special:
        rows = torch.randn(N, D, generator=g) * 0.05
        u = torch.randn(D, generator=g)
        u = u / u.norm()
        rows[j_star] = 6.0 * u + rows[j_star] * 0.1
        rows[j_star, :rank] += torch.linspace(-1, 1, rank)  # a latent that is easy to tell from noise
        q = torch.randn(Q, H, D, generator=g) * 0.05
        t_star, a_star = Q - 1, H - 1
        q[t_star, a_star] = 6.0 * u
        if Q > 1 and first <= j_star < N - 1:
            q[j_star - first, 0] = 6.0 * u  # the query at the key's own place sees it; the one before must not
            if j_star - first >= 1:
                q[j_star - first - 1, 0] = 6.0 * u
        gates = torch.rand(Q, H, generator=g) * 0.5 + 0.5
        q, rows = q.to(dtype).float(), rows.to(dtype).float()
        want = _attention_reference(q, rows, positions, rank, 1.0, window, gates)
        pool, table = _paged(rows, page, dtype, j_star)
        out = torch.empty((Q, H, rank), device="cuda", dtype=dtype)
        ops.latent_attention_simple(_dev(q, dtype), _dev(pool), out, _dev(gates), _i32(positions), _i32([0] * Q), _i32(table).view(1, -1),
                                    page, H, rank, rot, 1.0, window)
        err = _rel(out, want)
        assert err < TOL[dtype], f"key {j_star} of {N} (page {page}, window {window}): error {err:.3g}"
        if dtype == torch.bfloat16 and ops.latent_attention_mma_supported(rank, rot):
            # the tensor-core kernel: the same rows as a second sequence of a batch whose first sequence is
            # short, whole and cut into key ranges
            short = 5
            q2 = torch.cat([q[:1].expand(short, H, D), q]).contiguous()
            g2 = torch.cat([gates[:1].expand(short, H), gates]).contiguous()
            tables = torch.full((2, len(table)), -1, dtype=torch.int32)
            tables[0, 0] = table[0]
            tables[1] = torch.tensor(table, dtype=torch.int32)
            for splits in (1, 3, 8):
                if splits > 1 and Q > 4:
                    continue
                out2 = torch.full((short + Q, H, rank), float("nan"), device="cuda", dtype=dtype)
                ops.latent_attention_mma(_dev(q2, dtype), _dev(pool), out2, _dev(g2), _i32([0, short, short + Q]), _i32([short, N]),
                                         _dev(tables), page, 2, max(short, Q), H, rank, rot, 1.0, window, splits)
                err = _rel(out2[short:], want)
                assert err < TOL[dtype], f"tensor cores, {splits} splits, key {j_star} of {N} (page {page}, window {window}): error {err:.3g}"
                assert bool(torch.isfinite(out2[:short].float()).all())


REBUILT_CASES = [
    # heads, rank, page, window, sinks, gates, portions (new tokens, context): tiles of 128 tokens in pairs, key blocks of 96
    (1, 64, 16, 0, False, False, [(5, 5)]),
    (2, 64, 16, 0, True, True, [(128, 128), (129, 130), (1, 95), (95, 96)]),
    (3, 72, 8, 0, False, True, [(256, 256), (257, 353), (7, 384)]),
    (2, 64, 4, 100, True, False, [(300, 700), (40, 40), (96, 193), (130, 1000)]),
    (2, 512, 32, 1, False, False, [(33, 97), (385, 385)]),
    (2, 512, 16, 4096, False, True, [(1, 2000), (515, 515)]),
]


@pytest.mark.parametrize("H, rank, page, window, sinks, gated, portions", REBUILT_CASES)
def test_latent_portions_with_rebuilt_keys(H, rank, page, window, sinks, gated, portions):
    """Gathered rows, keys and values made of them, and the tcgen05 attention, against float64 attention on the same rebuilt
    (rounded) keys and values: what is left is P rounded to bfloat16 (2^-9 of a weight) and the result's rounding, 1e-2
    of the largest entry as for the other bfloat16 attentions.  Pages that nobody sees are given back (NaN, table -1)."""
    from tokensprint_b200 import ops

    g = torch.Generator().manual_seed(H * 1000 + rank + page)
    D, B = rank + 64, len(portions)
    need = [-(-ctx // page) for _, ctx in portions]
    pool = torch.full((sum(need) + 3, page, D), float("nan"), dtype=torch.bfloat16)
    order, table, rows = torch.randperm(sum(need) + 3, generator=g).tolist(), torch.full((B, max(need)), -1, dtype=torch.int32), []
    for b, (n, ctx) in enumerate(portions):
        rows.append(torch.randn(ctx, D, generator=g).to(torch.bfloat16))
        lo = max(0, ctx - n - window + 1) if window else 0
        for j in range(lo // page * page, ctx):
            table[b, j // page] = order[sum(need[:b]) + j // page]
            pool[table[b, j // page], j % page] = rows[b][j]
    ahead = 3 * (H - 1)  # tokens of other sequences in front
    T = ahead + sum(n for n, _ in portions)
    q = torch.randn(T, H * 192, generator=g).to(torch.bfloat16)
    q_rot = torch.randn(T, H, 64, generator=g).to(torch.bfloat16)
    weight = (torch.randn(H * 256, rank, generator=g) / rank ** 0.5).to(torch.bfloat16)
    gates = torch.rand(T, H, generator=g) + 0.5 if gated else None
    sink = torch.randn(H, generator=g) if sinks else None
    cu = [ahead]
    for n, _ in portions:
        cu.append(cu[-1] + n)
    kept = [ops.latent_kept_keys(window, n, ctx) for n, ctx in portions]
    cached = torch.full((sum(kept), D), float("nan"), device="cuda", dtype=torch.bfloat16)
    starts, lens = _i32(cu), _i32([ctx for _, ctx in portions])
    ops.latent_gather(_dev(pool), cached, starts, lens, _dev(table), page, B, max(kept), window)
    at = 0
    for b, (n, ctx) in enumerate(portions):
        lo = max(0, ctx - n - window + 1) if window else 0
        want_rows = rows[b][ctx - kept[b]:].clone()
        want_rows[: lo - (ctx - kept[b])] = 0
        assert torch.equal(cached[at:at + kept[b]].cpu(), want_rows)
        at += kept[b]
    kv = ops.library_mm(cached[:, :rank], _dev(weight))
    wide = torch.full((T, H * 192 + 8), float("nan"), device="cuda", dtype=torch.bfloat16)  # rows that are not side by side
    wide[:, :-8] = _dev(q)
    out = torch.full((T, H, 128), float("nan"), device="cuda", dtype=torch.bfloat16)
    scale = 192 ** -0.5
    ops.latent_rebuilt_attention(wide[:, :-8], _dev(q_rot[ahead:]), kv, cached, out, None if gates is None else _dev(gates), starts, lens, B,
                                 max(n for n, _ in portions), H, rank, scale, window, None if sink is None else _dev(sink))
    ops.check_device_errors()
    made, at = kv.double().cpu(), 0
    for b, (n, ctx) in enumerate(portions):
        kb = made[at:at + kept[b]]
        see = torch.arange(ctx - n, ctx)[:, None] - torch.arange(ctx - kept[b], ctx)[None, :]
        see = (see >= 0) & (see < window) if window else see >= 0
        want = torch.empty(n, H, 128, dtype=torch.float64)
        for a in range(H):
            qa = torch.cat([q[cu[b]:cu[b + 1], a * 192:a * 192 + 128], q_rot[cu[b]:cu[b + 1], a]], 1).double()
            ka = torch.cat([kb[:, a * 128:a * 128 + 128], cached[at:at + kept[b], rank:].double().cpu()], 1)
            s = (qa @ ka.T * scale).masked_fill(~see, -math.inf)
            if sink is not None:
                s = torch.cat([s, sink[a].double().expand(n, 1)], 1)
            w = torch.softmax(s, 1)[:, :kept[b]]
            want[:, a] = w @ kb[:, (H + a) * 128:(H + a + 1) * 128] * (1.0 if gates is None else gates[cu[b]:cu[b + 1], a, None].double())
        assert _rel(out[cu[b]:cu[b + 1]], want) < 1e-2, f"portion {b}"
        at += kept[b]


def _rebuilt_one_head(keys, values, scale, gates=None):
    """latent_rebuilt_attention of a whole prompt of len(keys) tokens, one head; every query is the first unit vector."""
    from tokensprint_b200 import ops

    n = keys.shape[0]
    q = torch.zeros(n, 192)
    q[:, 0] = 1.0
    rows, out = torch.zeros(n, 128, device="cuda", dtype=torch.bfloat16), torch.empty(n, 1, 128, device="cuda", dtype=torch.bfloat16)
    q = _dev(q, torch.bfloat16)
    ops.latent_rebuilt_attention(q, q[:, 128:].contiguous(), _dev(torch.cat([keys, values], 1), torch.bfloat16), rows, out, gates, _i32([0, n]),
                                 _i32([n]), 1, n, 1, 64, scale)
    ops.check_device_errors()
    return out[:, 0].double().cpu()


@pytest.mark.parametrize("mantissa", [0, 3, 17, 40, 64, 71, 97, 110, 127])
@pytest.mark.parametrize("side", [2e-5, -2e-5])
def test_latent_rebuilt_weights_are_rounded_exponentials(mantissa, side):
    """Key 0 scores `scale`, all others 0, and exp(-scale) lies 2e-5 above or below the middle of two bfloat16
    numbers: every weight must round to the right one of them, wherever in a block its key stands.  Value entry c is 1 for the
    keys c modulo 8.  A wrong unit is at least 2^-8 of a weight and moves its columns by 7/8 of that; the results' own rounding, up
    to 2^-8 either way with a deviation of 1.6e-3, averages out over the rows (1.2e-4 for 190 of them; five times that is 6e-4)."""
    n = 200
    middle = (1 + (mantissa + 0.5) / 128) / 2 * (1 + side)
    w = float(torch.tensor(middle, dtype=torch.float64).to(torch.bfloat16))
    keys, values = torch.zeros(n, 128), torch.zeros(n, 128)
    keys[0, 0] = 1.0
    for j in range(1, n):
        values[j, j % 8] = 1.0
    out = _rebuilt_one_head(keys, values, -math.log(middle))
    count = values[:, :8].double().cumsum(0)
    want = count * w / (1.0 + torch.arange(n).double()[:, None] * w)
    assert float(((out[8:, :8] - want[8:]) / want[8:]).mean(0).abs().max()) < 1e-3


def test_latent_rebuilt_weights_add_up_to_one():
    """All values alike: the result is that value, whatever the weights were rounded to, up to float32 sums (200 terms, 2e-5).
    The gates bring the product within 1e-4 of the middle of two bfloat16 numbers, so a bias of the sum would show."""
    n = 200
    keys, values = torch.randn(n, 128, generator=torch.Generator().manual_seed(3)) * 3.0, torch.full((n, 128), 1.5)
    keys[0, 0] = 4.0
    for side in (1e-4, -1e-4):
        gate = torch.full((n, 1), (1.0 + 1.0 / 256) * (1.0 + side) / 1.5)
        out = _rebuilt_one_head(keys, values, 1.0, _dev(gate))
        assert torch.equal(out, torch.full_like(out, 1.0 + (1.0 / 128 if side > 0 else 0.0)))


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("tag, layer", [("a", 0), ("b", 0), ("b", 1), ("c", 1)])
def test_latent_mixer_whole_prompt(dtype, tag, layer):
    """The mixer part alone (projection, prepare kernel, absorbing products, attention, value
    products, output) against the plain function that rebuilds keys and values per head."""
    from tokensprint_b200.models.fegetar import build_fegetar_spec, FegetarConfig
    from tokensprint_b200.parts.base import BuildContext, GroupTables, LayerCache, StepContext, build_part

    cfg = FEG[tag]
    W = fegetar_weights(cfg, 17, sharp=2.0)
    spec = build_fegetar_spec(FegetarConfig.from_dict(cfg)).layers[layer].params["mixer"]
    mixer = build_part("mixer", spec, BuildContext(torch.device("cuda"), dtype))
    mixer.load({s.name: _dev(W[s.name], torch.float32 if s.role == "vector" else dtype) for s in mixer.tensor_specs()})
    T, page = 45, 16
    x = torch.randn(T, cfg["width"], generator=torch.Generator().manual_seed(5)).to(dtype)
    want = plain.latent_attention(x.double(), list(range(T)), {k: v.double() for k, v in W.items()}, f"l{layer}.mix.", cfg["layers"][layer]["mixer"],
                                  cfg["norm"]["eps"])
    pages = [2, 0, 3]
    pool = torch.full((4, page, mixer.key_dim), float("nan"), device="cuda", dtype=dtype)
    slots = [pages[j // page] * page + j % page for j in range(T)]
    step = StepContext(num_tokens=T, num_seqs=1, token_ids=_i32([0] * T), positions=_i32(range(T)), seq_index=_i32([0] * T),
                       cu_seqlens_q=_i32([0, T]), context_lens=_i32([T]), state_slots=_i32([0]),
                       groups=[GroupTables(_i32(pages).view(1, -1), _i32(slots))], page_size=page, max_seqlen_q=T, max_context_len=T)
    got = mixer.forward(_dev(x), step, LayerCache(group=0, k_pages=pool, writes=True))
    assert _rel(got, want) < (2e-5 if dtype == torch.float32 else 3e-2)


# ---------------------------------------------------------------------------
# routed experts


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("tag, layer, tokens", [("a", 0, 1), ("a", 0, 70), ("b", 1, 9), ("c", 0, 200), ("c", 1, 3)])
def test_routed_experts(dtype, tag, layer, tokens):
    from tokensprint_b200.models.fegetar import build_fegetar_spec, FegetarConfig
    from tokensprint_b200.parts.base import BuildContext, build_part

    cfg = FEG[tag]
    W = fegetar_weights(cfg, 23)
    spec = build_fegetar_spec(FegetarConfig.from_dict(cfg)).layers[layer].params["feed_forward"]
    part = build_part("feed_forward", spec, BuildContext(torch.device("cuda"), dtype))
    part.load({s.name: _dev(W[s.name], torch.float32 if s.role == "vector" else dtype) for s in part.tensor_specs()})
    x32 = torch.randn(tokens, cfg["width"], generator=torch.Generator().manual_seed(tokens))
    x = x32.to(dtype)
    want = plain.routed_ff(x.double(), {k: v.double() for k, v in W.items()}, f"l{layer}.mlp.", cfg["layers"][layer]["mlp"])
    got = part.forward(_dev(x), None, residual=_dev(x.float()))
    assert _rel(got, want) < (2e-5 if dtype == torch.float32 else 3e-2)
    # a token's result does not depend on the tokens beside it
    if tokens > 2:
        alone = part.forward(_dev(x[1:2]), None, residual=_dev(x[1:2].float()))
        assert _rel(alone, got[1:2]) < 1e-6 if dtype == torch.float32 else torch.equal(alone, got[1:2])


def test_router_picks_by_score_and_breaks_ties_by_index():
    from tokensprint_b200 import ops

    logits = torch.tensor([[0.0, 2.0, -1.0, 2.0, 1.0], [5.0, -5.0, 0.5, 0.25, 0.125]], device="cuda")
    ids = torch.empty((2, 3), dtype=torch.int32, device="cuda")
    w = torch.empty((2, 3), dtype=torch.float32, device="cuda")
    ops.router_topk(logits, 3, False, ids, w)
    assert ids.tolist() == [[1, 3, 4], [0, 2, 3]]
    assert torch.allclose(w.cpu(), torch.sigmoid(torch.tensor([[2.0, 2.0, 1.0], [5.0, 0.5, 0.25]])))
    ops.router_topk(logits, 3, True, ids, w)
    assert torch.allclose(w.sum(-1).cpu(), torch.ones(2))


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("T, W, E, top", [(1, 72, 7, 3), (9, 256, 12, 1), (130, 1000, 33, 4), (5, 70, 4, 4), (600, 128, 9, 2), (2100, 64, 5, 1)])
def test_router_in_one_kernel(dtype, T, W, E, top):
    from tokensprint_b200 import ops

    g = torch.Generator().manual_seed(T)
    x, r = torch.randn(T, W, generator=g).to(dtype), torch.randn(E, W, generator=g) / W ** 0.5
    ids = torch.empty((T, top), dtype=torch.int32, device="cuda")
    w = torch.empty((T, top), dtype=torch.float32, device="cuda")
    ops.router(_dev(x), _dev(r), top, False, ids, w)
    score = torch.sigmoid(x.double() @ r.double().T)
    want_w, want_e = torch.topk(score, top, dim=-1)
    assert torch.equal(ids.cpu().long(), want_e)
    assert torch.allclose(w.cpu().double(), want_w, atol=1e-6)


@pytest.mark.parametrize("P, E, K, I", [(1, 3, 64, 48), (70, 5, 96, 200), (300, 4, 520, 72), (40, 9, 128, 24), (36, 3, 72, 136)])
def test_expert_products_on_tensor_cores_against_cuda_cores(P, E, K, I, monkeypatch):
    """The same plan through both kernels; bfloat16, float32 sums in both."""
    from tokensprint_b200 import ops

    g = torch.Generator().manual_seed(P)
    top = 2 if P % 2 == 0 else 1
    T = P // top
    x = torch.randn(T, K, generator=g).to(torch.bfloat16).cuda()
    gate, up = (torch.randn(E, I, K, generator=g) / K ** 0.5).to(torch.bfloat16).cuda(), (torch.randn(E, I, K, generator=g) / K ** 0.5).to(torch.bfloat16).cuda()
    down = (torch.randn(E, K, I, generator=g) / I ** 0.5).to(torch.bfloat16).cuda()
    ids = torch.stack([torch.randperm(E, generator=g)[:top] for _ in range(T)]).to(torch.int32).cuda()
    w = (torch.rand(T * top, generator=g) * 0.8 + 0.1).cuda()
    results = []
    for mma in (True, False):
        monkeypatch.setattr(ops, "MOE_MMA", mma)
        plan = ops.moe_plan(ids, E, ops.moe_row_tile(ops.moe_on_tensor_cores(torch.bfloat16, K, I), T * top, E))
        act = torch.zeros((T * top, I), dtype=torch.bfloat16, device="cuda")
        out = torch.zeros((T * top, K), dtype=torch.bfloat16, device="cuda")
        ops.moe_gate_up(x, w, plan, gate, up, act, top, 1.5, 1.702)
        ops.moe_down(act, plan, down, out)
        results.append((act.float().cpu(), out.float().cpu()))
    # against float64, pair by pair
    for pair in range(T * top):
        e, h = int(ids.view(-1)[pair]), x[pair // top].double().cpu() * float(w[pair])
        a = (gate[e].double().cpu() @ h).clamp(max=1.5)
        b = (up[e].double().cpu() @ h).clamp(-1.5, 1.5)
        want = down[e].double().cpu() @ (a * torch.sigmoid(1.702 * a) * (b + 1))
        for act, out in results:
            assert float((out[pair].double() - want).abs().max()) < 3e-2 * float(want.abs().max()) + 1e-3
    assert float((results[0][1] - results[1][1]).abs().max()) < 2e-2 * float(results[1][1].abs().max())


@pytest.mark.parametrize("rows, E, K, I", [(1, 2, 64, 128), (31, 3, 72, 130), (32, 1, 200, 264), (33, 2, 64, 520), (127, 2, 136, 72), (128, 1, 64, 136),
                                           (129, 2, 72, 264), (400, 2, 264, 200), (3, 1100, 64, 16)])
@pytest.mark.parametrize("activation", ["capped_glu", "gelu"])
def test_expert_products_at_the_edges_of_their_tiles(rows, E, K, I, activation):
    """About `rows` pairs per expert (one expert gets none where there are several): row tiles of 32 and 128, weight tiles of 128
    and 256 rows, remainders of all of them, more experts than shared memory holds offsets for; a pair that points past the experts has
    no place.  Against float64 on the rounded inputs: the first product and the activation round to bfloat16 (2^-9 each)."""
    from tokensprint_b200 import ops

    g = torch.Generator().manual_seed(rows * 7 + E)
    T = rows if E > 8 else rows * max(1, E - 1)
    ids = torch.randint(0, max(1, E - 1), (T, 1), generator=g).to(torch.int32)
    if E > 1:
        ids[0] = E  # an identity expert: not in the plan
    x = torch.randn(T, K, generator=g).to(torch.bfloat16).cuda()
    matrix = lambda a, b: (torch.randn(E, a, b, generator=g) / b ** 0.5).to(torch.bfloat16).cuda()  # noqa: E731
    gate, up, down = None if activation == "gelu" else matrix(I, K), matrix(I, K), matrix(K, I)
    w = (torch.rand(T, generator=g) + 0.5).cuda()
    for tile in (ops.moe_row_tile(True, 1, 1), ops.moe_row_tile(True, 99, 1)):
        plan = ops.moe_plan(ids.cuda(), E, tile)
        places = plan[2].cpu()[: int(plan[0][-1])].long().cuda()
        e, h = ids.view(-1).cuda()[places].long(), x[places].double()
        product = lambda m, r: torch.stack([m[int(n)].double() @ row for n, row in zip(e, r)])  # noqa: E731
        for weight in (w, None):
            act = torch.full((T, I), float("nan"), dtype=torch.bfloat16, device="cuda")
            ops.moe_gate_up(x, weight, plan, gate, up, act, 1, 7.0, 1.702, activation)
            if not len(places):  # nobody's pair has a place: nothing is written
                assert bool(torch.isnan(act.float()).all())
                continue
            factor = 1.0 if weight is None else weight[places, None].double()
            u = factor * product(up, h)
            if gate is None:
                want = torch.nn.functional.gelu(u)
            else:
                a, u = (factor * product(gate, h)).clamp(max=7.0), u.clamp(-7.0, 7.0)
                want = a * torch.sigmoid(1.702 * a) * (u + 1.0)
            assert _rel(act[: len(places)], want) < 1e-2
        if len(places) and I % 8 == 0:
            out = torch.full((T, K), float("nan"), dtype=torch.bfloat16, device="cuda")
            ops.moe_down(act, plan, down, out)
            assert _rel(out[places], product(down, act[: len(places)].double())) < 5e-3
    ops.check_device_errors()


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("T, W, E", [(1, 8, 1), (7, 2048, 16), (296, 4104, 33), (297, 136, 5), (1535, 64, 32), (1536, 200, 65), (1601, 1160, 31), (40, 44, 6), (300, 42, 7)])
def test_router_logits_do_not_depend_on_the_kernel(dtype, T, W, E):
    """A CTA a token, tiles of 8 and of 16 tokens, and the kernel for odd rows add a token's logits up in the same order: the weights
    (sigmoid of the logits) are bit by bit those of the token alone, and close to float64."""
    from tokensprint_b200 import ops

    g = torch.Generator().manual_seed(T + W)
    x, r, bias = torch.randn(T, W, generator=g).to(dtype).cuda(), (torch.randn(E, W, generator=g) / W ** 0.5).cuda(), torch.randn(E, generator=g).cuda()
    top = min(E, 3)
    ids, w = torch.full((T, top), -1, dtype=torch.int32, device="cuda"), torch.full((T, top), float("nan"), device="cuda")
    ops.router(x, r, top, False, ids, w, bias=bias)
    for t in sorted({0, T // 2, T - 1}):
        one_id, one_w = torch.empty(1, top, dtype=torch.int32, device="cuda"), torch.empty(1, top, device="cuda")
        ops.router(x[t:t + 1].clone(), r, top, False, one_id, one_w, bias=bias)
        assert torch.equal(one_id[0], ids[t]) and torch.equal(one_w[0], w[t])
    z = x.double() @ r.double().T + bias.double()
    assert float((w.double() - torch.sigmoid(z.gather(1, ids.long()))).abs().max()) < 1e-5
    assert float((torch.topk(z, top).values - z.gather(1, ids.long())).abs().max()) < 1e-5


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("T, W, E, groups", [
    (592, 64, 8, None), (593, 64, 8, None), (148, 128, 20, None), (149, 128, 20, (4, 2)), (296, 1024, 20, None), (297, 1024, 20, None),
    (600, 136, 33, None), (1184, 64, 17, None), (1185, 64, 17, (17, 2)), (2368, 136, 16, None), (2369, 136, 40, (8, 3)), (2500, 72, 16, (4, 2)),
    # the logits of 16 tokens beside six slabs: up to 824 float32 entries (experts and groups), 1,208 of bfloat16 rows; four slabs
    # up to 1,616; beyond that the kernel without tiles
    (1185, 64, 824, None), (1185, 64, 825, None), (2368, 64, 1024, None), (2368, 64, 1024, (256, 200)), (1200, 64, 1024, (1024, 900)), (2400, 64, 1024, None),
])
def test_router_takes_every_number_of_experts(dtype, T, W, E, groups):
    """Every tile and ring that the sizes choose gives a token the choice and, bit by bit, the weights of the token alone (the kernel
    with a CTA a token), with expert groups and a correction too; the logits behind the weights are those of float64."""
    from tokensprint_b200 import ops

    g = torch.Generator().manual_seed(T + E)
    x, r = torch.randn(T, W, generator=g).to(dtype).cuda(), (torch.randn(E, W, generator=g) / W ** 0.5).cuda()
    correction = 0.1 * torch.randn(E, generator=g).cuda()
    top = min(E, 6)
    if groups is not None:
        top = min(top, groups[1] * (E // groups[0]))
    ids, w = torch.full((T, top), -1, dtype=torch.int32, device="cuda"), torch.full((T, top), float("nan"), device="cuda")
    ops.router(x, r, top, False, ids, w, score="softmax_all", correction=correction, groups=groups)
    for t in sorted({0, 7, 8, 15, 16, T // 2, T - 9, T - 1}):
        one_id, one_w = torch.empty(1, top, dtype=torch.int32, device="cuda"), torch.empty(1, top, device="cuda")
        ops.router(x[t:t + 1].clone(), r, top, False, one_id, one_w, score="softmax_all", correction=correction, groups=groups)
        assert torch.equal(one_id[0], ids[t]) and torch.equal(one_w[0], w[t])
    assert int(ids.min()) >= 0 and int(ids.max()) < E
    z = x.double() @ r.double().T
    assert float((w.double() - torch.softmax(z, 1).gather(1, ids.long())).abs().max()) < 1e-5


@pytest.mark.parametrize("T, E, top", [(3, 40, 40), (20, 33, 32), (2, 70, 33), (300, 70, 66), (1200, 100, 64), (4, 16, 8)])
@pytest.mark.parametrize("renormalize, scale", [(True, 1.0), (False, 2.5), (False, 1.0), (True, 0.5)])
def test_router_choices_in_order(T, E, top, renormalize, scale):
    """Many choices (a lane keeps every 32nd), ties, infinities: the order of the choices and the weights are those of a stable
    sort.  Weights: float32 sums of up to 66 sigmoids, 1e-5."""
    from tokensprint_b200 import ops

    g = torch.Generator().manual_seed(T + E + top)
    z = torch.round(torch.randn(T, E, generator=g) * 4) / 4  # quarters: many ties
    z[0, : E // 2] = -math.inf
    z[T - 1, E - 1] = math.inf
    r = torch.eye(E)  # rows are the logits themselves
    finite = z.clamp(-1e4, 1e4)
    order = torch.sort(finite, dim=1, descending=True, stable=True).indices[:, :top]
    for through in ("logits", "rows"):
        ids, w = torch.empty((T, top), dtype=torch.int32, device="cuda"), torch.empty((T, top), device="cuda")
        if through == "logits":
            ops.router_topk(z.cuda(), top, renormalize, ids, w, scale=scale)
        else:
            ops.router(finite.cuda(), r.cuda(), top, renormalize, ids, w, scale=scale)
        assert torch.equal(ids.cpu().long(), order)
        want = torch.sigmoid((z if through == "logits" else finite).double().gather(1, order))
        if renormalize:
            want = want / (want.sum(1, keepdim=True) + 1e-20)
        assert float((w.cpu().double() - want * scale).abs().max()) < 1e-5
