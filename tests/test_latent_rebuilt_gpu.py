"""Prompt portions of latent attention whose keys and values are rebuilt (heads of 128 + 64 entries and values of 128, the only
sizes that the kernel has), through the engine: small Fegetar, Vasosun and Mugulorn models of these sizes against the plain models,
whole, in portions and beside decoded tokens, with the choice between the two routes forced either way; gathered rows
that a reading layer uses again; the bound on the memory that the rebuilt route takes; the rule that chooses.

Pages that a window has passed are given back with NaN in them, so a row that nobody may see shows."""

from types import SimpleNamespace

import pytest
import torch

from tests.fegetar_configs import _mixer as feg_mixer, _moe as feg_moe, fegetar_weights, write_fegetar_folder
from tests.mugulorn_configs import _lat as mug_lat, _layer as mug_layer, _model as mug_model, _rec, _yarn, mugulorn_weights, random_ids, write_mugulorn_folder
from tests.plain import fegetar_plain, mugulorn_plain, vasosun_plain
from tests.replay_helpers import first_bad, replay_in_process, trace_decode_tail, trace_mixed, trace_portions, trace_whole, worst_error
from tests.vasosun_configs import _dense, _lat as vas_lat, _layer as vas_layer, _model as vas_model, vasosun_weights, write_vasosun_folder
from tokensprint_b200.parts import latent_attention as latent

TOLERANCE = 8e-2  # of the largest |logit|, as for the other bfloat16 runs of these designs (their files say why)

# no window; gates, sinks or none by design; the absorbed steps of a latent of 72 entries run on the simple kernel
FEG = {"architecture": "Fegetar", "vocab": 211, "width": 96, "norm": {"eps": 1e-5}, "layers": [
    {"type": "latent_attention", "mixer": feg_mixer(8, 128, 64, 128, 72, 10000.0, 32), "mlp": feg_moe(5, 2, 48, 1.5, (72, 0.75))},
    {"type": "latent_attention", "mixer": feg_mixer(8, 128, 64, 128, 512, 10000.0, 64), "mlp": {"kind": "dense", "ff": 160}}]}
_V_ROT = (1000.0, 64, _yarn(4.0, 32, 8.0, 1.0))
VAS = vas_model(130, 72, 3e-6, 3, 61, 31, 1, 50.0, [
    vas_layer(vas_lat(2, 128, 64, 128, 512, 48, 0.08, *_V_ROT), _dense(40)),
    vas_layer(vas_lat(3, 128, 64, 128, 512, 40, 0.07, *_V_ROT, kv_from=0), _dense(56))])
# the writer's window, a longer one, the writer's again, another head count, none: readers with equal and different windows
_M_ROT = (1000.0, _yarn(4.0, 32, 8.0, 1.0))
MUG = mug_model(97, 100, 2e-5, 1.0, 0.5, [
    mug_layer(mug_lat(2, 128, 64, 128, 512, 24, 0.08, *_M_ROT, window=48), 52),
    mug_layer(mug_lat(3, 128, 64, 128, 512, 32, 0.07, *_M_ROT, window=48, kv_from=0)),
    mug_layer(_rec(52, 13, 2), 52),
    mug_layer(mug_lat(1, 128, 64, 128, 512, 16, 0.09, *_M_ROT, window=130, kv_from=0), 40),
    mug_layer(mug_lat(2, 128, 64, 128, 512, 16, 0.08, *_M_ROT, kv_from=0)),
    mug_layer(mug_lat(2, 128, 64, 128, 72, 16, 0.08, *_M_ROT, window=7))])

DESIGNS = {
    "fegetar": (FEG, lambda cfg: fegetar_weights(cfg, 61, routed_share=0.01), write_fegetar_folder, lambda ids, w, cfg: fegetar_plain.forward(ids, w, cfg)[0]),
    "vasosun": (VAS, lambda cfg: vasosun_weights(cfg, 62), write_vasosun_folder, lambda ids, w, cfg: vasosun_plain.forward_logits(ids, w, cfg)),
    "mugulorn": (MUG, lambda cfg: mugulorn_weights(cfg, 63), write_mugulorn_folder, lambda ids, w, cfg: mugulorn_plain.forward_logits(ids, w, cfg)),
}


class Oracle:
    def __init__(self, cfg, weights, forward):
        self.cfg, self.weights, self.forward, self._cache = cfg, weights, forward, {}

    def logits(self, ids):
        key = tuple(ids)
        if key not in self._cache:
            self._cache[key] = self.forward(ids, self.weights, self.cfg)
        return self._cache[key]


@pytest.fixture(scope="module")
def models(tmp_path_factory):
    out = {}
    for name, (cfg, make, write, forward) in DESIGNS.items():
        weights = make(cfg)
        requests = {f"r{i}": random_ids(cfg, n, 900 + i) for i, n in enumerate([5, 95, 130, 231])}
        out[name] = (write(tmp_path_factory.mktemp(name), cfg, weights), cfg, requests, Oracle(cfg, weights, forward))
    return out


def _replayer(folder, max_tokens=512, **kw):
    from tokensprint_b200.engine.replay import TraceReplayer

    r = TraceReplayer.from_folder(folder, "bfloat16", max_tokens, page_size=16, max_live=4, **kw)
    r.runner.poison_freed_pages = True
    return r


def _check(got, requests, oracle, what):
    worst, where = worst_error(got, requests, oracle)
    bad = first_bad(got, requests, oracle, TOLERANCE)
    assert bad is None, f"{what}: first wrong token at request {bad[0]} position {bad[1]} (error {bad[2]:.3g}); worst {worst:.3g} at {where}"
    assert len(got) == sum(len(v) for v in requests.values())


@pytest.fixture
def calls(monkeypatch):
    """Counts the launches of the rebuilt route."""
    from tokensprint_b200 import ops

    counts = {"latent_gather": 0, "latent_rebuilt_attention": 0, "beside": 0}
    for name in ("latent_gather", "latent_rebuilt_attention"):
        def counted(*args, _inner=getattr(ops, name), _name=name, **kw):
            counts[_name] += 1
            if _name == "latent_rebuilt_attention":
                counts["beside"] += args[1].shape[0] < args[0].shape[0]  # decoded tokens in front
            return _inner(*args, **kw)

        monkeypatch.setattr(ops, name, counted)
    return counts


@pytest.mark.gpu
@pytest.mark.parametrize("cut", ["whole", "decode tail", "portions", "mixed"])
@pytest.mark.parametrize("design", sorted(DESIGNS))
def test_both_routes_in_every_cutting(models, calls, monkeypatch, design, cut):
    folder, cfg, requests, oracle = models[design]
    steps = {"whole": lambda: trace_whole(requests), "decode tail": lambda: trace_decode_tail(requests, 12),
             "portions": lambda: trace_portions(requests, (33, 2, 97, 5, 64, 16)), "mixed": lambda: trace_mixed(requests, 512, seed=5)}[cut]()
    got = {}
    for pays in (True, False):
        monkeypatch.setattr(latent, "rebuilding_pays", lambda *a, **k: pays)
        before = dict(calls)
        got[pays] = replay_in_process(_replayer(folder), steps)
        _check(got[pays], requests, oracle, f"{cut}, rebuilt {pays}")
        ran = {k: v - before[k] for k, v in calls.items()}
        assert (ran["latent_rebuilt_attention"] > 0) == pays
        if pays and cut == "mixed":
            assert ran["beside"] > 0, "no portion stood beside decoded tokens"
    if cut == "whole":
        assert any(bool((got[True][k] != got[False][k]).any()) for k in got[True]), "both runs took the same route"


@pytest.mark.gpu
def test_gathered_rows_are_used_again_and_given_up(models, calls, monkeypatch):
    """The writer gathers; the reader of the same window does not; the ones of other windows gather again, and the last reader
    leaves nothing behind, nor does a layer whose rows nobody reads (the last one)."""
    folder, cfg, requests, oracle = models["mugulorn"]
    monkeypatch.setattr(latent, "rebuilding_pays", lambda *a, **k: True)
    held = []
    plan = latent.LatentAttentionMixer._rebuild_plan

    def watched(self, step, *args):
        held.append(list(step.shared.get("latent rows", {}).values()))
        return plan(self, step, *args)

    monkeypatch.setattr(latent.LatentAttentionMixer, "_rebuild_plan", watched)
    replay_in_process(_replayer(folder), trace_whole({"r": requests["r3"]}))
    assert calls["latent_rebuilt_attention"] == 5 and calls["latent_gather"] == 4
    assert [len(h) for h in held] == [0, 1, 1, 1, 0]
    assert held[1][0][1] is held[2][0][1] and held[1][0][0] == (48, 0) and held[3][0][0] == (130, 0)


@pytest.mark.gpu
@pytest.mark.parametrize("spare", [0, -1])
def test_the_bound_counts_everything_that_is_held(models, calls, monkeypatch, spare):
    """A bound that holds the first layer's rows, keys and values, and not a byte less."""
    folder, cfg, requests, oracle = models["mugulorn"]
    n = len(requests["r2"])
    monkeypatch.setattr(latent, "rebuilding_pays", lambda *a, **k: True)
    monkeypatch.setattr(latent, "LATENT_REBUILD_MAX_BYTES", n * (2 * 256 + 576) * 2 + spare)
    got = replay_in_process(_replayer(folder), trace_whole({"r": requests["r2"]}))
    _check(got, {"r": requests["r2"]}, oracle, "bounded")
    # layers of two heads fit (the first, the fourth reader, the last with its shorter rows), the one of three does not, one of one does
    assert calls["latent_rebuilt_attention"] == (4 if spare == 0 else 2)


@pytest.mark.gpu
def test_the_pool_is_sized_with_the_route_that_takes_more(models, monkeypatch):
    from tokensprint_b200.engine.runner import ModelRunner
    from tokensprint_b200.models.api import load_model

    folder, cfg, requests, oracle = models["fegetar"]
    model, _ = load_model(folder, device="cuda", dtype="bfloat16")
    peaks = []
    for on in (True, False):
        monkeypatch.setattr(latent, "LATENT_REBUILD", on)
        monkeypatch.setattr(latent, "rebuilding_pays", lambda *a, **k: True)
        runner = ModelRunner(model, page_size=16, num_slots=2, max_num_batched_tokens=600, gpu_memory_utilization=0.05, max_model_len=512)
        peaks.append(runner.sizing["step_peak_bytes"])
        del runner
    assert peaks[0] == peaks[1]


def _step(starts, lens, decode_seqs=0, **kw):
    return SimpleNamespace(num_tokens=sum(lens), num_seqs=len(lens), max_seqlen_q=max(lens), host_seq_starts=starts, host_seq_lens=lens,
                           decode_seqs=decode_seqs, shared={}, sizing=False, **kw)


def _plan(monkeypatch, step, heads=16, window=0, others=0, offset=0):
    """_rebuild_plan of a layer of these sizes, without a GPU."""
    from tokensprint_b200 import ops

    def kept(window, n, context):
        first = max(0, context - n - window + 1) if window else 0
        return context - first // 96 * 96

    monkeypatch.setattr(ops, "latent_kept_keys", kept)
    monkeypatch.setattr(ops, "_sm_count", lambda device: 148)
    cache = SimpleNamespace(group=0, k_pages=torch.empty(1))
    if others:
        step.shared["latent rows"] = {(1, 2): ((0, 0), torch.empty(others // 2, dtype=torch.bfloat16, device="meta"))}
    layer = SimpleNamespace(kv_weight=torch.empty(heads * 256, 512, device="meta"), window=window, num_heads=heads, key_dim=576,
                            _held_key=latent.LatentAttentionMixer._held_key)
    q = torch.empty(sum(step.host_seq_lens), heads * 192 + offset, dtype=torch.bfloat16)
    return latent.LatentAttentionMixer._rebuild_plan(layer, step, q, cache)


def test_plan_of_a_step(monkeypatch):
    assert _plan(monkeypatch, _step([0], [8191])) == (0, [8191])
    assert _plan(monkeypatch, _step([8000], [2000]), window=512) == (0, [10000 - 7489 // 96 * 96])
    assert _plan(monkeypatch, _step([0, 100], [3000, 2000])) == (0, [3000, 2100])
    step, asked = _step([0, 100], [3000, 2000]), []
    pays = latent.rebuilding_pays
    monkeypatch.setattr(latent, "rebuilding_pays", lambda *a: asked.append(a) or pays(*a))
    for window, heads in ((0, 16), (0, 16), (0, 8), (512, 16), (512, 16)):
        _plan(monkeypatch, step, heads, window)
    assert len(asked) == 3, "layers of one kind share the plan of a step"
    many = _step([900] * 4 + [0, 7000], [1] * 4 + [4000, 4000], decode_seqs=4)
    assert _plan(monkeypatch, many) == (4, [4000, 11000])


def test_beside_decoded_tokens_the_device_must_save_what_the_host_pays():
    """The two sides of the line (measured steps): a prompt of 1,024 tokens with 16 heads saves the device 177 us a layer and
    loses, the same with 32 heads saves 381 and wins; alone both are rebuilt."""
    for portions, heads, pays in (([(700, 700), (420, 420)], 16, False), ([(1024, 1024)], 16, False), ([(500, 500)] * 4, 16, False),
                                  ([(700, 700)] * 2, 32, True), ([(1024, 1024)], 32, True), ([(1024, 1024)] * 2, 16, True), ([(2048, 2048)], 16, True)):
        assert latent.rebuilding_pays(portions, heads, 148)
        assert latent.rebuilding_pays(portions, heads, 148, beside_decodes=True) == pays
    assert not latent.rebuilding_pays([(40, 40)], 16, 148)


def test_plan_keeps_to_absorbed_queries(monkeypatch):
    whole = lambda step: (step.num_tokens, [])  # noqa: E731
    for step in (_step([0], [40]), _step([5000], [4]), _step([100] * 8, [1] * 8, decode_seqs=8)):  # short, a few tokens, decode
        assert _plan(monkeypatch, step) == whole(step)
    step = _step([0], [8191])
    assert _plan(monkeypatch, step, offset=4) == whole(step)  # rows that are not 16 bytes apart
    step.sizing = True
    assert _plan(monkeypatch, step) == whole(step)
    row = (16 * 256 + 576) * 2  # bytes of a kept row and what is made of it
    most = latent.LATENT_REBUILD_MAX_BYTES // row
    assert _plan(monkeypatch, _step([most - 4000], [4000])) == (0, [most])
    assert _plan(monkeypatch, _step([most + 1 - 4000], [4000])) == (4000, [])
    assert _plan(monkeypatch, _step([most - 4000], [4000]), others=row) == (4000, [])  # beside rows that another cache's readers wait for
    monkeypatch.setattr(latent, "LATENT_REBUILD", False)
    assert _plan(monkeypatch, _step([0], [8191])) == (8191, [])
