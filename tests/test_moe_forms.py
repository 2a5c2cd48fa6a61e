"""Which form of a GEMM is taken: the MoE layer's rule by rows per expert, its overrides, what autotune() keeps, and the plain product."""
import pytest

from dlslime_b200.models.moe import ExpertGemmForm, ExpertParallelMoE, expert_gemm_form

ROWS = {1: ExpertGemmForm(False, 0, 64, 64), 32: ExpertGemmForm(False, 0, 64, 64), 64: ExpertGemmForm(False, 0, 0, 128),
        128: ExpertGemmForm(False, 0, 0, 192), 175.9: ExpertGemmForm(False, 0, 0, 192), 320: ExpertGemmForm(False, 0, 0, 0),
        500: ExpertGemmForm(False, 0, 0, 0), 512: ExpertGemmForm(True, 0, 0, 0), 1023: ExpertGemmForm(True, 0, 0, 0), 4096: ExpertGemmForm(True, 0, 0, 0)}


@pytest.mark.parametrize("depth", [256, 1024, 2048, 7168])
@pytest.mark.parametrize("rows,form", ROWS.items())
def test_rule_by_rows_per_expert(rows, form, depth):
    assert expert_gemm_form(rows, depth, {}) == form


@pytest.mark.parametrize("depth,pair", [(256, False), (768, False), (1024, False), (1536, "swap"), (2048, "swap"), (7168, "swap")])
@pytest.mark.parametrize("rows", [176, 200, 300, 319.9])
def test_swapped_pairs_only_where_the_products_are_deep(rows, depth, pair):
    """Narrow layers lose up to 1.5x on swapped pairs (256 experts of 1024 x 256, 256 rows each: 569 us a step against 348)."""
    assert expert_gemm_form(rows, depth, {}) == ExpertGemmForm(pair, 0, 0, 0)


@pytest.mark.parametrize("rows", [40, 200, 500])
def test_overrides_are_taken_in_every_range(rows):
    """A tile override is one of the single-CTA forms, so it also holds where swapped pairs would be the default."""
    assert expert_gemm_form(rows, 2048, {"SLIME_EP_TILE_TOKENS": "128"})[::3] == (False, 128)
    assert expert_gemm_form(rows, 2048, {"SLIME_EP_TILE_N": "192"})[:2] == (False, 192)
    assert expert_gemm_form(rows, 2048, {"SLIME_EP_TILE_N": "192"}).tile_tokens == 0
    assert expert_gemm_form(rows, 2048, {"SLIME_EP_TILE_M": "64"})[:3] == (False, 0, 64)
    assert expert_gemm_form(rows, 2048, {"SLIME_EP_PAIR_GEMM": "0"}).pair is False
    assert expert_gemm_form(rows, 2048, {"SLIME_EP_PAIR_GEMM": "1"}).pair is True
    assert expert_gemm_form(rows, 2048, {"SLIME_EP_PAIR_GEMM": "swap", "SLIME_EP_TILE_M": "0"}).pair == "swap"


class _Timed(ExpertParallelMoE):
    """The layer without a GPU: a step takes what the table says for the form that is set."""

    def __init__(self, rows, times):
        form = expert_gemm_form(rows, 2048, {})
        self._default_pair_gemm = self.pair_gemm = form.pair
        self.tile_tokens, self.fuse_dequant, self.streamed = form.tile_tokens, False, False
        self.times, self.timed = times, []

    def _time_step(self, x, logits, out, steps):
        self.timed.append("streamed" if self.streamed else self.pair_gemm)
        return self.times[self.timed[-1]]


@pytest.mark.parametrize("rows,times,pair,streamed", [
    (200, {"swap": 2.64, False: 3.14, True: 3.00, "streamed": 3.2}, "swap", False),   # the layer's own choice is one of the candidates
    (200, {"swap": 2.64, False: 2.62, True: 3.00, "streamed": 2.65}, "swap", False),  # less than 1 % does not replace it
    (200, {"swap": 2.64, False: 2.50, True: 3.00, "streamed": 2.4}, False, True),
    (1024, {False: 2.81, True: 2.82, "streamed": 2.9}, True, False),
    (128, {False: 4.7, True: 5.4, "streamed": 5.0}, False, False),
])
def test_autotune_keeps_the_layers_choice_unless_another_form_wins(rows, times, pair, streamed):
    layer = _Timed(rows, times)
    got = layer.autotune(None, None)
    assert layer.timed[0] == layer._default_pair_gemm and {False, True} <= set(layer.timed)
    assert layer.pair_gemm is pair or layer.pair_gemm == pair
    assert layer.streamed is streamed and got["streamed"] is streamed and got["pair_gemm"] == layer.pair_gemm
    assert got["serial_ms"] == times[pair] and got["streamed_ms"] == times["streamed"]


def test_autotune_times_every_form_on_request(monkeypatch):
    monkeypatch.setenv("SLIME_EP_AUTOTUNE_ALL", "1")
    layer = _Timed(500, {"swap": 3.0, False: 3.0, True: 3.5, "wide": 2.5, "streamed": 3.0})
    assert layer.autotune(None, None)["serial_cta_pair_wide_ms"] == 2.5 and layer.pair_gemm == "wide"
    assert layer.timed == [False, True, "wide", "swap", "streamed"]


@pytest.mark.parametrize("shared,m,k,entries", [
    (True, 500, 7168, ["slime_gemm_bf16_few"]), (False, 500, 7168, ["slime_gemm_bf16_few", "slime_gemm_bf16_pair"]),
    (True, 500, 1024, ["slime_gemm_bf16_pair"]), (True, 255, 1024, ["slime_gemm_bf16"]), (False, 72, 7168, ["slime_gemm_bf16"]),
    (True, 513, 7168, ["slime_gemm_bf16_pair"])])
def test_products_of_few_tiles_follow_the_launchers_rule(monkeypatch, shared, m, k, entries):
    """gemm_bf16 leaves it to the launcher whether a tile's K is shared over a cluster; where it is not (clusters that do not fit, a
    smaller device) a product with a full 256-row tile goes to CTA pairs. Products of many tiles do not ask."""
    import torch

    from dlslime_b200.ops import gemm

    calls = []

    def call(name, *args):
        calls.append(name)
        return int(name == "slime_gemm_bf16_few" and not shared)

    monkeypatch.setattr(gemm, "require_cuda", lambda *t: None)
    monkeypatch.setattr(gemm, "_sms", lambda device: 148)
    monkeypatch.setattr(gemm, "ptr", lambda t: 0)
    monkeypatch.setattr(gemm, "stream_ptr", lambda *a: 0)
    monkeypatch.setattr(gemm, "default_status", lambda: type("S", (), {"dev_ptr": 0}))
    monkeypatch.setattr(gemm._lib, "call", call)
    a, b = torch.empty(m, k, dtype=torch.bfloat16), torch.empty(2048, k, dtype=torch.bfloat16)
    assert gemm.gemm_bf16(a, b).shape == (m, 2048)
    assert [c.replace("_wide", "_pair") for c in calls] == entries


@pytest.mark.parametrize("world,fuse,thin,trace,names", [
    (1, False, False, None, ["route", "dispatch_quant_expand", "gate_up_swiglu_gemm", "down_gemm_combine_push", "combine_wait_reduce"]),
    (1, True, False, None, ["route", "dispatch_quant_push", "recv_wait_dequant", "gate_up_swiglu_gemm", "down_gemm_combine_push", "combine_wait_reduce"]),
    (1, False, True, None, ["route", "dispatch_quant_push", "recv_wait_dequant", "gate_up_swiglu_gemm", "down_gemm_combine_push", "combine_wait_reduce"]),
    (1, False, False, 7, ["route", "dispatch_quant_push", "recv_wait_dequant", "gate_up_swiglu_gemm", "down_gemm_combine_push", "combine_wait_reduce"]),
    (2, False, False, None, ["route", "dispatch_quant_push", "recv_wait_dequant", "gate_up_swiglu_gemm", "down_gemm_combine_push", "combine_wait_reduce"]),
])
def test_a_step_runs_the_phases_it_reports(world, fuse, thin, trace, names):
    """forward() launches exactly what phases() names (bench.py times those one by one): one rank expands in dispatch, unless
    the receive kernel is needed."""
    import torch

    ran = []
    layer = ExpertParallelMoE.__new__(ExpertParallelMoE)
    layer.world, layer.fuse_dequant, layer.thin_waits, layer.streamed, layer.xd = world, fuse, thin, False, None
    layer.buf = type("B", (), {"trace": trace, "dispatch_expand": lambda self, *a: ran.append("dispatch_quant_expand")})()
    for attr, name in (("step_route", "route"), ("step_dispatch", "dispatch_quant_push"), ("step_recv", "recv_wait_dequant"),
                       ("step_gate_up", "gate_up_swiglu_gemm"), ("step_down", "down_gemm_combine_push"), ("step_combine", "combine_wait_reduce")):
        setattr(layer, attr, lambda *a, _n=name, **k: ran.append(_n))
    x = torch.zeros(3, 8)
    phases = layer.phases(x, x, x)
    assert [n for n, _ in phases] == names
    layer.forward(x, x)
    assert ran == names
    for _, launch in phases:
        launch()
    assert ran == 2 * names
