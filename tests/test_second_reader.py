"""A call that reads a recurrent state which another call of the same step has moved on: its kernel waits for that call."""
import contextlib
import types

import pytest
import torch

import bolonex_cases as bx
import helpers
import lurisun_cases as lu
import petanex_cases as px

gpu = pytest.mark.gpu
DEV = "cuda:0"


class _Recorder:
    """Stands in for the compiled library: keeps the last entry point's name and arguments."""

    def __getattr__(self, name):
        def call(*args):
            if name.endswith("_supported"):
                return 1
            self.last = (name, args)
            return 0
        return call


def _calls(ops, ctx, writes):
    """Every operation on a fixed state in a step of single rows -> (entry point, arguments)."""
    f = lambda *s: torch.zeros(*s)
    lib = ops.library()
    out = []
    for run in (lambda: ops.ssm_scan(f(2, 24), f(2, 4), 0, f(2), f(2), f(2), f(2, 2, 4, 8), f(2, 8), 2, 1, 4, 8, ctx, writes),
                lambda: ops.delta_rule(f(2, 24), 0, 8, 16, f(2, 2), 0, f(2, 2), 0, False, f(2), f(2), f(2, 2, 4, 4), f(2, 8), 2, 2, 4, 4, ctx, writes),
                lambda: ops.short_conv(f(2, 8), 0, None, f(8, 3), None, "silu", f(2, 2, 8), f(2, 8), ctx, commit_inline=writes),
                lambda: ops.decay_memory(f(2, 24), 0, 8, 16, None, f(2, 513), f(2, 2, 4, 4), f(2, 8), 2, 4, 4, ctx, writes),
                lambda: ops.add_rmsnorm_conv(f(2, 8), f(8), 1e-5, f(2, 8), f(8, 3), f(2, 2, 8), f(2, 8), ctx, writes)):
        run()
        out.append(lib.last)
    return out


@pytest.mark.parametrize("writes", [True, False])
@pytest.mark.parametrize("settled", [True, False, None])
def test_states_are_read_early_only_by_the_writer_of_a_step(monkeypatch, writes, settled):
    """The flag before the stream says that the state may be read before the kernels ahead have finished: only for the call
    that moves it on, and only under a context that says the states were last written before the step."""
    from kungfu_b200 import ops
    lib = _Recorder()
    monkeypatch.setattr(ops, "_lib", lib)
    monkeypatch.setattr(ops, "_p", lambda t: t)
    monkeypatch.setattr(ops, "_stream", lambda: "stream")
    ints = torch.zeros(2, dtype=torch.int32)
    ctx = types.SimpleNamespace(n_reqs=2, decode_only=True, req_row_start=ints, req_n_rows=ints, req_state_slot=ints, row_req=ints)
    if settled is not None:
        ctx.states_settled = settled
    names = set()
    for name, args in _calls(ops, ctx, writes):
        names.add(name)
        assert args[-1] == "stream" and args[-2] == int(writes and settled is True), name
    assert names == {"kf_ssm_scan", "kf_delta_rule", "kf_short_conv", "kf_decay_memory", "kf_add_rmsnorm_conv"}


def test_a_step_says_that_its_states_are_settled():
    from kungfu_b200.engine import StepContext
    from kungfu_b200.parts.model import DecoderModel, LayerCall
    assert StepContext.states_settled is True
    head, block = types.SimpleNamespace(vocab=4), object()          # what that rests on: one writing call per slot, readers after it
    for bad in ([LayerCall(0, 0), LayerCall(0, 0)], [LayerCall(0, 0, writes=False), LayerCall(0, 0)]):
        with pytest.raises(ValueError):
            DecoderModel(object(), [block], head, bad)


@gpu
@pytest.mark.parametrize("family,kind", [("bolonex", "Mamba2Mixer"), ("petanex", "GatedDeltaMixer"), ("lurisun", "LightningAttention")])
@pytest.mark.parametrize("graphs", [False, True])
def test_a_second_call_that_only_reads(tmp_path, family, kind, graphs):
    """The schedule runs a recurrent layer a second time on the same slot without writing: prompts of unequal length, then
    decode steps of three requests, to the bit what launches in full order give."""
    from kungfu_b200 import api, ops
    from kungfu_b200.engine import StepEntry
    from kungfu_b200.parts.model import DecoderModel, LayerCall
    cases, cfg_dict = {"bolonex": (bx, bx.BX_E), "petanex": (px, px.PX_E), "lurisun": (lu, lu.LU_E)}[family]
    folder = cases.write_model(str(tmp_path / "m"), cfg_dict, seed=4)
    toks = {f"r{i}": helpers.random_tokens(n + 12, cfg_dict["vocab"], 50 + i) for i, n in enumerate((3, 40, 9))}
    runs = []
    for order in (contextlib.nullcontext(), ops.plain_launches()):
        with order:
            cfg, model = api.load_model(folder, dtype="bfloat16", device=DEV)
            sched = []
            for call in model.schedule:
                sched.append(call)
                if type(model.layers[call.layer].mixer).__name__ == kind:
                    sched.append(LayerCall(call.layer, call.cache, writes=False))
            assert len(sched) > len(model.schedule)
            twice = DecoderModel(model.embedding, model.layers, model.head, sched)
            runner = api.make_runner(cfg, twice, dtype="bfloat16", device=DEV, page_size=64, max_tokens=512, max_requests=3,
                                     max_context=256, cuda_graphs=graphs)
            rows = []
            for r in toks:
                runner.cache.add_request(r)
            rows.append(runner.step([StepEntry(r, t[:-12], [len(t) - 13]) for r, t in toks.items()]).clone())
            for k in range(12, 0, -1):
                rows.append(runner.step([StepEntry(r, [t[-k]], [0]) for r, t in toks.items()]).clone())
            ops.raise_on_device_error(torch.device(DEV))
            runs.append(torch.cat(rows))
    assert bool(torch.isfinite(runs[0]).all()) and torch.equal(runs[0], runs[1])
