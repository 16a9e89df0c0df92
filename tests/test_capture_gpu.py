"""Captured steps of the 32-bit path (the bits of the eager path, results that later steps leave alone), and the streams that captures
and side branches run on (never one and the same)."""
import pytest
import torch

import helpers as H

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("name", ["a", "b", "c"])
def test_float32_steps_are_captured_and_their_results_stay(name):
    from infer_b200 import StepEntry
    from test_engine_gpu import _engine
    cfg = H.TINY[name]
    engines = [_engine(name, torch.float32, cuda_graphs=g) for g in (False, True)]
    assert engines[1].use_graphs
    ids = {r: H.random_ids(cfg, 30, 70 + i) for i, r in enumerate("xy")}
    kept = []
    for eng in engines:
        outs = []
        for r in "xy":
            eng.add_request(r)
        outs.append(eng.step([StepEntry(r, ids[r][:20], [19]) for r in "xy"]))
        for t in range(20, 30):
            outs.append(eng.step([StepEntry(r, ids[r][t:t + 1], [0]) for r in "xy"]))
        eng.check_status()
        kept.append(outs)
    assert len(engines[1]._graphs) > 0
    for t, (a, b) in enumerate(zip(*kept)):
        assert torch.equal(a, b), f"step {t}"


def test_streams_of_captures_and_side_branches_differ():
    from infer_b200 import fast_ops
    from infer_b200.parts.block import _side_streams
    device = torch.device(DEV)
    sides = _side_streams(device)
    for _ in range(31):                                  # (torch hands out 32 streams in turn)
        torch.cuda.Stream(device)
    handles = [s.cuda_stream for s in (*sides, fast_ops.capture_stream(device), fast_ops.own_stream(device))]
    assert len(set(handles)) == 4
    assert fast_ops.capture_stream(device) is fast_ops.capture_stream(device)


# ------------------------------------------------------------------------------------------------ what decides the bits of a step

def _one_layer(heads, kv):
    return dict(architectures=["Qwen2ForCausalLM"], hidden_size=heads * 128, num_hidden_layers=1, num_attention_heads=heads,
                num_key_value_heads=kv, intermediate_size=256, vocab_size=320, rope_theta=1000000.0, rms_norm_eps=1e-6,
                max_position_embeddings=4096, tie_word_embeddings=True)


# (contexts that are no multiple of a page or a tile, where the attention's form or parts for the true context are not those for the
# table's width: (64 keys, 3 parts) and (128, 1); (128, 4) and (64, 3))
@pytest.mark.parametrize("heads,kv,first,n", [(12, 2, 915, 2048), (28, 4, 732, 300)])
def test_bits_of_a_portion_do_not_depend_on_what_was_captured(heads, kv, first, n, monkeypatch):
    """Whether a shape is captured, and when, follows from measured times; the step's result may not."""
    from infer_b200 import Engine, StepEntry
    from infer_b200.engine import engine as module
    cfg = _one_layer(heads, kv)
    ids = H.random_ids(cfg, first + n, heads)
    results = []
    for worth in (True, False):
        def decide(self, ms_per_launch, worth=worth):
            if self.launches:                            # (it has run eagerly once, as every shape does first)
                self.worth = worth
            return bool(self.worth)
        monkeypatch.setattr(module._PortionRun, "decide", decide)
        eng = Engine(H.spec_of(cfg), H.make_weights(cfg, 3), max_tokens=4096, max_requests=1)
        for _ in range(module.PORTION_GRAPH_LATER + 2):
            eng.add_request("r")
            eng.step([StepEntry("r", ids[:first], [])])
            results.append(eng.step([StepEntry("r", ids[first:], [0, n // 2, n - 1])]).clone())
            eng.end_request("r")
        eng.check_status()
        assert eng._graphs
    for i, r in enumerate(results[1:]):
        assert torch.equal(r, results[0]), f"pass {i + 1}"


def test_a_capture_without_memory_leaves_the_step_to_the_eager_way(monkeypatch):
    """No room for a graph's activations is no reason for a step to fail."""
    from infer_b200 import StepEntry
    from test_engine_gpu import _engine
    ids = H.random_ids(H.TINY["a"], 30, 5)
    outs = []
    for short in (False, True):
        eng = _engine("a", torch.float32, cuda_graphs=short)
        run_model = eng._run_model

        def none_left(ctx):
            if torch.cuda.is_current_stream_capturing():
                raise torch.cuda.OutOfMemoryError("no room for a graph")
            return run_model(ctx)
        if short:
            monkeypatch.setattr(eng, "_run_model", none_left)
        eng.add_request("r")
        outs.append([eng.step([StepEntry("r", ids[:20], [19])])] + [eng.step([StepEntry("r", ids[t:t + 1], [0])]) for t in range(20, 30)])
        eng.check_status()
        assert not eng._graphs or not any(e.graphs for e in eng._graphs.values())
    for a, b in zip(*outs):
        assert torch.equal(a, b)


@pytest.mark.parametrize("own_streams", [True, False])
def test_engines_in_two_threads_capture_their_steps(own_streams):
    """Steps of float32 engines in threads of their own, each on its own stream or both on the default one: new shapes (and so captures) all the time in both, and
    device memory asked for outside of a capture while the other captures."""
    import threading
    from infer_b200 import StepEntry
    from test_engine_gpu import _engine
    cfg = H.TINY["b"]
    ids = {r: H.random_ids(cfg, 40, 30 + i) for i, r in enumerate("abcd")}

    def run(eng, stream, out, keep):
        with torch.cuda.stream(stream):
            for batch in (1, 2, 3, 4):
                rids = "abcd"[:batch]
                for r in rids:
                    eng.add_request(r)
                out.append(eng.step([StepEntry(r, ids[r][:20], [19]) for r in rids]))
                for t in range(20, 40):
                    out.append(eng.step([StepEntry(r, ids[r][t:t + 1], [0]) for r in rids]))
                    keep.append(torch.empty((1 << 20) + 4096 * len(keep), dtype=torch.uint8, device=DEV))
                for r in rids:
                    eng.end_request(r)
            stream.synchronize()
    want, results, errors = [], [[], []], []
    run(_engine("b", torch.float32, cuda_graphs=False), torch.cuda.default_stream(), want, [])

    def guarded(i, eng, stream):
        try:
            run(eng, stream, results[i], [])
        except Exception as e:
            errors.append(e)
    engines = [_engine("b", torch.float32) for _ in range(2)]
    torch.cuda.synchronize()
    threads = [threading.Thread(target=guarded, args=(i, engines[i], torch.cuda.Stream() if own_streams else torch.cuda.default_stream())) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for got in results:
        assert len(got) == len(want) and all(torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16], ids=["f32", "bf16"])
def test_a_capture_after_the_last_graph_has_gone(dtype, monkeypatch):
    """The shapes of single tokens take turns in a table of two: the only captured one leaves for shapes that have not been captured yet."""
    from infer_b200 import StepEntry
    from infer_b200.engine import engine as module
    from test_engine_gpu import _engine
    monkeypatch.setattr(module, "MAX_GRAPHS", 2)
    cfg = H.TINY["a"]
    ids = H.random_ids(cfg, 60, 5)
    outs = []
    for graphs in (False, True):
        eng = _engine("a", dtype, cuda_graphs=graphs)
        at = {r: 0 for r in "abc"}

        def some(rids, n):
            for _ in range(n):
                outs[-1].append(eng.step([StepEntry(r, ids[at[r]:at[r] + 1], [0]) for r in rids]).clone())
                for r in rids:
                    at[r] += 1
        outs.append([])
        for r in "abc":
            eng.add_request(r)
        some("a", 4)
        assert not graphs or [len(e.graphs) for e in eng._graphs.values()] == [2]
        some("ab", 1)
        some("abc", 1)
        assert not any(e.graphs for e in eng._graphs.values())
        some("ab", 4)
        some("a", 4)
        some("abc", 4)
        torch.randn(4, device=DEV)
        eng.check_status()
    for i, (a, b) in enumerate(zip(*outs)):
        assert (a - b).abs().max() < (1e-6 if dtype == torch.float32 else 0.05), f"step {i}"


# ------------------------------------------------------------------------------------------------ parts that change after they were captured

def test_float32_steps_see_what_was_replaced():
    """A method or a matrix that is replaced between steps is in use from the next step on, as without graphs; with the package's own
    method back in its place steps are captured again."""
    from infer_b200 import StepEntry
    from test_engine_gpu import _engine
    cfg = H.TINY["b"]
    ids = H.random_ids(cfg, 60, 9)
    calls = []

    def run(eng):
        eng.add_request("r")
        outs = [eng.step([StepEntry("r", ids[:10], [9])])]
        at = 10

        def some(n):
            nonlocal at
            for _ in range(n):
                outs.append(eng.step([StepEntry("r", ids[at:at + 1], [0])]))
                at += 1
        some(6)
        mixer = eng.model.blocks[1].mixer
        own = type(mixer).forward

        def counted(*a, **k):
            calls.append(eng)
            return own(mixer, *a, **k)
        mixer.forward = counted
        before = len(calls)
        some(5)
        assert len(calls) == before + 5
        del mixer.forward
        some(6)
        assert len(calls) == before + 5
        eng.model.head.linear.weight = eng.model.head.linear.weight * 2.0
        some(6)
        eng.model.blocks[0], eng.model.blocks[2] = eng.model.blocks[2], eng.model.blocks[0]
        some(6)
        eng.end_request("r")
        return outs
    eager, captured = _engine("b", torch.float32, cuda_graphs=False), _engine("b", torch.float32)
    for i, (a, b) in enumerate(zip(run(eager), run(captured))):
        assert torch.equal(a, b), f"step {i}"
    assert captured.use_graphs and any(e.graphs for e in captured._graphs.values())


@pytest.mark.parametrize("cases", ["ruvenex", "notirax", "pefazen", "bolelix", "fozerax", "biravik"])
def test_the_packages_designs_are_its_own(cases):
    import importlib
    from infer_b200 import Engine
    mod = importlib.import_module(cases + "_cases")
    for name, cfg in mod.CASES.items():
        spec = mod.spec_of(cfg)
        from infer_b200.weights import random_weights
        eng = Engine(spec, random_weights(spec, 1, torch.float32), dtype=torch.float32, max_tokens=64, max_requests=1)
        assert eng.use_graphs, name


def test_a_mixer_from_elsewhere_beside_another_is_run_eagerly():
    """One of two mixers side by side is registered from elsewhere: the 32-bit path runs every step."""
    from dataclasses import replace
    import ruvenex_cases as rc
    from infer_b200 import Engine, StepEntry
    from infer_b200.parts.base import part_class, register_mixer, unregister
    from infer_b200.weights import random_weights
    cfg = rc.CASES["p"]
    spec = rc.spec_of(cfg)
    second = spec.layers[0].parts["mixer"][1]["second"]
    runs = []

    class Elsewhere(part_class("mixer", second.kind)):
        def forward(self, *a, **k):
            runs.append(1)
            return super().forward(*a, **k)
    register_mixer("from_elsewhere")(Elsewhere)
    try:
        spec.layers[0].parts["mixer"][1].params["second"] = replace(second, kind="from_elsewhere")
        eng = Engine(spec, random_weights(spec, 1, torch.float32), dtype=torch.float32, max_tokens=64, max_requests=1)
        assert not eng.use_graphs
        ids = H.random_ids({"vocab_size": cfg["vocab"]}, 20, 1)
        eng.add_request("r")
        for t in range(20):
            eng.step([StepEntry("r", ids[t:t + 1], [0])])
        assert len(runs) == 20
    finally:
        unregister("mixer", "from_elsewhere")
