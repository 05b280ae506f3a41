"""GPU tests of what the encoder's one-call inference keeps between calls (flashdeberta_b200/engine.py): when it is made again, and
who may rely on it.  The reference for every output is the module walk (taken when the layers' hidden states are asked for)."""
import pytest
import torch

from tests.test_configs_gpu import _close, _ragged, _small_config

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _model(**kw):
    from flashdeberta_b200 import FlashDebertaV2Model
    torch.manual_seed(0)
    return FlashDebertaV2Model(_small_config("b200", **kw)).eval().to(DEV).bfloat16()


def _walk(model, ids, mask):
    return model(input_ids=ids, attention_mask=mask, output_hidden_states=True).last_hidden_state


def _capture(run):
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        out = run()
    return graph, out


@pytest.mark.parametrize("rows", [40, 600])
def test_capture_after_a_weight_was_written(rows):
    """The position tables depend on the key projection.  Written to between the warm-up and the capture, a graph has to gather
    them itself, and the calls around it (eager, before and after a replay) have to be right too."""
    from flashdeberta_b200 import ops
    model = _model()
    ids, mask = _ragged(1, rows, (rows - 3,))
    run = lambda: model(input_ids=ids, attention_mask=mask).last_hidden_state
    with torch.no_grad():
        old = run()
        for layer in model.encoder.layer:
            layer.attention.self.key_proj.weight.mul_(3.0)
        graph, out = _capture(run)
        eager = run()                   # before the graph has ever run
        assert not torch.equal(eager, old)
        _close(eager, _walk(model, ids, mask), 0.1, 5e-3, "eager after the capture")
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, eager)
        for layer in model.encoder.layer:
            layer.attention.self.key_proj.weight.mul_(0.5)
        graph.replay()                  # the graph that gathers sees the weights of its replay
        torch.cuda.synchronize()
        assert torch.equal(out, run())
    ops.check_status()


def test_first_call_of_a_plan_inside_a_capture():
    """A parameter replaced between warm-up and capture: the plan of the captured call is the graph's own."""
    model = _model()
    ids, mask = _ragged(2, 300, (300, 170))
    run = lambda: model(input_ids=ids, attention_mask=mask).last_hidden_state
    with torch.no_grad():
        run()
        proj = model.encoder.layer[0].attention.self.key_proj
        proj.weight = torch.nn.Parameter(proj.weight * 2)
        graph, out = _capture(run)
        eager = run()
        _close(eager, _walk(model, ids, mask), 0.1, 5e-3, "eager after the capture")
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, eager)


def test_tables_are_published_behind_their_event(monkeypatch):
    """A second thread that calls the model while the first one is still gathering the tables must not take them for gathered: it waits
    until the gathering and its event are on the first one's stream, and has its own stream wait for that event."""
    import threading
    from flashdeberta_b200 import ops
    from flashdeberta_b200.attention import FlashDisentangledSelfAttention
    model = _model()
    ids, mask = _ragged(1, 600, (500,))
    with torch.no_grad():
        model(input_ids=ids, attention_mask=mask)  # plan and buffers
        model.encoder.layer[2].attention.self.key_proj.weight.mul_(3.0)
        want = _walk(model, ids, mask)
    torch.cuda.synchronize()
    started, go_on, outs, errors = threading.Event(), threading.Event(), {}, []
    position_tables = FlashDisentangledSelfAttention._position_tables

    def late_tables(self, *a, **kw):
        torch.cuda._sleep(50_000_000)              # the gathering takes some 80 ms on its stream
        return position_tables(self, *a, **kw)

    class LateEvent(torch.cuda.Event):             # the moment between the making of an event and its record
        def record(self, *a, **kw):
            started.set()
            go_on.wait(2.0)
            return super().record(*a, **kw)

    monkeypatch.setattr(FlashDisentangledSelfAttention, "_position_tables", late_tables)
    monkeypatch.setattr(torch.cuda, "Event", LateEvent)

    def call(name):
        try:
            with torch.no_grad(), torch.cuda.stream(torch.cuda.Stream()):
                outs[name] = model(input_ids=ids, attention_mask=mask).last_hidden_state
                torch.cuda.current_stream().synchronize()
        except Exception as e:  # noqa: BLE001 (reported below)
            errors.append(e)

    first = threading.Thread(target=call, args=("first",))
    first.start()
    started.wait(10.0)
    second = threading.Thread(target=call, args=("second",))
    second.start()
    second.join(0.3)
    go_on.set()
    first.join(), second.join()
    assert not errors, errors
    assert torch.equal(outs["first"], outs["second"])
    _close(outs["second"], want, 0.1, 5e-3, "second thread")
    ops.check_status()


def _scribble(nbytes, n=24):
    """Memory of this size from the current stream's pool, overwritten."""
    return [torch.full((nbytes // 2,), float("nan"), dtype=torch.bfloat16, device=DEV) for _ in range(n)]


def test_tables_outlive_the_calls_of_other_streams():
    """A call on another stream still reads the tables when a weight is replaced and the plan they belong to goes: their memory must
    not be handed out before that call is over."""
    model = _model()
    ids, mask = _ragged(1, 600, (500,))
    run = lambda: model(input_ids=ids, attention_mask=mask).last_hidden_state
    side = torch.cuda.Stream()
    with torch.no_grad():
        size = 3 * 2 * 4 * 1527 * 64 * 2  # layers, terms, heads, rows, features, bytes
        proj = model.encoder.layer[0].attention.self.key_proj
        for _ in range(2):  # (a kernel's first launch may wait for the device)
            proj.weight = torch.nn.Parameter(proj.weight.clone())
            want = run()
            junk = _scribble(size)
        del junk
        torch.cuda.synchronize()
        with torch.cuda.stream(side):
            torch.cuda._sleep(200_000_000)
            got = run()
        assert not side.query()
        held, proj.weight = proj.weight, torch.nn.Parameter(proj.weight.clone())
        run()
        junk = _scribble(size, 48)
        torch.cuda.synchronize()
        assert torch.equal(got, want)
    del held, junk


def test_tables_outlive_the_plan_a_graph_was_captured_with():
    """Another plan for the same weights (a module was swapped): a graph captured before still reads valid tables."""
    model = _model()
    ids, mask = _ragged(1, 600, (500,))
    run = lambda: model(input_ids=ids, attention_mask=mask).last_hidden_state
    with torch.no_grad():
        want = run()
        graph, out = _capture(run)
        model.encoder.layer[0].output.dropout = torch.nn.Dropout(0.0).eval()
        assert torch.equal(run(), want)
        junk = _scribble(3 * 2 * 4 * 1527 * 64 * 2)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want)
    del junk


def test_tables_of_a_weight_with_other_storage():
    """The same parameter with other storage (no version counted): the tables are gathered again."""
    model = _model()
    ids, mask = _ragged(2, 300, (300, 170))
    with torch.no_grad():
        model(input_ids=ids, attention_mask=mask)
        for layer in model.encoder.layer:
            weight = layer.attention.self.query_proj.weight
            weight.data = weight.data * 3
        got = model(input_ids=ids, attention_mask=mask).last_hidden_state
        _close(got, _walk(model, ids, mask), 0.1, 5e-3, "other storage")


def _all_layers(set_one):
    return lambda model: [set_one(layer) for layer in model.encoder.layer]


@pytest.mark.parametrize("change", [
    _all_layers(lambda l: setattr(l.attention.self, "attn_fp8", True)),
    _all_layers(lambda l: setattr(l.attention.output.LayerNorm, "eps", 0.5)),
    _all_layers(lambda l: setattr(l.output.LayerNorm, "eps", 0.5)),
    lambda model: model.encoder.layer[0].attention.self.pos_att_type.remove("p2c"),  # (one list, which the layers share)
    _all_layers(lambda l: setattr(l.attention.self, "max_relative_positions", 300)),
    _all_layers(lambda l: setattr(l.intermediate, "_erf_gelu", False) or setattr(l.intermediate, "intermediate_act_fn", torch.nn.ReLU())),
    lambda model: setattr(model.encoder.layer[1].attention.self, "attn_fp8", True),
    lambda model: setattr(model.encoder.LayerNorm, "eps", 0.5),
], ids=["attn_fp8", "attention eps", "output eps", "pos_att_type", "max_relative_positions", "activation", "attn_fp8 of one layer", "table eps"])
def test_encoder_call_notices_settings(change):
    """A setting of a module, changed between two calls, holds from the next one on (and so does changing it back)."""
    from flashdeberta_b200 import ops
    model = _model()
    ids, mask = _ragged(2, 600, (600, 333))
    with torch.no_grad():
        first = model(input_ids=ids, attention_mask=mask).last_hidden_state
        change(model)
        got = model(input_ids=ids, attention_mask=mask).last_hidden_state
        assert not torch.equal(got, first)
        _close(got, _walk(model, ids, mask), 0.1, 5e-3, "changed")
    ops.check_status()


def test_settings_back_and_forth():
    model = _model()
    ids, mask = _ragged(1, 40, (40,))
    run = lambda: model(input_ids=ids, attention_mask=mask).last_hidden_state
    ln = model.encoder.layer[0].output.LayerNorm
    with torch.no_grad():
        first = run()
        eps, ln.eps = ln.eps, 0.5
        assert not torch.equal(run(), first)
        ln.eps = eps
        assert torch.equal(run(), first)


def test_hooks_on_every_module_are_called():
    from torch.nn.modules.module import register_module_forward_hook, register_module_forward_pre_hook
    model = _model()
    ids, mask = _ragged(1, 40, (40,))
    run = lambda: model(input_ids=ids, attention_mask=mask).last_hidden_state
    with torch.no_grad():
        first = run()
        for register in (register_module_forward_hook, register_module_forward_pre_hook):
            seen = []
            hook = register(lambda m, *a: seen.append(m))
            try:
                _close(run(), first, 0.1, 5e-3, "with a hook")
            finally:
                hook.remove()
            assert {*model.encoder.layer, model.embeddings} <= set(seen)
        assert torch.equal(run(), first)


def test_weights_that_are_no_parameters_are_read_where_they_are():
    """A sharding wrapper puts plain tensors in the place of parameters, others for every forward: nothing of the model may be read
    where it was the time before."""
    model = _model()
    ids, mask = _ragged(2, 300, (300, 170))
    linears = [m for m in model.encoder.modules() if type(m) is torch.nn.Linear]
    with torch.no_grad():
        first = model(input_ids=ids, attention_mask=mask).last_hidden_state
        flat = [(m, m._parameters.pop("weight").detach()) for m in linears]

        def forward(scale):
            for m, w in flat:
                m.__dict__["weight"] = w * scale
            got = model(input_ids=ids, attention_mask=mask).last_hidden_state
            want = _walk(model, ids, mask)
            held = [m.__dict__.pop("weight") for m, _ in flat]
            for t in held:
                t.fill_(float("nan"))
            return got, want

        got, want = forward(1.0)
        _close(got, want, 0.1, 5e-3, "gathered weights")
        _close(got, first, 0.1, 5e-3, "gathered weights")
        got, want = forward(1.5)
        _close(got, want, 0.1, 5e-3, "gathered weights, others")
        assert not torch.equal(got, first)


def test_parameters_of_a_subclass_go_through_the_modules():
    class Wrapped(torch.nn.Parameter):
        pass

    model = _model()
    ids, mask = _ragged(1, 40, (40,))
    with torch.no_grad():
        want = model(input_ids=ids, attention_mask=mask).last_hidden_state
        for layer in model.encoder.layer:
            layer.output.dense.weight = Wrapped(layer.output.dense.weight.data)
        _close(model(input_ids=ids, attention_mask=mask).last_hidden_state, want, 0.1, 5e-3, "subclass")
        assert not model._engine.plan.ok


def test_model_from_before_there_was_an_engine():
    """A model pickled whole by an earlier version has no ``_engine``."""
    model = _model()
    ids, mask = _ragged(1, 40, (40,))
    with torch.no_grad():
        want = model(input_ids=ids, attention_mask=mask).last_hidden_state
        del model.__dict__["_engine"]
        assert torch.equal(model(input_ids=ids, attention_mask=mask).last_hidden_state, want)


def test_replica_of_data_parallel():
    """torch.nn.DataParallel runs shallow copies of the model with plain tensors for parameters, in threads: they must neither use nor
    disturb what the original keeps."""
    model = _model()
    ids, mask = _ragged(2, 300, (300, 170))
    with torch.no_grad():
        want = model(input_ids=ids, attention_mask=mask).last_hidden_state
        plan = model._engine.plan
        replica, = torch.nn.parallel.replicate(model, [torch.device(DEV, torch.cuda.current_device())], detach=True)
        got = replica(input_ids=ids, attention_mask=mask).last_hidden_state
        _close(got, want, 0.1, 5e-3, "replica")
        assert model._engine.plan is plan


@pytest.mark.parametrize("lens", [(597,), (500, 129), (0, 0), (1, 600)])
def test_masked_call_does_not_depend_on_what_memory_held(lens):
    """The same bits whatever the workspace was used for before: rows behind the valid ones are nobody's."""
    model = _model()
    ids, mask = _ragged(len(lens), 600, lens)
    run = lambda: model(input_ids=ids, attention_mask=mask).last_hidden_state
    with torch.no_grad():
        for layer in model.encoder.layer:  # (scores that spread widely: the running maxima move)
            layer.attention.self.query_proj.weight.mul_(8.0)
            layer.attention.self.key_proj.weight.mul_(8.0)
        first = run()
        for value in (0.0, 50.0, -3.0, float("inf"), float("nan")):
            pool = [torch.full((n // 2,), value, dtype=torch.bfloat16, device=DEV) * torch.randn(n // 2, device=DEV).bfloat16()
                    for n in (1 << 20, 2 << 20, 4 << 20, 8 << 20, 16 << 20, 32 << 20) for _ in range(4)]
            del pool
            assert torch.equal(run(), first), value
        if any(lens):  # (the walk does not take a batch without a token)
            _close(first, _walk(model, ids, mask), 0.1, 5e-3, "against the walk")
        else:
            assert torch.count_nonzero(first) == 0


def test_captures_of_the_module_leave_each_other_alone():
    """The attention module called for the first time inside a capture, and again in a second one before the first has run: neither
    relies on what the other would set up, nor does an eager call on the same stream."""
    from flashdeberta_b200 import ops
    module, warm = (_model().encoder.layer[0].attention.self for _ in range(2))
    x, rel = torch.randn(2, 300, 256, device=DEV).bfloat16(), torch.randn(512, 256, device=DEV).bfloat16()
    lens = torch.tensor([300, 131], dtype=torch.int32, device=DEV)
    stream = torch.cuda.Stream()
    with torch.no_grad():
        want = warm(x, lens, rel_embeddings=rel)[0]  # (the bucket table, and the kernels)
        torch.cuda.synchronize()
        graphs = []
        for _ in range(2):
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=stream):
                out = module(x, lens, rel_embeddings=rel)[0]
            graphs.append((graph, out))
        with torch.cuda.stream(stream):
            eager = module(x, lens, rel_embeddings=rel)[0]
        for graph, out in reversed(graphs):
            graph.replay()
            torch.cuda.synchronize()
            assert torch.equal(out, want)
        assert torch.equal(eager, want)
    ops.check_status()


def test_mask_analysed_in_a_capture_is_analysed_again():
    """A batch that stays padded (pack_sequences off): the lengths counted in a capture are the graph's."""
    from flashdeberta_b200 import ops
    model = _model(pack_sequences=False)
    ids, mask = _ragged(2, 300, (300, 131))
    run = lambda m: model(input_ids=ids, attention_mask=m).last_hidden_state
    with torch.no_grad():
        want = run(mask)
        other = mask.clone()
        graph, out = _capture(lambda: run(other))
        assert torch.equal(run(other), want)
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want)
    ops.check_status()
