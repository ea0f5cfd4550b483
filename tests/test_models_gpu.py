"""Model zoo on a GPU in 16-bit precision: the native kernels (tcgen05 GEMM / convolution,
layer norm, softmax, fused softmax-cross-entropy, batch norm, fused optimizer) carry a few
training steps of every model family."""
import math
import os
import subprocess
import sys

import pytest
import torch

import lbann_b200 as lbann
from lbann_b200.exec.trainer import ExecTrainer
from lbann_b200.ops import native
from lbann_b200.utils import options as opts
from test_models_cpu import _reader

pytestmark = pytest.mark.gpu


def _train_gpu(model, reader, steps, mb, dtype, optimizer=None, graph=False):
    o = opts.reset()
    o.set("default_dtype", dtype)
    if graph:
        o.set("use_cuda_graph", True)
    exp = lbann.proto.serialize.build_experiment(
        trainer=lbann.Trainer(mini_batch_size=mb, random_seed=3), model=model, data_reader=reader,
        optimizer=optimizer or lbann.Adam(learn_rate=2e-3, beta1=0.9, beta2=0.99, eps=1e-8))
    tr = ExecTrainer(exp)
    m = tr.build_model(exp.model)
    dc = tr.data_coordinator
    dc.start_epoch("training")
    b = dc.next_batch("training")
    n0 = native.launches()
    losses = []
    for _ in range(steps):
        m.train_step(b.tensors, b.global_size)
        losses.append(float(m.last_objective))
    assert native.consume_status() == 0
    assert native.launches() > n0, "no native kernel ran"
    if graph:
        assert m._graph_mode and any("graph" in e for e in m._graphs.values()), "step was not captured"
    tr.shutdown()
    assert all(math.isfinite(v) for v in losses), losses
    return losses


def test_gpt_bf16():
    from lbann_b200.models.transformer import construct_gpt_model
    torch.manual_seed(0)
    model = construct_gpt_model(vocab_size=256, seq_len=64, d_model=128, num_heads=4, num_layers=2,
                                ffn_dim=512)
    losses = _train_gpu(model, _reader(8, [65], "randint:256"), steps=20, mb=8, dtype="bf16")
    assert losses[0] == pytest.approx(math.log(256), rel=0.25)
    assert losses[-1] < 0.9 * losses[0], losses


def test_resnet18_bf16():
    from lbann_b200.models import ResNet18, construct_classifier
    torch.manual_seed(0)
    model = construct_classifier(ResNet18(16, width=0.5), 16)
    losses = _train_gpu(model, _reader(16, [3, 64, 64], "normal", label_classes=16), steps=10, mb=16,
                        dtype="bf16", optimizer=lbann.SGD(learn_rate=0.05, momentum=0.9))
    assert losses[-1] < losses[0], losses


def test_unet3d_fp16():
    from lbann_b200.models import construct_unet3d_model
    torch.manual_seed(0)
    model = construct_unet3d_model(num_classes=3, base_channels=8, levels=2)
    r = _reader(2, [1, 32, 32, 32], "samples:normal responses:randint:3", response_dims=[32, 32, 32])
    losses = _train_gpu(model, r, steps=8, mb=2, dtype="fp16")
    assert losses[-1] < losses[0], losses


def test_attention_score_fusion_matches_unfused(monkeypatch):
    """Folding 1/sqrt(d) and the causal mask into the softmax kernel does not change the
    training trajectory beyond 16-bit rounding."""
    from lbann_b200.models.transformer import construct_gpt_model

    def run():
        torch.manual_seed(0)
        model = construct_gpt_model(vocab_size=128, seq_len=32, d_model=64, num_heads=4, num_layers=2,
                                    ffn_dim=128, name="gptf")
        return _train_gpu(model, _reader(8, [33], "randint:128"), steps=6, mb=8, dtype="bf16")

    fused = run()
    monkeypatch.setenv("LBANN_DISABLE_ATTENTION_FUSION", "1")
    plain = run()
    for a, b in zip(fused, plain):
        assert abs(a - b) < 3e-2 * max(1.0, abs(b)), (fused, plain)



@pytest.mark.parametrize("family", ["cosmoflow_amp", "gpt"])
def test_cuda_graph_replay_matches_eager_steps(family):
    """The training step captured as a CUDA graph (after three ordinary steps) and replayed
    gives the losses of the step-by-step run: same kernels, same order, device-side
    optimizer step counter and loss-scale schedule."""
    def build():
        torch.manual_seed(0)
        if family == "gpt":
            from lbann_b200.models.transformer import construct_gpt_model
            m = construct_gpt_model(vocab_size=256, seq_len=64, d_model=128, num_heads=4, num_layers=2,
                                    ffn_dim=512)
            return m, _reader(8, [65], "randint:256"), "bf16"
        from lbann_b200.models.cosmoflow import construct_cosmoflow_model, synthetic_reader
        m = construct_cosmoflow_model(32, 4, 4, num_epochs=1, channels=(16, 32, 32), pool_mode="max",
                                      conv_bias=False, fc_sizes=(64, 32))
        m.amp = lbann.AmpOptions(enabled=True, init_scale=1024.0)
        return m, synthetic_reader(8, 32, 4, 4), "fp16"

    model, reader, dt = build()
    sgd = lambda: lbann.Adam(learn_rate=1e-4, beta1=0.9, beta2=0.99, eps=1e-8)      # noqa: E731
    eager = _train_gpu(model, reader, steps=10, mb=8, dtype=dt, optimizer=sgd())
    model, reader, dt = build()
    again = _train_gpu(model, reader, steps=10, mb=8, dtype=dt, optimizer=sgd())
    model, reader, dt = build()
    replay = _train_gpu(model, reader, steps=10, mb=8, dtype=dt, optimizer=sgd(), graph=True)
    # tolerance: what two step-by-step runs differ by (fp32 atomics in the filter gradients)
    noise = max(abs(a - b) for a, b in zip(eager, again))
    for a, b in zip(eager, replay):
        assert abs(a - b) <= max(5.0 * noise, 2e-3 * max(1.0, abs(a))), (eager, again, replay)


def test_learning_rate_change_reaches_a_captured_step():
    """A learning-rate schedule keeps working under graph replay: the optimizer kernel reads
    its hyper-parameters from a device table that is refreshed before a replay."""
    from lbann_b200.models.transformer import construct_gpt_model
    torch.manual_seed(0)
    o = opts.reset()
    o.set("default_dtype", "bf16")
    o.set("use_cuda_graph", True)
    model = construct_gpt_model(vocab_size=128, seq_len=32, d_model=64, num_heads=2, num_layers=1, ffn_dim=128)
    exp = lbann.proto.serialize.build_experiment(
        trainer=lbann.Trainer(mini_batch_size=4, random_seed=3), model=model,
        data_reader=_reader(4, [33], "randint:128"), optimizer=lbann.SGD(learn_rate=0.05))
    tr = ExecTrainer(exp)
    m = tr.build_model(exp.model)
    dc = tr.data_coordinator
    dc.start_epoch("training")
    b = dc.next_batch("training")
    for _ in range(6):
        m.train_step(b.tensors, b.global_size)
    assert any("graph" in e for e in m._graphs.values())
    before = m.arena.master.detach().clone()
    m.train_step(b.tensors, b.global_size)
    moved = float((m.arena.master - before).abs().max())
    for s in m.arena.slots:
        s.hp["learn_rate"] = 0.0
    before = m.arena.master.detach().clone()
    m.train_step(b.tensors, b.global_size)
    frozen = float((m.arena.master - before).abs().max())
    tr.shutdown()
    assert native.consume_status() == 0
    assert moved > 0.0 and frozen == 0.0, (moved, frozen)


def test_kfac_on_gpu_beats_plain_sgd():
    """K-FAC preconditioning (Kronecker factors, damped inverses) with the layers' native
    kernels underneath reaches a lower objective than plain SGD in the same epochs."""
    from test_algorithms_cpu import _fit
    sgd = lbann.BatchedIterativeOptimizer("sgd", epoch_count=3)
    kfac = lbann.KFAC("kfac", sgd, damping_act="1e-2", damping_err="1e-2", kronecker_decay=0.9,
                      update_intervals="1", compute_interval=1)
    plain = _fit(sgd, cuda=True)
    second = _fit(kfac, cuda=True)
    assert native.consume_status() == 0
    assert math.isfinite(second) and second < plain, (plain, second)


@pytest.mark.parametrize("graph", [False, True])
def test_overwritten_gradients_equal_accumulated_ones(graph, monkeypatch):
    """Fully-connected gradients with one writer are overwritten instead of cleared and added to: the same
    gradients and weights after several steps, with a weight that two layers share and one that no objective
    reaches (cleared: it has stale values, then zeros)."""
    from lbann_b200.exec.model import ExecModel

    def run(least):
        monkeypatch.setattr(ExecModel, "_OVERWRITE_MIN", least)
        o = opts.reset()
        o.set("default_dtype", "bf16")
        o.set("use_cuda_graph", graph)
        x = lbann.Input(data_field="samples")
        target = lbann.Input(data_field="responses")
        shared = lbann.Weights(name="shared", initializer=lbann.HeNormalInitializer())
        h = lbann.Relu(lbann.FullyConnected(x, num_neurons=40, has_bias=True, name="first"))
        h = lbann.FullyConnected(h, num_neurons=40, has_bias=False, weights=[shared], name="a")
        h = lbann.FullyConnected(h, num_neurons=40, has_bias=False, weights=[shared], name="b")
        lbann.FullyConnected(h, num_neurons=16, has_bias=False, name="aside")
        y = lbann.FullyConnected(h, num_neurons=4, has_bias=True, name="last")
        loss = lbann.MeanSquaredError(y, target)
        model = lbann.Model(1, layers=lbann.traverse_layer_graph(x), objective_function=loss)
        exp = lbann.proto.serialize.build_experiment(
            trainer=lbann.Trainer(mini_batch_size=8, random_seed=3), model=model,
            data_reader=_reader(8, [24], "samples:normal responses:normal", response_dims=[4]),
            optimizer=lbann.SGD(learn_rate=1e-3, momentum=0.9))
        tr = ExecTrainer(exp)
        m = tr.build_model(exp.model)
        m.weights_by_name["aside_linearity_weights"].gradient.fill_(3.0)
        g = torch.Generator(device="cuda").manual_seed(1)
        outs = []
        for step in range(6):
            rows = 8 if step != 5 else 5
            batch = {"samples": torch.randn(rows, 24, generator=g, device="cuda"),
                     "responses": torch.randn(rows, 4, generator=g, device="cuda")}
            m.train_step(batch, rows)
            # (detached: a copy that remembers the weights keeps the step from being captured)
            outs += [t.detach().clone() for w in m.weights for t in (w.gradient, w.values)]
            assert not m.weights_by_name["aside_linearity_weights"].gradient.any()
        names = {id(w.handle): w.name for w in m.weights}
        found = {names[id(h)] for h in m._overwritten_gradients()}
        assert not graph or any("graph" in e for e in m._graphs.values())
        tr.shutdown()
        assert native.consume_status() == 0
        return outs, found

    want, none = run(1 << 40)
    got, found = run(1)
    assert not none and found == {"first_linearity_weights", "aside_linearity_weights", "last_linearity_weights"}
    for a, b in zip(want, got):
        assert torch.isfinite(a).all() and torch.equal(a, b)


def test_evaluation_replays_equal_eager_steps():
    """Evaluation steps as graphs: losses and activations of several steps are held and compared at the end (a
    replay must not write over what a caller holds), weights and running statistics change in between, a ragged
    last mini-batch has a graph of its own, and the statistics add up."""
    def run(graph):
        o = opts.reset()
        o.set("default_dtype", "bf16")
        o.set("use_cuda_graph", graph)
        x = lbann.Input(data_field="samples")
        target = lbann.Input(data_field="responses")
        h = lbann.Reshape(x, dims=[8, 6, 6])
        h = lbann.Convolution(h, num_dims=2, out_channels=16, kernel_size=3, padding=1, has_bias=False, name="conv")
        h = lbann.Relu(lbann.BatchNormalization(h))
        h = lbann.FullyConnected(h, num_neurons=4, has_bias=True, name="last_product")
        shift = lbann.WeightsLayer(dims=[4], weights=[lbann.Weights(initializer=lbann.ConstantInitializer(value=0.1))])
        h = lbann.Add(h, shift, name="last")       # an activation that is a view of the weights
        loss = lbann.MeanSquaredError(h, target, name="mse")
        model = lbann.Model(1, layers=lbann.traverse_layer_graph(x), objective_function=loss,
                            metrics=[lbann.Metric(loss, name="mse")])
        exp = lbann.proto.serialize.build_experiment(
            trainer=lbann.Trainer(mini_batch_size=8, random_seed=3), model=model,
            data_reader=_reader(8, [288], "samples:normal responses:normal", response_dims=[4]),
            optimizer=lbann.SGD(learn_rate=1e-2, momentum=0.9))
        tr = ExecTrainer(exp)
        m = tr.build_model(exp.model)
        g = torch.Generator(device="cuda").manual_seed(1)
        losses, outs, held = [], [], []
        for step in range(30):
            rows = 5 if step % 5 == 4 else 8
            batch = {"samples": torch.randn(rows, 288, generator=g, device="cuda"),
                     "responses": torch.randn(rows, 4, generator=g, device="cuda")}
            if step % 4 == 1:
                m.train_step(batch, rows)
            losses.append(m.evaluate_step(batch, "validation" if step % 3 else "testing", rows))
            # held for good, as it is and by the step's mapping; later for the next step only
            outs.append(m.activation("last") if step < 16 else m.activation("last").clone())
            last = m.activation("conv")[1:]
            if step < 16:
                held.append(m.acts)
            assert m.current_mini_batch_size == rows and m.current_inputs["samples"] is batch["samples"]
        held = [a["conv"][0] for a in held]
        stats = [m.reduce_statistics(mode) for mode in ("validation", "testing")]
        graphs = sum(e["graph"] is not None for e in m._eval_graphs.values())
        assert last.shape[0] == rows - 1
        tr.shutdown()
        assert native.consume_status() == 0
        return losses, outs, held, stats, graphs

    want, got = run(False), run(True)
    assert want[4] == 0 and got[4] >= 3        # of four signatures
    for a, b in zip(want[:3], got[:3]):
        for t, u in zip(a, b):
            assert torch.equal(t, u)
    assert want[3] == got[3]


def _switching_model(graph):
    """A model with an activation that a mutation replaces and a loss term that freezing switches off."""
    o = opts.reset()
    o.set("default_dtype", "bf16")
    o.set("use_cuda_graph", graph)
    x = lbann.Input(data_field="samples")
    target = lbann.Input(data_field="responses")
    h = lbann.FullyConnected(x, num_neurons=24, has_bias=True, name="first")
    h = lbann.Relu(lbann.Identity(h), name="act")
    y = lbann.FullyConnected(h, num_neurons=4, has_bias=True, name="last")
    terms = [lbann.IdentityZero(lbann.MeanSquaredError(y, target), name="switch"),
             lbann.IdentityZero(lbann.MeanAbsoluteError(y, target), name="other")]
    model = lbann.Model(1, layers=lbann.traverse_layer_graph(x), objective_function=lbann.ObjectiveFunction(terms))
    exp = lbann.proto.serialize.build_experiment(
        trainer=lbann.Trainer(mini_batch_size=8, random_seed=3), model=model,
        data_reader=_reader(8, [24], "samples:normal responses:normal", response_dims=[4]),
        optimizer=lbann.SGD(learn_rate=1e-2, momentum=0.9))
    tr = ExecTrainer(exp)
    return tr, tr.build_model(exp.model)


@pytest.mark.parametrize("training", [False, True])
@pytest.mark.parametrize("change", ["mutation", "params", "phases"])
def test_replays_follow_changes_of_the_layers(change, training):
    """A layer changes between steps, after they have been captured: replayed steps equal ordinary ones.  A
    mutation replaces an activation, a parameter is set in place, a callback freezes one loss and then the other."""
    from lbann_b200.exec.ltfb import Mutation

    def run(graph):
        tr, m = _switching_model(graph)
        assert not getattr(m.layer("act"), "fused_into_parent", False)
        mutation = Mutation("replace_activation", seed=1)
        g = torch.Generator(device="cuda").manual_seed(1)
        losses, types = [], set()
        for step in range(38):
            batch = {"samples": torch.randn(8, 24, generator=g, device="cuda"),
                     "responses": torch.randn(8, 4, generator=g, device="cuda")}
            if change == "mutation" and step % 8 == 7:
                mutation.mutate(m, step)
            elif change == "params" and step % 8 == 7:
                while m.layer("act").type != "leaky_relu":
                    mutation.mutate(m, step)
                m.layer("act").params.negative_slope = 0.1 * step
            elif change == "phases":
                for name, on in (("switch", step // 4 % 2), ("other", 1 - step // 4 % 2)):
                    m.layer(name).frozen = bool(on)
            types.add(m.layer("act").type)
            if training:
                losses.append(m.train_step(batch, 8).clone())
            else:
                losses.append(m.evaluate_step(batch, "validation", 8).clone())
        entries = m._graphs if training else m._eval_graphs
        captured = sum("graph" in e if training else e["graph"] is not None for e in entries.values())
        tr.shutdown()
        assert native.consume_status() == 0
        return torch.stack(losses), captured, types

    want, none, _ = run(False)
    got, captured, types = run(True)
    assert not none and captured == (2 if change == "phases" else 1)
    assert change == "phases" or len(types) > 1
    assert torch.equal(want, got), (want - got).abs()


@pytest.mark.parametrize("where", ["main", "side", "mapping"])
def test_activations_of_replays_may_be_read_on_other_streams(where):
    """What a replayed evaluation step hands out obeys the allocator's rules: read late on another stream (asked for
    here, there, or through the step's mapping), marked with record_stream and dropped, while the next step runs."""
    tr, m = _switching_model(True)
    side = torch.cuda.Stream()
    g = torch.Generator(device="cuda").manual_seed(1)
    batches = [{"samples": torch.randn(8, 24, generator=g, device="cuda"),
                "responses": torch.randn(8, 4, generator=g, device="cuda")} for _ in range(10)]
    want, got = [], []
    for b in batches:
        m._evaluate_step_eager(b, "testing", 8, 0)
        want.append(m.activation("last").clone())
    for b in batches:
        m.evaluate_step(b, "validation", 8)
        main = torch.cuda.current_stream()
        y = m.activation("last") if where == "main" else m.acts if where == "mapping" else None
        side.wait_stream(main)
        with torch.cuda.stream(side):
            torch.cuda._sleep(20_000_000)            # the next step starts meanwhile
            if where != "main":
                y = (y["last"][0] if where == "mapping" else m.activation("last"))
            got.append(y * 1)
        y.record_stream(side)
        del y
    torch.cuda.synchronize()
    assert m._eval_graphs
    tr.shutdown()
    assert native.consume_status() == 0
    for a, b in zip(want, got):
        assert torch.equal(a, b)


def test_evaluation_whose_activations_are_kept_is_replayed():
    """A list of all steps' logits: every step beyond the first four is a replay, none writes over what is kept."""
    tr, m = _switching_model(True)
    g = torch.Generator(device="cuda").manual_seed(1)
    kept, want, ordinary, eager = [], [], 0, m._evaluate_step_eager

    def counted(*args):
        nonlocal ordinary
        ordinary += 1
        return eager(*args)

    for step in range(50):
        b = {"samples": torch.randn(8, 24, generator=g, device="cuda"),
             "responses": torch.randn(8, 4, generator=g, device="cuda")}
        eager(b, "testing", 8, 0)
        want.append(m.activation("last").clone())
        m._evaluate_step_eager = counted
        m.evaluate_step(b, "validation", 8)
        m._evaluate_step_eager = eager
        kept.append(m.activation("last"))
    assert ordinary == 4                  # three and the capture
    tr.shutdown()
    assert native.consume_status() == 0
    for a, b in zip(want, kept):
        assert torch.equal(a, b)


def test_capture_of_an_evaluation_step_leaves_the_allocator_alone():
    """Blocks that the allocator keeps are still there after a capture."""
    tr, m = _switching_model(True)
    block = torch.empty(64 << 20, device="cuda")
    del block
    frees = torch.cuda.memory_stats()["num_device_free"]
    batch = {"samples": torch.ones(8, 24, device="cuda"), "responses": torch.ones(8, 4, device="cuda")}
    losses = [float(m.evaluate_step(batch, "validation", 8)) for _ in range(6)]
    assert any(e["graph"] is not None for e in m._eval_graphs.values())
    assert torch.cuda.memory_stats()["num_device_free"] == frees
    tr.shutdown()
    assert native.consume_status() == 0 and len(set(losses)) == 1


def test_evaluation_steps_that_cannot_be_captured(capsys):
    tr, m = _switching_model(True)
    eager = m._evaluate_step_eager

    def step(*args):
        out = eager(*args)
        if torch.cuda.is_current_stream_capturing():
            raise RuntimeError("not this one")
        return out

    m._evaluate_step_eager = step
    batch = {"samples": torch.ones(8, 24, device="cuda"), "responses": torch.ones(8, 4, device="cuda")}
    losses = [float(m.evaluate_step(batch, "validation", 8)) for _ in range(6)]
    tr.shutdown()
    assert len(set(losses)) == 1 and m.stats["validation"].samples == 48 and native.consume_status() == 0
    assert capsys.readouterr().out.count("not this one") == 1


@pytest.mark.parametrize("training", [False, True])
def test_memory_freed_while_a_step_is_captured(training):
    """Pinned memory that any stream of PyTorch's pool has read may be freed, and reference cycles come apart, during
    a capture: neither becomes part of it, and both allocators work behind it."""
    import gc
    tr, m = _switching_model(True)
    pinned, seen = [], []
    for _ in range(64):
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            pinned.append(torch.zeros(1 << 20).pin_memory())
            pinned[-1].to("cuda", non_blocking=True)
    name = "_train_step_eager" if training else "_evaluate_step_eager"
    eager = getattr(m, name)

    def step(*args):
        if torch.cuda.is_current_stream_capturing():
            seen.append(gc.isenabled())
            pinned.clear()
        return eager(*args)

    setattr(m, name, step)
    batch = {"samples": torch.ones(8, 24, device="cuda"), "responses": torch.ones(8, 4, device="cuda")}
    losses = [float(m.train_step(batch, 8) if training else m.evaluate_step(batch, "validation", 8)) for _ in range(6)]
    again = [torch.zeros(1 << 20).pin_memory() for _ in range(64)]
    assert seen == [False] and gc.isenabled() and len(again) == 64 and all(math.isfinite(v) for v in losses)
    assert any(e.get("graph") is not None for e in (m._graphs if training else m._eval_graphs).values())
    tr.shutdown()
    assert native.consume_status() == 0


def test_which_evaluation_steps_keep_a_graph(monkeypatch):
    """Limits of the captured evaluation steps: of their number, with and without an idle one to drop, of memory, of
    what a replay would copy, of activations a layer, and of the signatures that are remembered."""
    from lbann_b200.exec.model import ExecModel
    tr, m = _switching_model(True)

    def steps(rows, n=5):
        for _ in range(n):
            m.evaluate_step({"samples": torch.ones(rows, 24, device="cuda"),
                             "responses": torch.ones(rows, 4, device="cuda")}, "validation", rows)
        return {k[6][0][1][0] for k, e in m._eval_graphs.items() if e["graph"] is not None}

    monkeypatch.setattr(ExecModel, "_EVAL_GRAPHS", 2)
    monkeypatch.setattr(ExecModel, "_EVAL_IDLE", 12)
    monkeypatch.setattr(ExecModel, "_EVAL_SIGNATURES", 5)
    assert steps(1) == {1} and steps(2) == {1, 2}
    assert steps(3) == {1, 2}                         # neither has been idle for long
    assert steps(2) == {1, 2} and steps(3) == {2, 3}  # the first has
    limits = (("_EVAL_LAYER_BYTES", 1), ("_EVAL_GRAPH_BYTES", 1), ("_EVAL_GRAPH_CASTS", -1))
    for rows, (limit, value) in enumerate(limits, 4):
        with monkeypatch.context() as mp:
            mp.setattr(ExecModel, limit, value)
            assert steps(rows, 20) == {2, 3}          # idle or not: nothing makes room for what gets no graph
        assert len(m._eval_refused) == rows - 3
    for rows in range(7, 15):
        steps(rows, 1)
    assert len(m._eval_graphs) == 5 and steps(3) == {2, 3}
    held = sum(e["graph"].bytes for e in m._eval_graphs.values() if e["graph"] is not None)
    assert (2 + 3) * (24 + 4) * 4 <= held <= ExecModel._EVAL_GRAPH_BYTES
    tr.shutdown()
    assert native.consume_status() == 0


def test_first_step_with_loss_scaling_imports_nothing_large():
    """A training step with AMP in a process of its own; errors of Python functions in backward keep their type."""
    code = """
import sys, torch
import lbann_b200 as lbann
from lbann_b200.exec.trainer import ExecTrainer
from lbann_b200.models.cosmoflow import construct_cosmoflow_model, synthetic_reader
from lbann_b200.ops import native
from lbann_b200.utils import options as opts
opts.reset().set("default_dtype", "fp16")
model = construct_cosmoflow_model(16, 4, 4, num_epochs=1, channels=(16, 32), pool_mode="max", conv_bias=False)
model.amp = lbann.AmpOptions(enabled=True, init_scale=128.0)
exp = lbann.proto.serialize.build_experiment(trainer=lbann.Trainer(mini_batch_size=2, random_seed=1), model=model,
    data_reader=lbann.reader_pb2.DataReader(), optimizer=lbann.Adam(learn_rate=1e-4, beta1=0.9, beta2=0.99, eps=1e-8))
import numpy as np
from lbann_b200.data.readers import ArrayReader
arrays = {"samples": np.zeros((1, 4, 16, 16, 16), np.float32), "responses": np.zeros((1, 4), np.float32)}
m = ExecTrainer(exp, readers={"train": ArrayReader(arrays)}, background_io=False).build_model(exp.model)
before = "sympy" in sys.modules
m.train_step({"samples": torch.rand(2, 4, 16, 16, 16, device="cuda").half(), "responses": torch.rand(2, 4, device="cuda")})
assert ("sympy" in sys.modules) == before, "sympy came in"
assert native.consume_status() == 0 and any(w.gradient.any() for w in m.weights)
class Bad(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x):
        return x * 2
    @staticmethod
    def backward(ctx, g):
        raise KeyError("mine")
x = torch.ones((), device="cuda", requires_grad=True)
try:
    native.nodes().backward(Bad.apply(x), torch.ones((), device="cuda"))
except KeyError as e:
    assert "mine" in str(e)
else:
    raise AssertionError("no error")
"""
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300,
                       cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
    assert r.returncode == 0, r.stderr[-2000:]
