"""train.py on one GPU: both sharding back ends, CPU offload (FSDP2 only), activation checkpointing."""
import pytest

from mp_util import run_ranks

pytestmark = pytest.mark.gpu


def _train(rank, world, extra, loss_log):
    import train

    train.main(["--synthetic", "--model-shape", "small", "--device", "cuda", "-b", "1", "-s", "512", "--lr", "1e-4",
                "--log-freq", "2", "--num-samples", "4", "--steps", "6", "--loss-log", loss_log] + extra)


def _losses(path):
    return [float(l.split()[1]) for l in open(path).read().split("\n") if l]


def test_flat_and_fsdp2_back_ends_train_on_one_gpu(tmp_path):
    logs = {k: str(tmp_path / f"{k}.log") for k in ("flat", "flat_ckpt", "fsdp2")}
    run_ranks(_train, 1, init_pg=False, backend="nccl", args=(["-q", "--zip-ccl", "--compress-rs"], logs["flat"]))
    run_ranks(_train, 1, init_pg=False, backend="nccl", args=(["--act-ckpt"], logs["flat_ckpt"]))
    run_ranks(_train, 1, init_pg=False, backend="nccl", args=(["--sharding", "fsdp2", "-q", "--zip-ccl"], logs["fsdp2"]))
    a, b, c = (_losses(logs[k]) for k in ("flat", "flat_ckpt", "fsdp2"))
    assert len(a) == len(b) == len(c) == 6
    assert a[-1] < a[0] and c[-1] < c[0]       # four samples, repeated: the loss falls
    assert a == b                              # recomputation is exact
    assert abs(a[0] - c[0]) < 0.2              # same shape, different initial values


def test_cpu_offload_runs_through_fsdp2(tmp_path):
    """``--cpu-offload`` (reference: train.py:95, 125, 261) keeps parameters, gradients and optimizer
    state on the host; it selects the FSDP2 back end."""
    log = str(tmp_path / "off.log")
    run_ranks(_train, 1, init_pg=False, backend="nccl", args=(["--cpu-offload", "--model-shape", "tiny"], log))
    ls = _losses(log)
    assert len(ls) == 6 and all(l == l for l in ls)


def _graph_worker(rank, world, family):
    import dataclasses

    import torch

    from fsdp_comm_opt_b200.engine import EngineConfig, TrainEngine
    from fsdp_comm_opt_b200.models import get_config

    cfg = dataclasses.replace(get_config("gpt2-tiny" if family == "gpt2" else "tiny"), vocab_size=1001 if family == "gpt2" else 8192)
    dev = torch.device("cuda", 0)

    def build(graphs):
        return TrainEngine(EngineConfig(model=cfg, lr=1e-3, seed=3, step_graphs=graphs, act_ckpt=family == "ckpt"), dev)

    a, b = build(True), build(False)
    g = torch.Generator().manual_seed(1)
    for i in range(14):
        s = (96, 130, 64)[i % 3] if i > 4 else 96                       # several recorded shapes, one of them odd-sized
        ids = torch.randint(0, cfg.vocab_size, (2, s), generator=g).pin_memory()
        if i % 4 == 3:
            la, lb = a.step_on_device(ids.to(dev)).item(), b.step_on_device(ids.to(dev)).item()
        else:
            la, lb = a.step(ids), b.step(ids)
        assert abs(la - lb) < 2e-3 * abs(lb), (i, la, lb)               # dQ is summed in any order
    assert a._graphs._recorded and b._graphs is None
    d = (a.flat.master.float() - b.flat.master.float()).norm() / b.flat.master.float().norm()
    assert d < 5e-3
    # a hook that was not there when the step was recorded is called: such a step runs eagerly
    calls = []
    h = next(m for m in a.model.modules() if type(m).__name__ in ("Linear", "BiasLinear")).register_forward_hook(
        lambda *x: calls.append(1))
    a.step(ids)
    assert calls
    h.remove()
    a.step(ids)
    assert len(calls) in (1, 2)                                         # twice with recomputation
    torch.cuda.synchronize()


@pytest.mark.parametrize("family", ["llama", "gpt2", "ckpt"])
def test_replayed_steps_equal_eager_steps(family):
    run_ranks(_graph_worker, 1, backend="nccl", args=(family,))


def _fp32_master_worker(rank, world, family):
    import torch

    from fsdp_comm_opt_b200.engine import EngineConfig, TrainEngine

    model, dev = "gpt2-tiny" if family == "gpt2" else "tiny", torch.device("cuda", 0)
    a, b = (TrainEngine(EngineConfig(model=model, lr=1e-3, seed=3, step_graphs=g, master_dtype=torch.float32), dev) for g in (True, False))
    ids = torch.randint(0, a.model_config.vocab_size, (2, 96), generator=torch.Generator().manual_seed(1)).pin_memory()
    losses = []
    for _ in range(8):
        la, lb = a.step(ids), b.step(ids)
        assert abs(la - lb) < 2e-3 * abs(lb), (la, lb)                  # dQ is summed in any order
        losses.append(la)
    assert a._graphs._recorded and losses[-1] < losses[0]
    assert a.flat.master.dtype == a.flat.grad_master.dtype == torch.float32
    assert all(torch.equal(g.grad_shard, g.grad_shard_c.float()) and g.grad_shard.any() for g in a.flat.groups)
    d = (a.flat.master - b.flat.master).norm() / b.flat.master.norm()
    assert d < 5e-3


@pytest.mark.parametrize("family", ["llama", "gpt2"])
def test_fp32_master_weights_on_one_gpu(family):
    run_ranks(_fp32_master_worker, 1, backend="nccl", args=(family,))


def _finished_worker(rank, world, graphs):
    import dataclasses

    import torch

    from fsdp_comm_opt_b200.engine import EngineConfig, TrainEngine
    from fsdp_comm_opt_b200.models import get_config

    # 2.6e8 table elements: the update takes about 0.6 ms, far longer than the way from the loss to the caller
    cfg = dataclasses.replace(get_config("tiny"), vocab_size=512_000)
    eng = TrainEngine(EngineConfig(model=cfg, seed=3, step_graphs=graphs), torch.device("cuda", 0))
    ids = torch.randint(0, cfg.vocab_size, (1, 64)).pin_memory()
    for _ in range(5):
        eng.step(ids)
        assert torch.cuda.current_stream().query()


@pytest.mark.parametrize("graphs", [True, False])
def test_a_step_has_finished_when_it_returns(graphs):
    """Parameters and moments may be read from another stream as soon as ``step`` is back."""
    run_ranks(_finished_worker, 1, backend="nccl", args=(graphs,))


def _engines(family="llama", act_ckpt=False, **changes):
    """The same small model with and without recorded steps."""
    import dataclasses

    import torch

    from fsdp_comm_opt_b200.engine import EngineConfig, TrainEngine
    from fsdp_comm_opt_b200.models import get_config

    cfg = dataclasses.replace(get_config("gpt2-tiny" if family == "gpt2" else "tiny"), vocab_size=1024, **changes)
    dev = torch.device("cuda", 0)
    return [TrainEngine(EngineConfig(model=cfg, lr=1e-3, seed=3, step_graphs=g, act_ckpt=act_ckpt), dev) for g in (True, False)]


def _same_steps(a, b, shapes, seed=1):
    import torch

    g = torch.Generator().manual_seed(seed)
    for i, shape in enumerate(shapes):
        ids = torch.randint(0, a.model_config.vocab_size, shape, generator=g).pin_memory()
        la, lb = a.step(ids), b.step(ids)
        assert abs(la - lb) < 2e-3 * abs(lb), (i, shape, la, lb)        # dQ is summed in any order


def _many_lengths_worker(rank, world):
    import torch

    from fsdp_comm_opt_b200.ops import rope

    a, b = _engines()
    # a long shape is recorded; a short one is seen twice; so many other lengths that the table cache is emptied; the
    # short one is recorded; the long one is replayed over whatever the short recording left in their common memory
    _same_steps(a, b, [(2, 512)] * 4 + [(2, 96)] * 2 + [(1, 101 + 3 * i) for i in range(18)] + [(2, 96), (2, 512)])
    assert len(a._graphs._recorded) == 2 and any(key[0] == 96 for key in rope._TABLES)
    segments = torch.cuda.memory_snapshot()
    for (seq, dim, theta, dev), tables in rope._TABLES.items():
        for t, r in zip(tables, rope.rope_tables(seq, dim, theta, dev)):
            (segment,) = [s for s in segments if 0 <= t.data_ptr() - s["address"] < s["total_size"]]
            assert segment["segment_pool_id"] == (0, 0), f"the table of {seq} lies in the graphs' memory"
            assert torch.equal(t, r), seq
    _same_steps(a, b, [(1, 96), (2, 96), (1, 512)])                     # eager and replayed readers of the tables
    # twenty lengths with two batch sizes, each often enough to be recorded
    _same_steps(a, b, [(1 + i % 2, 64 + 8 * (i // 2 % 20)) for i in range(160)])


def test_steps_of_many_lengths_equal_eager_steps():
    run_ranks(_many_lengths_worker, 1, backend="nccl")


def _many_shapes_worker(rank, world):
    from fsdp_comm_opt_b200.parallel.step_graph import StepGraphs

    StepGraphs.MAX_SHAPES, StepGraphs.IDLE_STEPS = 4, 40
    recorded, record = [], StepGraphs._record

    def counted(self, shape, *rest):
        recorded.append(shape)
        return record(self, shape, *rest)

    StepGraphs._record = counted
    a, b = _engines()
    _same_steps(a, b, [(1, 64 + 16 * (i % 6)) for i in range(48)])      # six shapes in turn, room for four
    assert recorded == [(1, 64 + 16 * i) for i in range(4)]
    _same_steps(a, b, [(2, 64 + 16 * (i % 2)) for i in range(45)])      # two others replace those that went idle
    assert recorded[4:] == [(2, 64), (2, 80)] and set(recorded[4:]) < set(a._graphs._recorded)


def test_more_shapes_than_are_kept_do_not_record_at_every_step():
    run_ranks(_many_shapes_worker, 1, backend="nccl")


def _key_change_worker(rank, world):
    from fsdp_comm_opt_b200.ops import gemm

    a, b = _engines()
    shape = (2, 96)
    for change in (lambda e: None, lambda e: setattr(e.model, "activation_checkpointing", True), lambda e: e.model.eval(),
                   lambda e: gemm.set_backend("cublas")):
        change(a), change(b)
        graph = next((r.graph for r in a._graphs._recorded.values()), None)
        _same_steps(a, b, [shape] * 4)
        assert a._graphs._recorded[shape].graph is not graph


def test_the_only_recorded_shape_is_recorded_again_when_an_option_changes():
    run_ranks(_key_change_worker, 1, backend="nccl")


def _little_memory_worker(rank, world):
    import torch

    a, b = _engines()
    # 4 GB that the allocator has cached and, as the driver is made to say here, little else
    torch.empty(1 << 32, dtype=torch.uint8, device="cuda")
    info = torch.cuda.mem_get_info
    torch.cuda.mem_get_info = lambda *x: (64 << 20, info(*x)[1])
    _same_steps(a, b, [(2, 512)] * 4)
    assert not a._graphs._recorded


def test_cached_blocks_of_the_allocator_are_no_room_for_a_recording():
    run_ranks(_little_memory_worker, 1, backend="nccl")


def _failed_recording_worker(rank, world, where):
    import warnings

    import torch

    from fsdp_comm_opt_b200.ops import swiglu
    from fsdp_comm_opt_b200.parallel.step_graph import StepGraphs

    attempts, record = [], StepGraphs._record
    StepGraphs._record = lambda self, *x: (attempts.append(x), record(self, *x))[1]
    a, b = _engines()

    def out_of_memory(*x):
        if torch.cuda.is_current_stream_capturing():
            raise torch.OutOfMemoryError("no block for the recording")

    if where == "forward":
        call = swiglu.swiglu
        swiglu.swiglu = lambda x: (out_of_memory(x), call(x))[1]
    else:                                                               # half of the gradients are in place by then
        pre = a.flat._pre_backward
        a.flat._pre_backward = lambda g: (out_of_memory(g) if g.name == "layers.0" else None, pre(g))[1]
    with warnings.catch_warnings(record=True) as caught:
        warnings.simplefilter("always")
        _same_steps(a, b, [(2, 96)] * 4 + [(2, 64)] * 4)
    assert len(attempts) == 1 and not a._graphs._recorded
    assert sum("no block for the recording" in str(w.message) for w in caught) == 1
    assert all(p.grad is None for p in a.model.parameters())


@pytest.mark.parametrize("where", ["forward", "backward"])
def test_a_recording_that_fails_leaves_the_step_to_run_eagerly(where):
    run_ranks(_failed_recording_worker, 1, backend="nccl", args=(where,))


def _refusal_worker(rank, world):
    import torch

    a, b = _engines(n_layers=16)
    bytes_of = a._graphs._activation_bytes
    need = bytes_of(2 * 512)
    a.model.activation_checkpointing = True
    room = bytes_of(2 * 512)
    a.model.activation_checkpointing = False
    info = torch.cuda.mem_get_info
    torch.cuda.mem_get_info = lambda *x: (4 * (room + need), info(*x)[1])   # an eighth of it: between the two
    _same_steps(a, b, [(2, 512)] * 3)
    assert not a._graphs._recorded
    a.model.activation_checkpointing = b.model.activation_checkpointing = True
    _same_steps(a, b, [(2, 512)] * 3)
    assert len(a._graphs._recorded) == 1


def test_a_shape_that_was_too_large_is_recorded_once_it_fits():
    run_ranks(_refusal_worker, 1, backend="nccl")


def _guard_worker(rank, world):
    import torch

    from fsdp_comm_opt_b200.parallel.step_graph import StepGraphs

    StepGraphs.MAX_SHAPES = 1
    a, b = _engines()
    shape = (2, 96)
    replayed, run = [], StepGraphs.run
    StepGraphs.run = lambda self, ids: (replayed.append(run(self, ids)), replayed[-1])[1]

    def steps(eager):
        replayed.clear()
        _same_steps(a, b, [shape] * 2)
        assert all((r is None) == eager for r in replayed) and len(replayed) == 2

    _same_steps(a, b, [shape] * 3)
    steps(False)
    seen = []
    norm, head = a.model.model.norm, a.model.lm_head
    both = [(e.model.model.norm, e.model.lm_head) for e in (a, b)]

    def called(*x):
        seen.append(1)

    # what is called, packed or counted at every step has to be so while it is there, and only then
    for watch in (lambda: norm.weight.register_hook(called),
                  lambda: norm.weight.register_post_accumulate_grad_hook(called),
                  lambda: head.register_forward_hook(called),
                  lambda: torch.nn.modules.module.register_module_forward_hook(called)):
        handle = watch()
        seen.clear()
        steps(True)
        assert seen
        handle.remove()
        seen.clear()
        steps(False)
        assert not seen
    with torch.autograd.graph.saved_tensors_hooks(lambda t: (called(), t)[1], lambda t: t):
        steps(True)
    assert seen
    # a hook in the place of another
    hooks = next(m._forward_hooks for m in a.model.modules() if m._forward_hooks)
    key, old = next(iter(hooks.items()))
    del hooks[key]
    hooks[key + 100_000] = old
    steps(True)
    del hooks[key + 100_000]
    hooks[key] = old
    steps(False)
    # other parts in the place of the model's own
    for n, h in both:
        n.eps = 0.5
    steps(True)
    for n, h in both:
        n.eps = a.model_config.norm_eps
        n.weight.data = n.weight.data.clone()
    steps(True)
    for n, h in both:
        e = a if n is norm else b
        g = e.flat.groups[-1]
        e.flat._replace_param_storage(g, g.full)
        own = h.forward
        h.forward = lambda x, own=own: own(x) * 0.5
    steps(True)
    for n, h in both:
        del h.forward
    steps(False)
    theta = a.model_config.rope_theta
    a.model_config.rope_theta = theta / 100                             # both engines' own configuration object
    steps(True)
    a.model_config.rope_theta = theta
    steps(False)
    for e in (a, b):
        e.model.model.layers[1] = torch.nn.Identity()                   # x alone: unpacking it as (x, delta) would fail
        e.model.model.layers[1].forward = lambda x, delta: (x, delta)
    steps(True)


def test_steps_with_hooks_modes_or_replaced_parts_run_eagerly():
    run_ranks(_guard_worker, 1, backend="nccl")
