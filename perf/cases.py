"""Timed cases: what a program that uses this library has it do.

Every case goes through the public entry points: a network that is built from
its description, run for a number of timesteps with ``Network.run`` and read
back with ``get_neuron_data`` / ``get_weight_matrix``; a ``Batch`` of instances;
a ``RateNetwork`` training step.  Sizes are those of this repository's
benchmark and configurations, and ragged ones of the same kinds.

Kinds (``case["kind"]``):

* ``encoding``   a feedforward net of rate_encoding layers in a loop with the
  program: a callback feeds a frame and another reads the answer every step;
* ``recurrent``  a rate_encoding layer with dense recurrent weights, driven
  through a 5x5 field;
* ``izhikevich`` relay -> Izhikevich, 5x5 field and dense inhibition, no
  learning (the 32x32 configuration's topology);
* ``plastic``    three Izhikevich layers, a learning 9x9 projection, stride-2
  divergent, one-to-one and subset connections (the 256x256 configuration's);
* ``spnet``      spnet layers with sparse, learning connections;
* ``life``       game_of_life boards;
* ``batch``      many uneven Izhikevich instances in one ``Batch``;
* ``adjoint``    loss and gradients of the differentiable rate network.
"""
import math

import numpy as np
import torch

from synaptogenesis_gb300 import batching
from synaptogenesis_gb300 import syngen as sg

sg.set_suppress_output(False)
sg.set_warnings(False)


# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # the smallest call: a small classifier stepped inside a program's own
        # loop, one frame in and ten values out per step
        {"name": "encoding 784-500-10", "kind": "encoding", "rows": 28, "cols": 28, "hidden": 500,
         "outputs": 10, "steps": 100},
        # a dense layer of the size where weights no longer fit a small cache
        {"name": "recurrent 64x64", "kind": "recurrent", "rows": 64, "cols": 64, "steps": 200},
        # the plain 32x32 configuration, at its stated length
        {"name": "izhikevich 32x32", "kind": "izhikevich", "rows": 32, "cols": 32, "steps": 1000},
        # a small experiment of odd sizes that learns on every kind of matrix
        {"name": "plastic 61x97", "kind": "plastic", "rows": 61, "cols": 97, "field": 7,
         "window": 21, "learn_window": True, "steps": 300},
        # the large plastic configuration, at its stated length
        {"name": "plastic 256x256", "kind": "plastic", "rows": 256, "cols": 256, "field": 9,
         "window": 64, "learn_window": False, "steps": 1000},
        # polychronisation network, sparse, learning
        {"name": "spnet 256x256", "kind": "spnet", "rows": 256, "cols": 256, "field": 15,
         "steps": 300},
        # the large board, at its stated length
        {"name": "life 2048x2048", "kind": "life", "rows": 2048, "cols": 2048, "steps": 10000},
        # a board of no particular size
        {"name": "life 500x333", "kind": "life", "rows": 500, "cols": 333, "steps": 1000},
        # a few small instances: a parameter sweep while working interactively
        {"name": "batch 12", "kind": "batch", "count": 12, "smin": 16, "smax": 48, "tile_rows": 4,
         "tile_colblocks": 2, "steps": 100},
        # a sweep that fills the GPU
        {"name": "batch 64", "kind": "batch", "count": 64, "smin": 16, "smax": 128, "tile_rows": 2,
         "tile_colblocks": 4, "steps": 100},
        # the differentiable configuration: a whole training step
        {"name": "adjoint 3x64x64", "kind": "adjoint", "layers": 3, "rows": 64, "cols": 64,
         "field": 5, "outputs": 10, "batch": 64, "steps": 100, "checkpoint": 10,
         "input_grad": True},
        # odd sizes; parameters are trained, the input is data
        {"name": "adjoint 4x30x45", "kind": "adjoint", "layers": 4, "rows": 30, "cols": 45,
         "field": 3, "outputs": 7, "batch": 5, "steps": 37, "checkpoint": 8,
         "input_grad": False},
    ]


def _log(rng, lo, hi):
    """An integer in [lo, hi], spread over its logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["encoding", "recurrent", "izhikevich", "plastic", "spnet", "life", "batch",
                       "adjoint"])
    if kind == "encoding":
        return {"kind": kind, "rows": _log(rng, 8, 64), "cols": _log(rng, 8, 64),
                "hidden": _log(rng, 32, 2048), "outputs": _log(rng, 2, 100),
                "steps": _log(rng, 50, 200)}
    if kind == "recurrent":
        return {"kind": kind, "rows": _log(rng, 12, 64), "cols": _log(rng, 12, 64),
                "steps": _log(rng, 50, 200)}
    if kind == "izhikevich":
        return {"kind": kind, "rows": _log(rng, 8, 64), "cols": _log(rng, 8, 64),
                "steps": _log(rng, 100, 1000)}
    if kind == "plastic":
        rows, cols = _log(rng, 24, 192), _log(rng, 24, 192)
        return {"kind": kind, "rows": rows, "cols": cols, "field": rng.choice([3, 5, 7, 9, 11]),
                "window": _log(rng, 8, min(rows, cols, 64)), "learn_window": rng.random() < 0.5,
                "steps": _log(rng, 50, 300)}
    if kind == "spnet":
        return {"kind": kind, "rows": 2 * _log(rng, 16, 112), "cols": 2 * _log(rng, 16, 112),
                "field": rng.choice([5, 9, 15]), "steps": _log(rng, 50, 300)}
    if kind == "life":
        return {"kind": kind, "rows": _log(rng, 32, 1500), "cols": _log(rng, 32, 1500),
                "steps": _log(rng, 200, 2000)}
    if kind == "batch":
        rows, colblocks = rng.choice([(1, 4), (2, 2), (4, 1), (2, 4), (4, 2), (8, 1)])
        return {"kind": kind, "count": _log(rng, 4, 48), "smin": 16, "smax": _log(rng, 24, 112),
                "tile_rows": rows, "tile_colblocks": colblocks, "steps": _log(rng, 32, 100)}
    steps = _log(rng, 10, 100)
    return {"kind": kind, "layers": rng.choice([2, 3, 4]), "rows": _log(rng, 12, 72),
            "cols": _log(rng, 12, 72), "field": rng.choice([3, 5, 7]),
            "outputs": rng.randint(1, 16), "batch": _log(rng, 1, 64), "steps": steps,
            "checkpoint": _log(rng, 2, min(steps, 25)), "input_grad": rng.random() < 0.5}


# ---------------------------------------------------------------------------
# Networks
# ---------------------------------------------------------------------------
class _Net:
    """A built network and what a program keeps beside it."""

    def __init__(self, description, modules=(), **args):
        self.net = sg.Network(description)
        self.net.build_state()
        self.environment = sg.Environment({"modules": list(modules)})
        self.args = args
        self.extra = {}

    def run(self):
        report = self.net.run(self.environment, self.args)
        if report.obj is None:
            raise RuntimeError("run failed: " + sg.last_error())
        report.free()

    def neuron(self, layer, key):
        return self.net.get_neuron_data("s", layer, key).to_np_array()

    def matrix(self, connection, key="weights"):
        return self.net.get_weight_matrix(connection, key).to_np_array()

    def read(self, values):
        """The state's own buffer, kept alive by the array; words as int32."""
        if values.dtype == np.uint32:
            values = values.view(np.int32)
        kept = values.view(_Kept)
        kept.owner = self
        return kept

    def words(self, layer):
        return self.read(self.neuron(layer, "output").view(np.int32))

    def values(self, layer, key):
        return self.read(self.neuron(layer, key))

    def __del__(self):
        self.environment.free()
        self.net.free()


class _Kept(np.ndarray):
    owner = None


def _layer(name, model, rows, cols, **more):
    return dict({"name": name, "neural model": model, "rows": rows, "columns": cols}, **more)


def _connection(name, source, to, kind, **more):
    return dict({"name": name, "from layer": source, "to layer": to, "type": kind,
                 "plastic": False, "opcode": "add"}, **more)


def _network(layers, connections):
    return {"structures": [{"name": "s", "type": "parallel", "layers": layers}],
            "connections": connections}


def _field(size, **more):
    return dict({"field size": size, "wrap": True}, **more)


def _numbers(case, seed):
    """Every injected quantity of an encoding or recurrent net, from the seed."""
    rng = np.random.default_rng(seed)
    normal = lambda *shape: rng.standard_normal(shape, dtype=np.float32)   # noqa: E731
    n = case["rows"] * case["cols"]
    if case["kind"] == "encoding":
        hid, out = case["hidden"], case["outputs"]
        return {"w1": normal(hid, n) * np.float32(1.5 / math.sqrt(n)),
                "w2": normal(out, hid) * np.float32(1.5 / math.sqrt(hid)),
                "frames": rng.random((case["steps"], n), dtype=np.float32)}
    return {"w_rec": normal(n, n) * np.float32(1.0 / math.sqrt(n)),
            "w_in": rng.random((n, 25), dtype=np.float32) * np.float32(0.1)}


def _prepare_encoding(case, seed):
    numbers = _numbers(case, seed)
    frames, at = numbers["frames"], {"in": 0, "out": 0}
    answers = np.zeros((case["steps"], case["outputs"]), np.float32)

    def feed(_, values):
        values[:] = frames[at["in"] % len(frames)]
        at["in"] += 1

    def take(_, values):
        answers[at["out"] % len(answers)] = values
        at["out"] += 1

    tag = "perf encoding %d" % sg.make_callback_id("encoding")
    state = _Net(_network(
        [_layer("in", "relay", case["rows"], case["cols"]),
         _layer("hidden", "rate_encoding", 1, case["hidden"]),
         _layer("out", "rate_encoding", 1, case["outputs"])],
        [_connection("c1", "in", "hidden", "fully connected"),
         _connection("c2", "hidden", "out", "fully connected")]),
        [sg.make_custom_input_module("s", ["in"], tag + " in", feed),
         sg.make_custom_output_module("s", ["out"], tag + " out", take)],
        iterations=case["steps"])
    state.matrix("c1")[:] = numbers["w1"].reshape(-1)
    state.matrix("c2")[:] = numbers["w2"].reshape(-1)
    state.extra["answers"] = answers
    return state


def _run_encoding(state):
    state.run()
    return {"answers": state.extra["answers"].copy(),
            "hidden": state.read(state.neuron("hidden", "output").view(np.float32)),
            "input": state.values("hidden", "input")}


def _prepare_recurrent(case, seed):
    numbers = _numbers(case, seed)
    rows, cols = case["rows"], case["cols"]
    state = _Net(_network(
        [_layer("drive", "relay", rows, cols, **{"init config": {"type": "flat", "value": 1.0}}),
         _layer("rate", "rate_encoding", rows, cols)],
        [_connection("c_in", "drive", "rate", "convergent", **{"arborized config": _field(5)}),
         _connection("c_rec", "rate", "rate", "fully connected")]),
        iterations=case["steps"])
    state.matrix("c_in")[:] = numbers["w_in"].reshape(-1)
    state.matrix("c_rec")[:] = numbers["w_rec"].reshape(-1)
    return state


def _run_recurrent(state):
    state.run()
    return {"rate": state.read(state.neuron("rate", "output").view(np.float32)),
            "input": state.values("rate", "input")}


def _prepare_izhikevich(case, seed):
    rows, cols = case["rows"], case["cols"]
    sg.set_seed(seed)
    state = _Net(_network(
        [_layer("in", "relay", rows, cols, **{"init config": {
            "type": "poisson", "rate": 10, "value": 1.0, "seed": seed}}),
         _layer("iz", "izhikevich", rows, cols, params="regular")],
        [_connection("c_in", "in", "iz", "convergent", **{
            "random delay": 3, "arborized config": _field(5),
            "weight config": {"type": "random", "max weight": 0.5}}),
         _connection("c_rec", "iz", "iz", "fully connected", opcode="sub", **{
             "random delay": 3,
             "weight config": {"type": "random", "max weight": 0.2, "fraction": 0.2}})]),
        iterations=case["steps"], **{"learning flag": False})
    state.matrix("c_in", "short term w")[:] = 0.5
    return state


def _run_izhikevich(state):
    state.run()
    return {"words": state.words("iz"), "voltage": state.values("iz", "voltage"),
            "recovery": state.values("iz", "recovery"),
            "trace": state.read(state.matrix("c_rec", "long trace"))}


def _prepare_plastic(case, seed):
    rows, cols, k = case["rows"], case["cols"], case["window"]
    r0, c0 = (rows - k) // 2, (cols - k) // 2
    sg.set_seed(seed)
    layer = lambda name, **more: _layer(name, "izhikevich", rows, cols, params="regular", **more)  # noqa: E731
    random = lambda top: {"random delay": 3, "weight config": {"type": "random", "max weight": top}}  # noqa: E731
    state = _Net(_network(
        [layer("L1", **{"init config": {"type": "poisson", "rate": 5, "value": 20, "seed": seed}}),
         layer("L2"), layer("L3")],
        [_connection("c12", "L1", "L2", "convergent", **random(0.3), **{
            "plastic": True, "learning rate": 0.004, "arborized config": _field(case["field"])}),
         _connection("c23", "L2", "L3", "divergent", **random(0.3), **{
             "arborized config": {"field size": 3, "stride": 2}}),
         _connection("c31", "L3", "L1", "one to one", opcode="sub", **random(0.5)),
         _connection("c23s", "L2", "L3", "subset", **random(0.05), **{
             "plastic": case["learn_window"], "learning rate": 0.004,
             "subset config": {
                 "from row start": r0, "from row end": r0 + k, "from column start": c0,
                 "from column end": c0 + k, "to row start": r0, "to row end": r0 + k,
                 "to column start": c0, "to column end": c0 + k}})]),
        iterations=case["steps"], **{"learning flag": True})
    rng = np.random.default_rng(seed)
    for name in ("L1", "L2", "L3"):          # 80% regular, 20% fast spiking
        fast = rng.random(rows * cols) < 0.2
        state.neuron(name, "a")[fast] = 0.1
        state.neuron(name, "d")[fast] = 2.0
    for name in ("c12", "c23", "c31"):
        state.matrix(name, "short term w")[:] = 0.5
    return state


def _run_plastic(state):
    state.run()
    got = {"weights": state.read(state.matrix("c12")),
           "derivative": state.read(state.matrix("c12", "weight derivatives")),
           "window": state.read(state.matrix("c23s")),
           "trace": state.read(state.matrix("c23s", "long trace"))}
    for name in ("L1", "L2", "L3"):
        got[name + " words"] = state.words(name)
        got[name + " voltage"] = state.values(name, "voltage")
    return got


def _prepare_spnet(case, seed):
    rows, cols = case["rows"], case["cols"]
    sg.set_seed(seed)
    # the same synapses for every seed; their weights and the drive differ
    weights = lambda top, graph: {"sparse": True, "weight config": {  # noqa: E731
        "type": "random", "min weight": 0.01, "max weight": top, "fraction": 0.5, "seed": graph}}
    between = {"myelinated": True, "delay": 1, "arborized config": _field(9, stride=2)}
    state = _Net(_network(
        [_layer("exc", "spnet", rows, cols, params="regular", **{
            "init config": {"type": "poisson", "rate": 5, "value": 20, "seed": seed}}),
         _layer("inh", "spnet", rows // 2, cols // 2, params="fast")],
        [_connection("ee", "exc", "exc", "convergent", **weights(6.0, 41), **{
            "plastic": True, "max weight": 10.0, "arborized config": _field(case["field"])}),
         _connection("ei", "exc", "inh", "convergent", **weights(8.0, 42), **between),
         _connection("ie", "inh", "exc", "divergent", opcode="sub", **weights(4.0, 43), **between)]),
        iterations=case["steps"], **{"learning flag": True})
    rng = np.random.default_rng(seed)
    for name in ("ee", "ei", "ie"):
        values = state.matrix(name)
        values *= rng.uniform(0.8, 1.0, values.size).astype(np.float32)
    return state


def _run_spnet(state):
    state.run()
    return {"exc words": state.words("exc"), "inh words": state.words("inh"),
            "voltage": state.values("exc", "voltage"),
            "weights": state.read(state.matrix("ee")),
            "trace": state.read(state.matrix("ee", "presyn trace"))}


def _prepare_life(case, seed):
    rows, cols = case["rows"], case["cols"]
    state = _Net(_network(
        [_layer("board", "game_of_life", rows, cols, survival_min=2, survival_max=3, birth_min=3,
                birth_max=3)],
        [_connection("nbr", "board", "board", "convergent", convolutional=True, **{
            "weight config": {"type": "flat", "weight": 1.0, "diagonal": False},
            "arborized config": _field(3)})]),
        iterations=case["steps"], **{"learning flag": False})
    rng = np.random.default_rng(seed)
    state.neuron("board", "output").view(np.uint32)[:] = \
        (rng.random(rows * cols) < 0.3).astype(np.uint32) << np.uint32(31)
    return state


def _run_life(state):
    state.run()
    return {"words": state.words("board"), "input": state.values("board", "input")}


# ---------------------------------------------------------------------------
# Batch and differentiable network
# ---------------------------------------------------------------------------
class _Batch:
    """Instances of the case's sizes and parameters; their weights, delays
    and drive are the seed's."""

    def __init__(self, case, seed):
        self.instances = [dict(one, seed=seed * 100003 + i) for i, one in enumerate(
            batching.batch_instances(case["count"], 3, case["smin"], case["smax"]))]
        self.batch = sg.Batch(self.instances, tile=(case["tile_rows"], case["tile_colblocks"]))
        self.steps = case["steps"]

    def __del__(self):
        if hasattr(self, "batch"):
            self.batch.close()


def _prepare_batch(case, seed):
    return _Batch(case, seed)


def _run_batch(state):
    state.batch.step(state.steps)
    every = range(len(state.instances))
    return {"words": np.concatenate([state.batch.read(i, "output") for i in every]).view(np.int32),
            "voltage": np.concatenate([state.batch.read(i, "voltage") for i in every]),
            "recovery": np.concatenate([state.batch.read(i, "recovery") for i in every])}


def _adjoint_inputs(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    n, c = case["rows"] * case["cols"], case
    normal = lambda *shape: torch.randn(shape, generator=g, device="cuda")   # noqa: E731
    return {"x": normal(c["steps"], c["batch"], n),
            "weights": normal(c["layers"] - 1, n, c["field"] ** 2) * 0.1,
            "readout": normal(c["outputs"], n) * 0.1,
            "tau": 8.0 + 4.0 * torch.rand(c["layers"], generator=g, device="cuda"),
            "target": torch.rand((c["batch"], c["outputs"]), generator=g, device="cuda")}


def _prepare_adjoint(case, seed):
    inputs = _adjoint_inputs(case, seed)
    for name in ("weights", "readout", "tau") + (("x",) if case["input_grad"] else ()):
        inputs[name].requires_grad_(True)
    shape = {k: case[k] for k in ("layers", "rows", "cols", "field", "outputs", "batch", "steps",
                                  "checkpoint")}
    return {"kind": "adjoint", "net": sg.RateNetwork(**shape), "inputs": inputs}


def _run_adjoint(state):
    inputs = state["inputs"]
    for t in inputs.values():
        t.grad = None
    loss = state["net"].loss(**inputs)
    loss.backward()
    got = {"d " + name: t.grad for name, t in inputs.items() if t.requires_grad}
    got["loss"] = loss.detach()
    return got


# ---------------------------------------------------------------------------
# prepare, run, work, exact
# ---------------------------------------------------------------------------
_PREPARE = {"encoding": _prepare_encoding, "recurrent": _prepare_recurrent,
            "izhikevich": _prepare_izhikevich, "plastic": _prepare_plastic,
            "spnet": _prepare_spnet, "life": _prepare_life, "batch": _prepare_batch,
            "adjoint": _prepare_adjoint}
_RUN = {"encoding": _run_encoding, "recurrent": _run_recurrent, "izhikevich": _run_izhikevich,
        "plastic": _run_plastic, "spnet": _run_spnet, "life": _run_life}


def prepare(case, seed):
    state = _PREPARE[case["kind"]](case, seed)
    if isinstance(state, _Net):
        state.kind = case["kind"]
    return state


def run(state):
    if isinstance(state, _Batch):
        return _run_batch(state)
    if isinstance(state, dict):
        return _run_adjoint(state)
    return _RUN[state.kind](state)


def work(case):
    """Per timestep: each synapse's and neuron's data once (the state of a
    step does not fit on the chip beside the next one's in general)."""
    kind, steps = case["kind"], case["steps"]
    if kind == "batch":
        n = [one["rows"] * one["cols"] for one in batching.batch_instances(
            case["count"], 3, case["smin"], case["smax"])]
        synapses, neurons = sum(0.2 * m * m for m in n), sum(n)
        # weight and source 8, traces read and written 16; convergent 20; neuron 24
        nbytes = 24 * synapses + (20 * 25 + 24) * neurons
        flops = 6 * synapses + (6 * 25 + 200) * neurons
        return {"bytes": nbytes * steps, "flops": flops * steps}
    n = case["rows"] * case["cols"]
    if kind == "encoding":
        w = n * case["hidden"] + case["hidden"] * case["outputs"]
        return {"bytes": 4 * steps * (w + n + case["hidden"] + case["outputs"]),
                "flops": 2 * w * steps}
    if kind == "recurrent":
        return {"bytes": 4 * steps * (n * n + 25 * n + 6 * n), "flops": 2 * steps * (n * n + 25 * n)}
    if kind == "izhikevich":
        return {"bytes": steps * (21 * n * n + 28 * 25 * n + 124 * n),
                "flops": steps * (6 * n * n + 6 * 25 * n + 300 * n)}
    if kind == "plastic":
        conv, window = n * case["field"] ** 2, case["window"] ** 4
        learned = conv + (window if case["learn_window"] else 0)
        active = 29 * conv + 21 * window + 32 * 2 * n * 9 // 4 + 32 * n
        return {"bytes": steps * (active + 40 * learned + 3 * 124 * n),
                "flops": steps * (6 * (conv + window) + 40 * learned + 3 * 300 * n)}
    if kind == "spnet":
        ee, between = n * case["field"] ** 2 // 2, n // 4 * 81 // 2
        return {"bytes": steps * (28 * ee + 12 * (ee + 2 * between) + 40 * n * 5 // 4),
                "flops": steps * (30 * ee + 2 * (ee + 2 * between) + 300 * n)}
    if kind == "life":
        # one bit per cell: the newest and the oldest read, one written
        return {"bytes": 3 * n * steps // 8, "flops": n * steps // 2}
    c = case
    per_layer = c["batch"] * n
    stencils = (c["layers"] - 1) * per_layer * c["field"] ** 2
    # forward, recompute, adjoint and weight gradients; input and its gradient
    return {"bytes": 4 * per_layer * steps * (2 if c["input_grad"] else 1)
            + 8 * n * ((c["layers"] - 1) * c["field"] ** 2 + c["outputs"]),
            "flops": 2 * steps * (4 * stencils + 3 * per_layer * c["outputs"])
            + 30 * steps * c["layers"] * per_layer}


def exact(case, seed):
    """In 64 bits: the rate nets and the gradients.  The spiking nets' spikes
    are decided by single-precision thresholds and have no such value."""
    if case["kind"] == "adjoint":
        return _exact_adjoint(case, seed)
    if case["kind"] not in ("encoding", "recurrent"):
        return None
    numbers = {k: torch.from_numpy(v).cuda().double() for k, v in _numbers(case, seed).items()}
    rate = lambda v: torch.tanh(torch.clamp(v, min=0.0))   # noqa: E731
    if case["kind"] == "encoding":
        # every layer reads what its source gave the step before
        before = hidden = values = None
        answers = []
        for frame in numbers["frames"]:
            answers.append(rate(numbers["w2"] @ hidden) if hidden is not None
                           else torch.zeros(case["outputs"], device="cuda", dtype=torch.double))
            values = numbers["w1"] @ before if before is not None \
                else torch.zeros(case["hidden"], device="cuda", dtype=torch.double)
            hidden, before = rate(values), frame
        got = {"answers": torch.stack(answers), "hidden": hidden, "input": values}
    else:
        n = case["rows"] * case["cols"]
        state = torch.zeros(n, device="cuda", dtype=torch.double)
        driven = torch.zeros_like(state)
        for _ in range(case["steps"]):
            values = driven + numbers["w_rec"] @ state
            state, driven = rate(values), numbers["w_in"].sum(1)
        got = {"rate": state, "input": values}
    return {k: v.cpu().numpy() for k, v in got.items()}


def _exact_adjoint(case, seed):
    c = case
    inputs = {k: v.double() for k, v in _adjoint_inputs(case, seed).items()}
    for name in ("weights", "readout", "tau") + (("x",) if c["input_grad"] else ()):
        inputs[name].requires_grad_(True)
    shape = (c["batch"], c["rows"] * c["cols"])
    v = [torch.zeros(shape, device="cuda", dtype=torch.double) for _ in range(c["layers"])]
    weights = [w.t() for w in inputs["weights"]]
    loss = 0.0
    for t in range(c["steps"]):
        r = [torch.sigmoid(u) for u in v]
        for l in range(c["layers"]):
            if l == 0:
                current = inputs["x"][t]
            else:
                windows = torch.nn.functional.unfold(
                    r[l - 1].view(c["batch"], 1, c["rows"], c["cols"]), c["field"],
                    padding=c["field"] // 2)
                current = (windows * weights[l - 1]).sum(1)
            v[l] = v[l] + (current - v[l]) / inputs["tau"][l]
        y = torch.sigmoid(v[-1]) @ inputs["readout"].t()
        loss = loss + ((y - inputs["target"]) ** 2).sum()
    loss = loss / (c["steps"] * c["batch"] * c["outputs"])
    loss.backward()
    got = {"d " + name: t.grad for name, t in inputs.items() if t.requires_grad}
    got["loss"] = loss.detach()
    return got
