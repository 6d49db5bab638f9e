"""GPU tests of kernels at the sizes where their tiles, chunks and remainders
begin and end, bit-exact against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def sg():
    from synaptogenesis_gb300 import syngen
    assert syngen.get_gpus(), "no CUDA GPU visible"
    syngen.set_warnings(False)
    return syngen


def layer(name, model, rows, cols, **more):
    return dict({"name": name, "neural model": model, "rows": rows, "columns": cols}, **more)


def connection(name, source, to, kind, **more):
    return dict({"name": name, "from layer": source, "to layer": to, "type": kind,
                 "plastic": False, "opcode": "add", "myelinated": True}, **more)


def network(layers, connections):
    return {"structures": [{"name": "s", "type": "parallel", "layers": layers}],
            "connections": connections}


def run_both(sg, net_dict, inject, steps, keys, learning=False, args=None):
    """The keys' arrays after ``steps`` on the GPU and on the oracle, started
    from the same injected arrays; a key is (layer, name) or (connection, name)
    with a leading "matrix"."""
    from oracle.oracle import OracleNetwork
    net, onet = sg.Network(net_dict), OracleNetwork(net_dict)
    net.build_state()

    def gpu(key):
        if key[0] == "matrix":
            return net.get_weight_matrix(key[1], key[2]).to_np_array()
        return net.get_neuron_data("s", key[0], key[1]).to_np_array()

    def cpu(key):
        return onet.get_weight_matrix(key[1], key[2]) if key[0] == "matrix" \
            else onet.get_neuron_data(*key)

    for key, values in inject.items():
        values = np.asarray(values)
        for dst in (gpu(key), cpu(key)):
            assert dst.size == values.size, key
            dst.view(values.dtype)[:] = values
    with sg.Engine(net, None, dict({"learning flag": learning}, **(args or {}))) as eng:
        eng.step(steps)
    for _ in range(steps):
        onet.step(learning=learning)
    return {k: (gpu(k).copy().view(np.uint32), np.asarray(cpu(k)).copy().view(np.uint32))
            for k in keys}


def assert_equal(results):
    for key, (got, want) in results.items():
        bad = np.flatnonzero(got != want)
        assert bad.size == 0, (key, bad.size, bad[:3], got[bad[:3]], want[bad[:3]])


# chunks of 256 sources, two in registers and one in shared memory ahead of the
# one being summed; sums by 16 sources; bands of 8 destinations
@pytest.mark.parametrize("sources,dests", [
    (1, 1), (15, 7), (17, 8), (255, 9), (256, 7), (257, 8), (512, 17), (769, 3), (1025, 33), (1281, 5),
    (40, 4873)])
@pytest.mark.parametrize("model,delay", [("relay", 0), ("game_of_life", 5)])
def test_dense_base_activator(sg, sources, dests, model, delay):
    rng = np.random.default_rng(sources * 7 + dests)
    net = network([layer("a", model, 1, sources), layer("b", "relay", 1, dests)],
                  [connection("c", "a", "b", "fully connected", delay=delay, opcode="sub")])
    words = rng.standard_normal(sources).astype(np.float32).view(np.uint32) if model == "relay" \
        else rng.integers(0, 2**32, sources, dtype=np.uint64).astype(np.uint32)
    inject = {("a", "output"): words,
              ("matrix", "c", "weights"): rng.standard_normal(sources * dests).astype(np.float32)}
    assert_equal(run_both(sg, net, inject, 1, [("b", "input"), ("b", "output")]))


@pytest.mark.parametrize("window", [(0, 1, 0, 1), (1, 12, 2, 13), (3, 20, 1, 16)])
def test_dense_base_activator_subset(sg, window):
    rng = np.random.default_rng(sum(window))
    r0, r1, c0, c1 = window
    net = network([layer("a", "relay", 20, 17), layer("b", "relay", 20, 17)],
                  [connection("c", "a", "b", "subset", **{"subset config": {
                      "from row start": r0, "from row end": r1, "from column start": c0,
                      "from column end": c1, "to row start": r0, "to row end": r1,
                      "to column start": c0, "to column end": c1}})])
    n = ((r1 - r0) * (c1 - c0)) ** 2
    inject = {("a", "output"): rng.standard_normal(20 * 17).astype(np.float32).view(np.uint32),
              ("matrix", "c", "weights"): rng.standard_normal(n).astype(np.float32)}
    assert_equal(run_both(sg, net, inject, 1, [("b", "input")]))


# 128 source rows a CTA, 4 a thread; bands of 8 destinations
@pytest.mark.parametrize("sources,dests", [(1, 1), (31, 9), (33, 8), (128, 7), (129, 17), (300, 3)])
@pytest.mark.parametrize("opcode", ["add", "sub"])
def test_dense_izhikevich_learning(sg, sources, dests, opcode):
    rng = np.random.default_rng(sources + dests)
    n = sources * dests
    net = network([layer("a", "izhikevich", 1, sources, params="regular"),
                   layer("b", "izhikevich", 1, dests, params="fast")],
                  [connection("c", "a", "b", "fully connected", opcode=opcode, plastic=True)])
    draw = lambda lo, hi, m: rng.uniform(lo, hi, m).astype(np.float32)    # noqa: E731
    inject = {("a", "output"): rng.integers(0, 2**32, sources, dtype=np.uint64).astype(np.uint32),
              ("a", "voltage"): draw(-70, 40, sources), ("b", "voltage"): draw(-70, 40, dests),
              ("b", "post trace"): draw(0, 0.004, dests),
              ("b", "time since spike"): rng.integers(0, 33, dests).astype(np.int32),
              ("matrix", "c", "weights"): np.where(rng.random(n) < 0.2, 0, draw(0, 0.5, n)),
              ("matrix", "c", "presyn trace"): draw(0, 0.004, n),
              ("matrix", "c", "weight derivatives"): draw(-1e-3, 1e-3, n),
              ("matrix", "c", "short term R"): draw(0.5, 1, n),
              ("matrix", "c", "short term w"): draw(0.2, 0.8, n)}
    inject[("matrix", "c", "weights")] = inject[("matrix", "c", "weights")].astype(np.float32)
    keys = [("matrix", "c", k) for k in ("weights", "presyn trace", "weight derivatives",
                                         "short term R", "short term w", "short trace")]
    assert_equal(run_both(sg, net, inject, 3, keys + [("b", "voltage")], learning=True))


def test_batches_side_by_side(sg):
    """Batches of few and many work units (the two forms of the step kernel)
    and of different shared-memory sizes, alive together and captured late:
    each equals itself run alone."""
    from synaptogenesis_gb300 import batching
    made = [([batching.instance(s, 40 + s, rows=s, cols=c) for s, c in sides], tile)
            for sides, tile in (([(61, 97), (16, 16), (128, 70)], (1, 1)), ([(20, 33), (5, 9)], (2, 2)))]

    def read(b, insts):
        return [b.read(i, k).view(np.uint32) for i in range(len(insts))
                for k in ("voltage", "recovery", "output")]

    alone = []
    for insts, tile in made:
        with sg.Batch(insts, tile=tile) as b:
            b.step(70)
            alone.append(read(b, insts))
    together = [sg.Batch(insts, tile=tile) for insts, tile in made]
    for b in together:
        b.step(70)
    for b, (insts, _), want in zip(together, made, alone):
        assert all(np.array_equal(x, y) for x, y in zip(read(b, insts), want))
        b.close()


# rows across a warp: 1, 2 or 4 words a lane up to 1024, 2048 and 4096 cells, a
# last word of any number of bits; whole runs of 12 steps a launch
@pytest.mark.parametrize("rows,cols,diagonal,low,high", [
    (1, 1, False, 2, 3), (5, 2, True, 2, 3), (3, 31, False, 2, 3), (40, 33, False, 1, 4),
    (7, 63, True, 3, 4), (200, 333, False, 2, 3), (19, 1000, False, 2, 3), (9, 1023, True, 2, 5),
    (8, 1025, False, 2, 3), (6, 1056, False, 2, 3), (11, 1999, True, 3, 4), (5, 2049, False, 2, 3),
    (4, 2080, False, 1, 3), (3, 4095, False, 2, 3)])
def test_gol_whole_runs_on_ragged_boards(sg, rows, cols, diagonal, low, high):
    net = network([layer("b", "game_of_life", rows, cols, survival_min=low, survival_max=high,
                         birth_min=3, birth_max=3)],
                  [connection("c", "b", "b", "convergent", convolutional=True, **{
                      "weight config": {"type": "flat", "weight": 1.0, "diagonal": diagonal},
                      "arborized config": {"field size": 3, "wrap": True}})])
    words = np.random.default_rng(rows * cols).integers(0, 2**32, rows * cols,
                                                       dtype=np.uint64).astype(np.uint32)
    for steps in (1, 12, 37):
        assert_equal(run_both(sg, net, {("b", "output"): words}, steps,
                              [("b", "output"), ("b", "input")]))


# tiles of 32 columns by 4 warps of 1, 2 or 8 rows, rows copied whole or by 4
# floats, segments longer than the checkpoint, groups of the batch; the field
# sizes that have their own tiles
@pytest.mark.parametrize("cfg", [
    dict(layers=2, rows=33, cols=36, field=1, outputs=1, batch=9, steps=5),
    dict(layers=3, rows=65, cols=64, field=3, outputs=16, batch=40, steps=6),
    dict(layers=2, rows=17, cols=31, field=5, outputs=9, batch=70, steps=34),
    dict(layers=2, rows=9, cols=33, field=5, outputs=8, batch=33, steps=11),
    dict(layers=3, rows=24, cols=68, field=7, outputs=3, batch=17, steps=7),
    dict(layers=2, rows=7, cols=40, field=9, outputs=5, batch=6, steps=12)])
def test_rate_tiles(cfg):
    """Loss and gradients against the FP64 restatement, and bit for bit the
    same whatever the checkpoint stride and the workspace's alignment."""
    import ctypes
    import torch
    from oracle import rate_adjoint as ra
    from synaptogenesis_gb300 import syngen
    from tests.test_gpu_rate import close, gpu_grads, make
    p = make(13, *(cfg[k] for k in ("layers", "rows", "cols", "field", "outputs", "batch", "steps")))
    nets = [syngen.RateNetwork(checkpoint=k, **cfg) for k in (1, 3, cfg["steps"])]
    results = [gpu_grads(torch, syngen, net, p) for net in nets]
    for other in results[1:]:
        for a, b in zip(other, results[0]):
            assert np.array_equal(np.asarray(a), np.asarray(b))
    want = ra.adjoint(dict(cfg, checkpoint=1, dt=1.0), p["x"], p["weights"], p["readout"], p["tau"],
                      p["target"])
    assert abs(results[0][0] - want[0]) <= 1e-5 * abs(want[0])
    for got, w in zip(results[0][1:], want[1:]):
        ok, norm = close(got, w)
        assert ok, norm
    # a workspace that starts 4 bytes off a 16-byte boundary
    net, t = nets[1], {k: torch.tensor(v, device="cuda") for k, v in p.items()}
    ws = torch.empty(net.workspace_bytes // 4 + 4, device="cuda")[1:]
    loss = torch.empty((), device="cuda")
    grads = [torch.empty_like(t[k]) for k in ("weights", "readout", "tau", "x")]
    args = [t[k].data_ptr() for k in ("x", "weights", "readout", "tau", "target")]
    stream = torch.cuda.current_stream().cuda_stream
    assert syngen._syn.sg_rate_forward(ctypes.byref(net.shape), *args, None, loss.data_ptr(),
                                       ws.data_ptr(), stream) == 0
    assert syngen._syn.sg_rate_backward(ctypes.byref(net.shape), *args, 1.0, ws.data_ptr(),
                                        *(g.data_ptr() for g in grads), stream) == 0
    for a, b in zip([loss] + grads, results[0]):
        np.testing.assert_allclose(a.cpu().numpy(), b, rtol=1e-4, atol=1e-4 * np.abs(b).max())


@pytest.mark.parametrize("opcode", ["add", "sub"])
@pytest.mark.parametrize("rows,cols", [(1, 7), (10, 33)])
def test_spnet_neurons_and_sparse_learning(sg, opcode, rows, cols):
    """Zero and nonzero traces and derivatives, spikes on either side, voltages
    on both sides of the threshold; two layers of different sizes in one launch."""
    from tests.golden.cases import Case
    from tests.harness import compare, run_library, run_oracle
    n, m = rows * cols, (rows + 2) * cols
    net = network([layer("a", "spnet", rows, cols, params="regular"),
                   layer("b", "spnet", rows + 2, cols, params="fast")],
                  [connection("c", "a", "b", "fully connected", opcode=opcode, plastic=True,
                              sparse=True)])

    def inject(rng, sizes):
        size, dense = sizes["conn:c"], sizes["dense:c"]
        draw = lambda lo, hi, k: rng.uniform(lo, hi, k).astype(np.float32)    # noqa: E731
        some = lambda v: np.where(rng.random(v.size) < 0.4, 0, v).astype(np.float32)  # noqa: E731
        words = rng.integers(0, 2**32, n, dtype=np.uint64).astype(np.uint32)
        kept = np.arange(dense) % 5 < 3                      # as many for every destination
        size = int(kept.sum()) if size == dense else size
        got = {("matrix", "c", "init weights"): np.where(kept, draw(0.1, 5, dense), 0).astype(np.float32),
               ("neuron", "s", "a", "output"): words, ("neuron", "s", "a", "voltage"): draw(-90, 45, n),
               ("neuron", "s", "b", "voltage"): draw(-90, 45, m),
               ("neuron", "s", "a", "recovery"): draw(-20, 20, n),
               ("neuron", "s", "b", "post trace"): some(draw(0, 1, m)),
               ("neuron", "s", "b", "time since spike"): rng.integers(0, 33, m).astype(np.int32)}
        if n % 5 == 0:
            got[("matrix", "c", "presyn trace")] = some(draw(0, 1, size))
            got[("matrix", "c", "weight derivative")] = some(draw(-0.1, 0.1, size))
        return got

    final = [("neuron", "s", "a", k) for k in ("voltage", "recovery", "output")]
    final += [("neuron", "s", "b", k) for k in ("voltage", "recovery", "post trace", "output", "input")]
    final += [("matrix", "c", k) for k in ("weights", "presyn trace", "weight derivative",
                                           "time since spike")]
    case = Case("spnet_edges", net, 40, rows * cols, inject=inject, final=final,
                inputs={"a": lambda rng, t, k: (rng.random(k) < 0.2) * 20.0,
                        "b": lambda rng, t, k: (rng.random(k) < 0.2) * 20.0})
    problems = compare(run_library(case, sg), run_oracle(case))
    assert not problems, problems[:3]


def test_state_moves_only_what_was_handed_out(sg, tmp_path):
    """A caller that reads and changes a few arrays, late and between runs, over a
    save and a load, sees what one that holds every array sees."""
    from tests.golden.configs import c0_inject, c0_net
    from tests.harness import case_sizes
    from tests.golden.cases import Case
    case = Case("state", c0_net(8), 1, 5, inject=lambda rng, sizes: c0_inject(rng, sizes, 8))
    inject = case.injections(case_sizes(case))
    net_dict = case.net
    for c in net_dict["connections"]:
        c["myelinated"] = True
    keys = [("iz", k) for k in ("voltage", "recovery", "output", "input", "nmda", "time since spike")]
    keys += [("in", "output"), ("in", "input")]
    keys += [("matrix", c, k) for c in ("c_in", "c_rec") for k in ("weights", "long trace", "delays")]

    def run(hold_all):
        net = sg.Network(net_dict)
        net.build_state()

        def get(key):
            if key[0] == "matrix":
                return net.get_weight_matrix(key[1], key[2]).to_np_array()
            return net.get_neuron_data("s", key[0], key[1]).to_np_array()

        def step(n):
            if hold_all:
                [get(k) for k in keys]
            net.run({"modules": []}, {"iterations": n, "learning flag": False, "graphs": False})

        for key, values in inject.items():
            dst = get(key[1:] if key[0] == "matrix" and False else
                      (key if key[0] == "matrix" else key[2:]))
            dst.view(values.dtype)[:] = values
        step(3)
        get(("iz", "voltage"))[:] -= 1.0
        step(2)
        kept = get(("matrix", "c_in", "long trace"))          # first handed out after runs
        kept *= 2.0
        step(4)
        get(("iz", "recovery"))
        kept *= 0.5                                           # refreshed by any getter
        step(2)
        path = str(tmp_path / ("state%d" % hold_all))
        get(("iz", "voltage"))[:] += 0.5
        net.save_state(path)
        step(3)
        net.load_state(path)
        step(5)
        return {k: get(k).copy().view(np.uint32) for k in keys}

    few, every = run(False), run(True)
    for k in keys:
        assert np.array_equal(few[k], every[k]), k


# summaries of up to 12 distinct delays among a source's last 32 visits, six to a
# word, and the scan beyond; 16 compacted synapses in flight
@pytest.mark.parametrize("model", ["izhikevich", "spnet"])
@pytest.mark.parametrize("delays,dests", [(1, 1), (6, 15), (7, 17), (12, 33), (13, 40), (31, 64)])
def test_time_since_spike_summaries(sg, model, delays, dests):
    from tests.golden.cases import Case
    from tests.harness import compare, run_library, run_oracle
    layers = [layer("a", model, 3, 13, params="regular"), layer("b", model, 1, dests, params="fast")]
    conns = [connection("c", "a", "b", "fully connected"), connection("r", "b", "a", "fully connected")]
    for c in conns:
        del c["myelinated"]
        c["sparse"] = model == "spnet"

    def inject(rng, sizes):
        got = {("neuron", "s", "a", "output"): rng.integers(0, 2**32, 39, dtype=np.uint64).astype(np.uint32)
               & rng.integers(0, 2**32, 39, dtype=np.uint64).astype(np.uint32)}
        for c in ("c", "r"):
            n = sizes["dense:" + c]
            got[("matrix", c, "init weights")] = rng.uniform(0.1, 1, n).astype(np.float32)
            got[("matrix", c, "delays")] = rng.integers(0, delays, n).astype(np.int32)
        return got

    final = [("matrix", c, "time since spike") for c in ("c", "r")]
    final += [("neuron", "s", l, k) for l in ("a", "b") for k in ("voltage", "input", "output")]
    case = Case("summaries", network(layers, conns), 6, delays + dests, inject=inject, final=final,
                inputs={"a": lambda rng, t, k: (rng.random(k) < 0.3) * 30.0})
    problems = compare(run_library(case, sg), run_oracle(case))
    assert not problems, problems[:3]


# blocks of 128 destinations and the sources they draw on, staged in shared memory
# (places past the layer's end, groups of 32 sources, ragged rows of 16 synapses) or
# too many to stage; spikes, numbers and whole numbers as outputs
@pytest.mark.parametrize("source", ["spnet", "relay", "game_of_life"])
@pytest.mark.parametrize("rows,cols,field,wrap", [
    (1, 127, 5, False), (16, 8, 9, True), (3, 43, 3, False), (20, 33, 7, True), (40, 40, 17, True),
    (120, 120, 3, True), (150, 160, 1, False)])
def test_spnet_source_windows(sg, source, rows, cols, field, wrap):
    from tests.golden.cases import Case
    from tests.harness import compare, run_library, run_oracle
    half = -(field // 2)                    # the field around its destination
    net = network([layer("a", source, rows, cols, **({"params": "regular"} if source == "spnet" else {})),
                   layer("b", "spnet", rows, cols, params="fast")],
                  [connection("c", "a", "b", "convergent", opcode="sub", sparse=True, plastic=False,
                              **{"arborized config": {"field size": field, "stride": 1, "wrap": wrap,
                                                      "offset": half}})])

    n, positions = rows * cols, field * field
    rng = np.random.default_rng(n + field)
    bits = rng.integers(0, 2**32, n, dtype=np.uint64).astype(np.uint32)
    output = {"spnet": bits, "relay": rng.normal(0, 3, n).astype(np.float32).view(np.uint32),
              "game_of_life": bits % 7}[source]
    weights = (rng.uniform(0.1, 5, (n, positions)) * (rng.random((n, positions)) < 0.7)).astype(np.float32)
    delays = rng.integers(0, 32, (n, positions)).astype(np.int32)
    # the delays of a destination's compacted synapses: nonzero weights inside the layer
    r, c = np.divmod(np.arange(n)[:, None], cols)
    dr, dc = np.divmod(np.arange(positions), field)
    inside = wrap | ((r + dr + half >= 0) & (r + dr + half < rows) & (c + dc + half >= 0) & (c + dc + half < cols))
    kept = inside & (weights != 0)
    compact = np.zeros((n, kept.sum(1).max()), np.int32)
    for d in range(n):
        compact[d, :kept[d].sum()] = delays[d, kept[d]]

    final = [("neuron", "s", l, k) for l in ("a", "b") for k in ("output", "input")]
    final += [("matrix", "c", "time since spike"), ("neuron", "s", "b", "voltage")]

    def case(delays):
        given = {("neuron", "s", "a", "output"): output, ("matrix", "c", "init weights"): weights.ravel(),
                 ("matrix", "c", "delays"): delays.ravel()}
        return Case("windows", net, 3, 1, inject=lambda rng, sizes: given, final=final,
                    inputs={"a": lambda rng, t, k: (rng.random(k) < 0.2) * 20.0})

    problems = compare(run_library(case(delays), sg), run_oracle(case(compact)))
    assert not problems, problems[:3]


# chunks of 256 source rows, sums of 16, columns padded to 32; the last width of the
# kernel; every output type (its fused weight with learning off)
@pytest.mark.parametrize("sources,dests", [(1, 1), (15, 9), (255, 8), (256, 7), (257, 17), (512, 3),
                                           (800, 8), (1536, 9)])
@pytest.mark.parametrize("model,opcode,learning", [("izhikevich", "add", True), ("izhikevich", "sub", False),
                                                   ("relay", "add", False), ("game_of_life", "mult", False)])
def test_one_pass_trace_activator(sg, sources, dests, model, opcode, learning):
    rng = np.random.default_rng(sources + dests)
    n = sources * dests
    net = network([layer("a", model, 1, sources, **({"params": "regular"} if model == "izhikevich" else {})),
                   layer("b", "izhikevich", 1, dests, params="fast")],
                  [connection("c", "a", "b", "fully connected", opcode=opcode, plastic=learning,
                              **({"learning rate": 0.1} if learning else {}))])
    draw = lambda lo, hi, m: rng.uniform(lo, hi, m).astype(np.float32)    # noqa: E731
    bits = rng.integers(0, 2**32, sources, dtype=np.uint64).astype(np.uint32)
    output = {"izhikevich": bits, "relay": draw(-2, 2, sources).view(np.uint32), "game_of_life": bits % 5}[model]
    inject = {("a", "output"): output, ("matrix", "c", "weights"): draw(0, 0.5, n),
              ("matrix", "c", "delays"): rng.integers(0, 32, n).astype(np.int32),
              ("matrix", "c", "short term R"): draw(0.5, 1, n),
              ("matrix", "c", "short term w"): draw(0.2, 0.8, n)}
    keys = [("matrix", "c", "short trace"), ("b", "voltage"), ("b", "input")]
    assert_equal(run_both(sg, net, inject, 4, keys, learning=learning))


# a CTA a group of 32 destinations while the tile's units are no more than the SMs:
# rounds of 28 slots, 112 of them in flight, convolutions of more and fewer positions
# than a round, ragged groups, more groups than resident CTAs
@pytest.mark.parametrize("sides", [[(5, 6)], [(7, 33), (16, 16)], [(31, 64), (9, 10), (48, 48)],
                                   [(64, 64), (40, 96), (33, 65)]])
@pytest.mark.parametrize("field", [3, 5, 7])
def test_batch_split_groups(sg, sides, field):
    from synaptogenesis_gb300 import batching
    insts = [dict(batching.instance(r + c, 70 + i, rows=r, cols=c), conv_field=field)
             for i, (r, c) in enumerate(sides)]
    for inst in insts:
        inst["input_rate"] = 0.1

    def run(more, tile):
        with sg.Batch(insts + more, tile=tile) as b:
            b.step(37)
            return [b.read(i, k).view(np.uint32) for i in range(len(insts))
                    for k in ("voltage", "recovery", "output")], int(b.report().properties["threads"])

    split, threads = run([], (8, 1))
    assert threads == 256
    # beside enough others the same instances take the tile's units
    whole, _ = run([dict(batching.instance(96, 300 + i), conv_field=field) for i in range(24)], (2, 1))
    assert all(np.array_equal(a, b) for a, b in zip(split, whole))


# derivatives, traces and weights that are not finite, as a float-valued source's words
# read as spikes make them: a NaN derivative makes a NaN weight, in the sparse kernel as
# in the dense one
@pytest.mark.parametrize("sparse", [True, False])
@pytest.mark.parametrize("source", ["spnet", "relay"])
@pytest.mark.parametrize("opcode", ["add", "sub"])
def test_spnet_learning_of_what_is_not_finite(sg, opcode, source, sparse):
    sources, dests = 9, 130
    n = sources * dests
    net = network([layer("a", source, 1, sources, **({"params": "regular"} if source == "spnet" else {})),
                   layer("b", "spnet", 1, dests, params="fast")],
                  [connection("c", "a", "b", "fully connected", opcode=opcode, plastic=True, sparse=sparse,
                              **{"weight config": {"type": "flat", "weight": 1.0}})])
    odd = np.array([np.nan, np.inf, -np.inf, 3e38, -3e38, 0, 2.0**-60, 2.0**-61, 1e-40, 0.1], np.float32)
    rng = np.random.default_rng(sources)
    draw = lambda: np.where(rng.random(n) < 0.5, rng.choice(odd, n),         # noqa: E731
                            rng.uniform(0, 1, n)).astype(np.float32)
    # (a relay's own words as numbers; the destinations' as spikes, floats among them NaN)
    words = rng.integers(0, 2**32, sources, dtype=np.uint64).astype(np.uint32)
    inject = {("a", "output"): words if source == "spnet" else rng.choice(odd[5:], sources),
              ("b", "output"): np.where(rng.random(dests) < 0.3, 0xFF800001,
                                        rng.integers(0, 2**32, dests, dtype=np.uint64)).astype(np.uint32),
              ("matrix", "c", "weights"): np.where(rng.random(n) < 0.2, odd[rng.integers(0, 10, n)],
                                                   rng.uniform(0.1, 5, n)).astype(np.float32),
              ("matrix", "c", "weight derivative"): draw(), ("matrix", "c", "presyn trace"): draw()}
    keys = [("matrix", "c", k) for k in ("weights", "weight derivative", "presyn trace")]
    results = run_both(sg, net, inject, 2, keys, learning=True)
    for key, (got, want) in results.items():
        g, w = got.view(np.float32), want.view(np.float32)
        bad = np.flatnonzero((got != want) & ~(np.isnan(g) & np.isnan(w)))
        assert bad.size == 0, (key, bad.size, g[bad[:3]], w[bad[:3]])
    assert np.isnan(results[keys[0]][1].view(np.float32)).sum() > 20


def rate_pass(net, p, y=None):
    """Loss and gradients of a RateNetwork for arrays p, as numpy."""
    import torch
    t = {k: torch.tensor(np.asarray(v, np.float32), device="cuda") for k, v in p.items()}
    loss, ws = net._forward(**t, y=y)
    args = [t[k] for k in ("x", "weights", "readout", "tau", "target")]
    grads = dict(zip(("x", "weights", "readout", "tau"), net._backward(ws, 1.0, *args)))
    return {k: v.cpu().numpy() for k, v in dict(grads, loss=loss).items()}


def test_rate_sigmoid(sg):
    """One step from rest with tau 1 makes v the input; the readout picks single
    neurons.  The exponential errs by at most 2 + 1.173 |v| units in the last place, the
    sum with 1 and the reciprocal by half of one each; where the exponential overflows
    (below -88.7) the sigmoid is less than 2^-128."""
    import torch
    batch, n = 65535, 16
    net = sg.RateNetwork(layers=1, rows=1, cols=n, field=1, outputs=n, batch=batch, steps=1)
    rng = np.random.default_rng(3)
    v = rng.uniform(-100, 40, (1, batch, n)).astype(np.float32)
    v[:, ::4] = rng.uniform(-89, -86, v[:, ::4].shape)
    v[0, 0] = [0, -0.0, 1e-30, -1e-30, 88, 100, -88, -150, 3e38, -3e38, np.inf, -np.inf, 17, -17, 1, -1]
    y = torch.empty((1, batch, n), device="cuda")
    rate_pass(net, {"x": v, "weights": np.zeros((0, n, 1)), "readout": np.eye(n), "tau": [1.0],
                    "target": np.zeros((batch, n))}, y)
    got, x = y.cpu().numpy().astype(np.float64), v.astype(np.float64)
    # an infinite neuron makes the zero weights' terms NaN only in its own batch element
    got, x = np.delete(got, 0, 1), np.delete(x, 0, 1)
    want = np.exp(np.minimum(x, 0)) / (1 + np.exp(-np.abs(x)))
    bound = ((2 + 1.173 * np.abs(x)) + 1) * 2.0**-23 * want + 2.0**-127
    bad = np.flatnonzero(~(np.abs(got - want) <= bound))
    assert bad.size == 0, (bad.size, x.ravel()[bad[:4]], got.ravel()[bad[:4]], want.ravel()[bad[:4]])


def test_rate_tau_gradient_of_equal_elements(sg):
    """2^14 equal batch elements of one neuron: the loss is one element's, and every
    quantity of the gradient is scaled by a power of two and added up to the same bits."""
    rng = np.random.default_rng(5)
    for _ in range(24):
        steps = 4
        x, tau = rng.normal(0, 1, (steps, 1, 1)), rng.uniform(2, 9, 1)
        readout, target = rng.normal(0, 1, (1, 1)), rng.uniform(0, 1, (1, 1))
        tau_grads = []
        for batch in (1, 1 << 14):
            net = sg.RateNetwork(layers=1, rows=1, cols=1, field=1, outputs=1, batch=batch, steps=steps)
            got = rate_pass(net, {"x": np.repeat(x, batch, 1), "weights": np.zeros((0, 1, 1)), "readout": readout,
                                  "tau": tau, "target": np.repeat(target, batch, 0)})
            tau_grads.append(got["tau"][0])
        assert tau_grads[0] == tau_grads[1], tau_grads


def test_rate_adjoint_adds_kernel_rows(sg):
    """Nine terms p of one kernel row beside +2^26 p and -2^26 p of the rows before and
    after: the row's sum 9 p is added whole (to a multiple of the large one's spacing,
    4 p to 8 p), where p by itself is less than half the spacing and would be lost."""
    side, h = 9, 4
    n = side * side
    net = sg.RateNetwork(layers=2, rows=side, cols=side, field=9, outputs=1, batch=1, steps=2)
    centre = h * side + h

    def input_gradient(rows):
        w = np.zeros((1, n, 81))
        for (kr, kc), value in rows.items():           # the destination that reads the centre at (kr, kc)
            w[0, (2 * h - kr) * side + 2 * h - kc, kr * 9 + kc] = value
        # a time constant of 2^60 keeps layer 1 at rest whatever its input is
        got = rate_pass(net, {"x": np.full((2, 1, n), 0.3), "weights": w, "readout": np.full((1, n), 0.37),
                              "tau": [3.0, 2.0**60], "target": [[0.2]]})
        return got["x"][0, 0, centre]

    one = input_gradient({(4, 4): 1.0})
    row = input_gradient({(0, 0): 2.0**26, (2, 0): -(2.0**26), **{(1, kc): 1.0 for kc in range(9)}})
    assert 5.0 <= row / one <= 13.0, (row, one)


# either side of the line between the two kernels of dense matrices (48 sources for few
# destinations, 186 for 10000, none for 98305), numbers and spikes
@pytest.mark.parametrize("sources,dests", [(47, 900), (48, 900), (185, 10000), (186, 10000), (3, 98304), (700, 1500),
                                           (50, 98305)])
@pytest.mark.parametrize("model,delay", [("relay", 0), ("game_of_life", 7)])
def test_dense_base_activators_by_size(sg, sources, dests, model, delay):
    rng = np.random.default_rng(sources + dests)
    net = network([layer("a", model, 1, sources), layer("b", "relay", 1, dests)],
                  [connection("c", "a", "b", "fully connected", delay=delay, opcode="sub")])
    words = rng.standard_normal(sources).astype(np.float32).view(np.uint32) if model == "relay" \
        else rng.integers(0, 2**32, sources, dtype=np.uint64).astype(np.uint32)
    inject = {("a", "output"): words,
              ("matrix", "c", "weights"): rng.standard_normal(sources * dests).astype(np.float32)}
    assert_equal(run_both(sg, net, inject, 1, [("b", "input"), ("b", "output")]))


def test_dense_base_activators_of_windows(sg):
    """Subset windows of few and of many sources, side by side with the dense form."""
    rng = np.random.default_rng(4)
    window = lambda k: {"subset config": {                                   # noqa: E731
        "from row start": 1, "from row end": 1 + k, "from column start": 2, "from column end": 2 + k,
        "to row start": 0, "to row end": 20, "to column start": 1, "to column end": 17}}
    net = network([layer("a", "relay", 20, 17), layer("b", "relay", 20, 17)],
                  [connection("few", "a", "b", "subset", **window(3)),
                   connection("many", "a", "b", "subset", opcode="sub", **window(15))])
    inject = {("a", "output"): rng.standard_normal(20 * 17).astype(np.float32).view(np.uint32)}
    for name, k in (("few", 3), ("many", 15)):
        inject[("matrix", name, "weights")] = rng.standard_normal(k * k * 320).astype(np.float32)
    assert_equal(run_both(sg, net, inject, 1, [("b", "input")]))


# registers of all layers in launches of 16, a neuron a thread up to 2^18 neurons and eight
# beyond; relay and rate layers of more than 8 blocks to an SM
def test_input_registers_of_many_and_large_layers(sg):
    from tests.golden.cases import Case
    from tests.harness import compare, run_library, run_oracle
    kinds = [None, {"type": "flat", "value": 0.75}, {"type": "uniform", "min": -1, "max": 2, "seed": 5},
             {"type": "poisson", "rate": 200, "value": 1.5, "seed": 7},
             {"type": "poisson", "rate": 300, "value": 2.5, "random": True, "seed": 8},
             {"type": "normal", "mean": 0.5, "std dev": 0.2, "seed": 9}]
    layers = [layer("l%d" % i, "relay", 1, 97 * i + 1, **({"init config": kinds[i % 6]} if kinds[i % 6] else {}))
              for i in range(35)]
    sizes = ((1 << 18) + 1, 311_297, 400_001)
    layers += [layer("big%d" % i, "relay" if i else "rate_encoding", 1, n, **{"init config": kinds[2 + i]})
               for i, n in enumerate(sizes)]
    fed = ["l%d" % i for i in (0, 3, 7, 11, 16, 17, 32, 34)] + ["big2"]
    final = [("neuron", "s", l["name"], k) for l in layers for k in ("input", "output")]
    case = Case("registers", network(layers, []), 5, 3, final=final,
                inputs={name: lambda rng, t, k: rng.standard_normal(k) for name in fed})
    # (tanh may differ in the last bit between the GPU and the host's library)
    problems = compare(run_library(case, sg), run_oracle(case), tol=1e-6, float_keys=("big0/output",))
    assert not problems, problems[:3]


# whole words, either side of the lines between strips and tiles
@pytest.mark.parametrize("rows,words", [(4096, 2), (4097, 8), (6080, 9), (6081, 16), (6081, 17), (400, 65), (401, 96),
                                        (3, 127), (5, 128)])
def test_gol_whole_runs_by_board(sg, rows, words):
    cols = 32 * words
    net = network([layer("b", "game_of_life", rows, cols, survival_min=2, survival_max=3, birth_min=3, birth_max=3)],
                  [connection("c", "b", "b", "convergent", convolutional=True, **{
                      "weight config": {"type": "flat", "weight": 1.0, "diagonal": False},
                      "arborized config": {"field size": 3, "wrap": True}})])
    board = np.random.default_rng(rows + cols).integers(0, 2**32, rows * cols, dtype=np.uint64).astype(np.uint32)
    assert_equal(run_both(sg, net, {("b", "output"): board}, 14, [("b", "output"), ("b", "input")]))


def test_arrays_kept_by_callbacks_move(sg):
    """Arrays that a weight and a delay callback kept show what was learned and take
    what the caller writes, like those of the getters."""
    kept = {}

    def weights(_, size, data):
        kept["weights"] = sg.FloatArray(size, data).to_np_array()
        kept["weights"][:] = np.linspace(0.1, 0.4, size, dtype=np.float32)

    def delays(_, size, __, data):
        kept["delays"] = sg.IntArray(size, data).to_np_array()
        kept["delays"][:] = np.arange(size) % 5

    sg.create_weight_callback("kept weights", weights)
    sg.create_delay_weight_callback("kept delays", delays)
    net = sg.Network(network(
        [layer("a", "izhikevich", 6, 6, params="regular", **{"init config": {"type": "flat", "value": 20.0}}),
         layer("b", "izhikevich", 6, 6, params="regular")],
        [connection("c", "a", "b", "fully connected", plastic=True, **{
            "learning rate": 0.1, "weight config": {"type": "flat", "weight": 0.5, "callback": "kept weights",
                                                    "delay callback": "kept delays"}})]))
    net.build_state()
    first = kept["weights"].copy()
    step = lambda: (net.run({"modules": []}, {"iterations": 20}),                # noqa: E731
                    net.get_neuron_data("s", "b", "voltage").to_np_array().copy())
    step()
    assert not np.array_equal(kept["weights"], first)
    kept["weights"][:] = 0.25
    kept["delays"][:] = 3
    step()
    assert kept["weights"].max() < first.max()
    assert np.array_equal(kept["weights"], net.get_weight_matrix("c").to_np_array())
    assert np.array_equal(net.get_weight_matrix("c", "delays").to_np_array(), np.full(36 * 36, 3))


# one form for a batch's number of groups, whatever the tile: 912 groups are three for
# each CTA of several warps to a group that 152 SMs hold, 608 two (16 x 16, whose groups
# have few slots), 456 three where an instance takes an SM
@pytest.mark.parametrize("sides,split", [([(64, 64)] * 7 + [(8, 64)], True), ([(64, 64)] * 7 + [(9, 64)], False),
                                         ([(128, 128)], True), ([(192, 192)], False), ([(16, 16)] * 38, True),
                                         ([(16, 16)] * 39, False)])
def test_batch_form_by_groups(sg, sides, split):
    from synaptogenesis_gb300 import batching
    insts = [batching.instance(r, 7 + i, rows=r, cols=c) for i, (r, c) in enumerate(sides)]
    seen, first = set(), None
    for tile in ((1, 1), (2, 2), (8, 1)):
        with sg.Batch(insts, tile=tile) as b:
            b.step(5)
            words = np.concatenate([b.read(i, "output") for i in range(len(insts))])
            report = b.report().properties
        assert (report["units"] == report["groups"] and int(report["threads"]) == 256) == split, (tile, report)
        first = words if first is None else first
        assert np.array_equal(words, first)
    # and the other form, beside enough others, gives the same
    more = [batching.instance(96, 300 + i) for i in range(24)]
    with sg.Batch(insts + more, tile=(2, 1)) as b:
        b.step(5)
        assert int(b.report().properties["threads"]) == 64
        assert np.array_equal(np.concatenate([b.read(i, "output") for i in range(len(insts))]), first)


# several segments of the backward pass and chunks of the forward one, the last of them
# short: networks whose steps are too large for one segment (5 to 10 steps of 64 MB), for
# every field, rows copied by 4 floats and one at a time, one row a thread and more
@pytest.mark.parametrize("cfg", [
    dict(layers=3, rows=300, cols=333, field=1, outputs=16, batch=2, steps=30),
    dict(layers=2, rows=333, cols=301, field=3, outputs=16, batch=2, steps=21),
    dict(layers=2, rows=250, cols=300, field=3, outputs=16, batch=1, steps=33),
    dict(layers=2, rows=140, cols=255, field=5, outputs=16, batch=1, steps=40),
    dict(layers=2, rows=140, cols=252, field=5, outputs=16, batch=1, steps=41),
    dict(layers=2, rows=201, cols=255, field=5, outputs=16, batch=1, steps=31),
    dict(layers=2, rows=170, cols=225, field=7, outputs=4, batch=1, steps=31),
    dict(layers=2, rows=120, cols=224, field=7, outputs=4, batch=1, steps=45),
    dict(layers=2, rows=101, cols=203, field=9, outputs=3, batch=1, steps=40),
    dict(layers=2, rows=104, cols=200, field=9, outputs=3, batch=1, steps=43)],
    ids=lambda c: "%(rows)dx%(cols)d-field%(field)d" % c)
def test_rate_segments(cfg):
    """Loss and gradients against the FP64 restatement, and bit for bit the same with
    the smallest segments, somewhat larger ones and a single one."""
    import torch
    from oracle import rate_adjoint as ra
    from synaptogenesis_gb300 import syngen
    from tests.test_gpu_rate import close, gpu_grads, make
    p = make(17, *(cfg[k] for k in ("layers", "rows", "cols", "field", "outputs", "batch", "steps")))
    nets = [syngen.RateNetwork(checkpoint=k, **cfg) for k in (1, 13, cfg["steps"])]
    assert len({net.workspace_bytes for net in nets}) == 3        # segments of three lengths
    results = [gpu_grads(torch, syngen, net, p) for net in nets]
    for other in results[1:]:
        for a, b in zip(other, results[0]):
            assert np.array_equal(np.asarray(a), np.asarray(b))
    want = ra.adjoint(dict(cfg, checkpoint=1, dt=1.0), p["x"], p["weights"], p["readout"], p["tau"],
                      p["target"])
    assert abs(results[0][0] - want[0]) <= 1e-5 * abs(want[0])
    for got, w in zip(results[0][1:], want[1:]):
        ok, norm = close(got, w)
        assert ok, norm


def test_spnet_groups_of_layers_and_connections(sg):
    """Eleven spnet layers and connections: neuron updates and time-since-spike updates go
    in launches of eight, of sizes that share blocks."""
    n = 11
    layers = [layer("n%d" % i, "spnet", 1, 23 + 61 * i % 257, params="fast" if i % 3 else "regular", **{
        "init config": {"type": "poisson", "rate": 150, "value": 25, "seed": 40 + i}}) for i in range(n)]
    conns = [connection("c%d" % i, "n%d" % i, "n%d" % ((i * 4 + 1) % n), "fully connected",
                        opcode="sub" if i % 4 == 3 else "add", plastic=True, sparse=i % 2 == 0,
                        **{"weight config": {"type": "flat", "weight": 0.5 + 0.1 * i}, "delay": i})
             for i in range(n)]
    keys = [("n%d" % i, k) for i in range(n) for k in ("voltage", "recovery", "output", "post trace",
                                                       "time since spike")]
    keys += [("matrix", "c%d" % i, k) for i in range(n) for k in ("weights", "time since spike")]
    results = run_both(sg, network(layers, conns), {}, 45, keys, learning=True)
    assert_equal(results)
    assert all((results[("n%d" % i, "output")][1] != 0).any() for i in range(n))


def test_report_of_moved_bytes(sg):
    """The bytes that a run moves each way: those of the arrays handed out so far."""
    net = sg.Network(network([layer("a", "relay", 5, 7), layer("b", "izhikevich", 3, 7, params="regular")],
                             [connection("c", "a", "b", "fully connected")]))
    net.build_state()

    def moved():
        return int(net.run({"modules": []}, {"iterations": 2}).properties["moved bytes"])

    assert moved() == 0
    net.get_neuron_data("s", "b", "voltage")
    assert moved() == 4 * 21
    net.get_neuron_data("s", "b", "voltage")
    net.get_weight_matrix("c")
    assert moved() == 4 * (21 + 35 * 21)


# a whole run of a board goes on in pieces between which an interrupt is seen, as it is
# between single steps (20 million steps of the ragged board take some 10 s)
@pytest.mark.parametrize("rows,cols", [(40, 33), (64, 64)])
def test_interrupt_of_whole_runs(sg, rows, cols):
    import threading
    import time
    net = sg.Network(network([layer("b", "game_of_life", rows, cols)],
                             [connection("c", "b", "b", "convergent", convolutional=True, **{
                                 "weight config": {"type": "flat", "weight": 1.0, "diagonal": False},
                                 "arborized config": {"field size": 3, "wrap": True}})]))
    net.build_state()
    net.run({"modules": []}, {"iterations": 10})
    steps = 20_000_000
    timer = threading.Timer(0.5, sg.interrupt_engine)
    timer.start()
    before = time.perf_counter()
    report = net.run({"modules": []}, {"iterations": steps})
    seconds = time.perf_counter() - before
    timer.join()
    assert 0 < int(report.properties["iterations"]) < steps and seconds < 5, (report.properties, seconds)
    # and the next run is whole again
    assert int(net.run({"modules": []}, {"iterations": 100_000}).properties["iterations"]) == 100_000


# a step's kernels as programmatic dependents inside graphs: dendritic trees and second
# order (copies among the kernels), sparse connections, every model and kind of structure,
# learning on one stream and on the side one
@pytest.mark.parametrize("name", ["base_all_types", "iz_c0_8", "iz_plastic", "iz_subset_columns", "iz_opcodes",
                                  "dendrites", "second_order", "sparse", "models", "spnet", "oscillator_som", "nvm",
                                  "structures", "debug"])
def test_graphs_equal_plain_launches(sg, name):
    import copy
    from tests.golden.cases import CASES, Case
    from tests.harness import compare, float_like_keys, run_library
    base = CASES[name]
    net = copy.deepcopy(base.net)
    for i, l in enumerate(l for s in net["structures"] for l in s["layers"]):
        if l["name"] in base.inputs:           # driven by noise in the place of a callback
            l["init config"] = {"type": "poisson", "rate": 200, "value": 15, "seed": 60 + i}
    case = Case(name, net, 75, base.seed, inject=base.inject, final=base.final, learning=base.learning)
    plain = run_library(case, sg, extra_args={"graphs": False, "overlap learning": False})
    for more in ({"overlap learning": False}, {"overlap learning": True}, {"overlap learning": True, "graphs": False}):
        problems = compare(run_library(case, sg, extra_args=dict({"graphs": True}, **more)), plain,
                           nan_keys=float_like_keys(case))
        assert not problems, (more, problems[:3])
