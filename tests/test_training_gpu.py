"""Whole training runs: the reference's own graph/autograd/optimiser code drives
the B200 backend through the vkml::Backend adapter (registered as a second
device), and the same run on the reference CPU backend is the oracle.  Same
graphs, same bytes in, loss curves compared step by step: the device-vs-CPU
training parity of vkML's suite (tests/python/test_vulkan_kernels.py:1575-1603,
tests/python/test_nn_vs_torch.py:344-398)."""
import os

import numpy as np
import pytest

import training
from helpers import REF_B200_SO

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib():
    if not os.path.exists(REF_B200_SO):
        pytest.skip("oracle/_ref/libvkml_ref_b200.so not built")
    return training.load(with_b200=True)


def rel(a, b):
    return np.max(np.abs(a - b) / np.maximum(np.abs(b), 1e-12))


def test_mnist_mlp_100_steps_loss_curve(lib):
    """MLP 784-128-10, batch 64, SGD lr 0.1 momentum 0.9, 100 steps: loss within 1e-4
    relative at every step, parameters within 1e-4 at the end."""
    widths, batch, steps = [784, 128, 10], 64, 100
    ws, bs, x, y = training.mlp_problem(widths, batch, steps)
    cpu_l, cpu_w, cpu_b = training.train_mlp(lib, training.CPU, widths, ws, bs, x, y, batch, steps)
    gpu_l, gpu_w, gpu_b = training.train_mlp(lib, training.B200, widths, ws, bs, x, y, batch, steps)
    assert np.all(np.isfinite(cpu_l)) and cpu_l[-1] < cpu_l[0] + 1.0
    assert rel(gpu_l, cpu_l) < 1e-4, (gpu_l[:5], cpu_l[:5])
    np.testing.assert_allclose(gpu_w, cpu_w, rtol=0, atol=1e-4)
    np.testing.assert_allclose(gpu_b, cpu_b, rtol=0, atol=1e-4)


def test_wide_mlp_reduced_tensor_core_path(lib):
    """The wide-MLP structure (4 Linear layers, ReLU) at widths that send every
    GEMM through the tensor-core path: 100 steps, loss within 1e-4 relative.

    lr 0.02: at lr 0.05 this random-label problem is chaotic enough that ANY change of
    summation order (the plain fp32 FMA kernel included) drifts to 1.5e-4 by step 100,
    so that setting measures the dynamics, not the kernels."""
    widths, batch, steps = [256, 512, 512, 512, 100], 128, 100
    ws, bs, x, y = training.mlp_problem(widths, batch, steps, data="normal")
    cpu_l, cpu_w, _ = training.train_mlp(lib, training.CPU, widths, ws, bs, x, y, batch, steps, lr=0.02)
    gpu_l, gpu_w, _ = training.train_mlp(lib, training.B200, widths, ws, bs, x, y, batch, steps, lr=0.02)
    assert rel(gpu_l, cpu_l) < 1e-4, (gpu_l[-5:], cpu_l[-5:])
    np.testing.assert_allclose(gpu_w, cpu_w, rtol=0, atol=1e-3)


def test_cnn_10_steps(lib):
    """conv3x3-ReLU-pool x3 + Linear (the CIFAR-style CNN at reduced width), conv
    through im2col + batched matmul, backward through col2im and
    max_pool2d_backward: 10 steps, loss within 1e-4 relative."""
    cfg = dict(cin=3, hw=32, c1=16, c2=32, c3=64, classes=100)
    batch, steps = 16, 10
    params, x, y = training.cnn_problem(batch=batch, steps=steps, **cfg)
    cpu_l, cpu_p = training.train_cnn(lib, training.CPU, params=params, x=x, y=y, batch=batch, steps=steps, **cfg)
    gpu_l, gpu_p = training.train_cnn(lib, training.B200, params=params, x=x, y=y, batch=batch, steps=steps, **cfg)
    assert np.all(np.isfinite(cpu_l))
    assert rel(gpu_l, cpu_l) < 1e-4, (gpu_l, cpu_l)
    np.testing.assert_allclose(gpu_p, cpu_p, rtol=0, atol=1e-4)


def _replay_mlp(backend, name, widths, batch, steps, ws, bs, x, y):
    """Replays a recorded program through the C ABI with real data; returns the loss curve."""
    import os
    from vkml_b200.replay import Replayer, load_program
    program = load_program(os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "programs",
                                        name + ".json.gz"))
    assert program["meta"]["widths"] == widths and program["meta"]["batch"] == batch
    params = [p for pair in zip(ws, bs) for p in pair]
    state = {"step": 0}

    def feed(tag, nbytes):
        if tag[0] == "pro":
            arr = params[tag[1]]
        else:
            s = state["step"]
            arr = x[s * batch:(s + 1) * batch] if tag[1] == 0 else y[s * batch:(s + 1) * batch]
        assert arr.nbytes == nbytes, (tag, arr.nbytes, nbytes)
        return arr

    r = Replayer(backend, program, feed)
    for s in range(steps):
        state["step"] = s
        r.step()
    backend.synchronize()
    losses = np.array([d.view(np.float32)[0] for _, d in r.downloads if d.nbytes == 4], dtype=np.float32)
    return losses, r


def test_recorded_program_replays_to_the_same_loss_curve(lib, backend):
    """The MNIST MLP step recorded from the reference framework (its compute spans,
    copies and allocations, captured by a logging backend) and replayed through the C
    ABI gives the CPU backend's loss curve: the replay IS the framework's traffic."""
    widths, batch, steps = [784, 128, 10], 64, 100
    ws, bs, x, y = training.mlp_problem(widths, batch, steps)
    cpu_l, _, _ = training.train_mlp(lib, training.CPU, widths, ws, bs, x, y, batch, steps)
    gpu_l, r = _replay_mlp(backend, "mlp_784_128_10_b64", widths, batch, steps, ws, bs, x, y)
    assert len(gpu_l) == steps
    assert rel(gpu_l, cpu_l) < 1e-4, (gpu_l[:5], cpu_l[:5])
    # steady state allocates nothing new from the driver: every buffer comes from the cache
    before = backend.stats()["driver_allocations"]
    for _ in range(5):
        r.step()
    backend.synchronize()
    assert backend.stats()["driver_allocations"] == before


def test_the_native_tape_replays_what_the_python_replay_does(lib, backend):
    """The library's own step tape (one foreign call per step) and the event-by-event Python
    replay issue the same backend calls: loss curves are bit-identical, for the MLP and the CNN."""
    import os
    from vkml_b200.replay import load_program
    from vkml_b200.tape import Tape
    widths, batch, steps = [784, 128, 10], 64, 30
    ws, bs, x, y = training.mlp_problem(widths, batch, steps)
    py_l, _ = _replay_mlp(backend, "mlp_784_128_10_b64", widths, batch, steps, ws, bs, x, y)
    program = load_program(os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "programs",
                                        "mlp_784_128_10_b64.json.gz"))
    tape = Tape(backend, program)
    tape.run_prologue([p for pair in zip(ws, bs) for p in pair])
    losses = []
    for s in range(steps):
        tape.step([x[s * batch:(s + 1) * batch], y[s * batch:(s + 1) * batch]])
        losses.append(tape.downloads[0].view(np.float32)[0])
    backend.synchronize()
    assert np.array_equal(np.array(losses, dtype=np.float32).view(np.uint32), py_l.view(np.uint32))
    # steady state through the single-call path, with nothing new from the driver
    before = backend.stats()["driver_allocations"]
    xs = np.ascontiguousarray(x[:batch])
    ys = np.ascontiguousarray(y[:batch])
    ptrs = tape.upload_ptrs(tape.template_for_step(steps), [xs.ctypes.data, ys.ctypes.data])
    for _ in range(5):
        tape.step_fast(ptrs)
    backend.synchronize()
    assert backend.stats()["driver_allocations"] == before
    assert np.isfinite(tape.downloads[0].view(np.float32)[0])
    tape.close()


@pytest.mark.parametrize("name", ["mlp_784_128_10_b64", "cnn_reduced_b16", "mlp_wide_reduced_b128"])
def test_graph_replay_is_bit_identical_to_eager_replay(backend, name):
    """Steady-state steps launched as captured CUDA graphs give the same loss bits as the same
    tape run eagerly, with fresh data in the page-locked upload buffers every step."""
    import os
    from vkml_b200.replay import load_program
    from vkml_b200.tape import Tape
    program = load_program(os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "programs",
                                        name + ".json.gz"))
    meta = program["meta"]
    batch, steps = meta["batch"], 24
    rng = np.random.default_rng(77)
    if meta["model"] == "mlp":
        widths = meta["widths"]
        params = []
        for fin, fout in zip(widths[:-1], widths[1:]):
            bound = 1.0 / np.sqrt(fin)
            params.append(rng.uniform(-bound, bound, (fout, fin)).astype(np.float32))
            params.append(rng.uniform(-bound, bound, (fout,)).astype(np.float32))
        x = rng.standard_normal((steps, batch, widths[0])).astype(np.float32)
        classes = widths[-1]
    else:
        cin, hw, classes = meta["cin"], meta["hw"], meta["classes"]
        feat = meta["c3"] * (hw // 8) ** 2
        params = []
        for cout, ci in ((meta["c1"], cin), (meta["c2"], meta["c1"]), (meta["c3"], meta["c2"])):
            bound = 1.0 / np.sqrt(ci * 9)
            params.append(rng.uniform(-bound, bound, (cout, ci, 3, 3)).astype(np.float32))
            params.append(rng.uniform(-bound, bound, (cout,)).astype(np.float32))
        bound = 1.0 / np.sqrt(feat)
        params.append(rng.uniform(-bound, bound, (classes, feat)).astype(np.float32))
        params.append(rng.uniform(-bound, bound, (classes,)).astype(np.float32))
        x = rng.random((steps, batch, cin, hw, hw)).astype(np.float32)
    y = rng.integers(0, classes, (steps, batch)).astype(np.int64)
    pin_x, pin_y = backend.alloc_host(x[0].nbytes), backend.alloc_host(y[0].nbytes)

    def run(graphs):
        tape = Tape(backend, program)
        tape.enable_graphs(graphs)
        tape.run_prologue(params)
        losses = []
        for s in range(steps):
            pin_x[:] = x[s].view(np.uint8).reshape(-1)
            pin_y[:] = y[s].view(np.uint8).reshape(-1)
            tape.step([pin_x.ctypes.data, pin_y.ctypes.data])
            losses.append(tape.downloads[0].view(np.float32)[0].copy())
        backend.synchronize()
        stats = tape.stats()
        tape.close()
        return np.array(losses, dtype=np.float32), stats

    eager, st_e = run(False)
    graph, st_g = run(True)
    assert st_e["graph_launches"] == 0
    assert st_g["graph_launches"] >= steps // 2 and 1 <= st_g["graph_captures"] <= 8, st_g
    assert np.all(np.isfinite(eager))
    assert np.array_equal(eager.view(np.uint32), graph.view(np.uint32)), (eager, graph)
    backend.free_host(pin_x)
    backend.free_host(pin_y)


@pytest.mark.parametrize("name", ["mlp_784_128_10_b64", "cnn_reduced_b16"])
def test_fused_groups_compute_what_the_separate_kernels_do(monkeypatch, name):
    """In-span fusion (bias add + ReLU mask + ReLU, the one-hot mask of cross_entropy, the backward
    of log_softmax) against the same recorded steps with VKML_B200_FUSE=0: fewer launches, and the
    same loss curve -- bit for bit wherever no sum is involved; the fused log_softmax backward adds
    its row in a different (fixed) order, so the curves are held to 1e-6 relative."""
    import vkml_b200
    from vkml_b200.replay import load_program
    from vkml_b200.tape import Tape
    program = load_program(os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "programs",
                                        name + ".json.gz"))
    meta = program["meta"]
    batch, steps = meta["batch"], 12
    rng = np.random.default_rng(5)
    if meta["model"] == "mlp":
        widths = meta["widths"]
        params = []
        for fin, fout in zip(widths[:-1], widths[1:]):
            bound = 1.0 / np.sqrt(fin)
            params += [rng.uniform(-bound, bound, (fout, fin)).astype(np.float32),
                       rng.uniform(-bound, bound, (fout,)).astype(np.float32)]
        x = rng.random((steps, batch, widths[0])).astype(np.float32)
        classes = widths[-1]
    else:
        cin, hw, classes = meta["cin"], meta["hw"], meta["classes"]
        feat = meta["c3"] * (hw // 8) ** 2
        params = []
        for cout, ci in ((meta["c1"], cin), (meta["c2"], meta["c1"]), (meta["c3"], meta["c2"])):
            bound = 1.0 / np.sqrt(ci * 9)
            params += [rng.uniform(-bound, bound, (cout, ci, 3, 3)).astype(np.float32),
                       rng.uniform(-bound, bound, (cout,)).astype(np.float32)]
        bound = 1.0 / np.sqrt(feat)
        params += [rng.uniform(-bound, bound, (classes, feat)).astype(np.float32),
                   rng.uniform(-bound, bound, (classes,)).astype(np.float32)]
        x = rng.random((steps, batch, cin, hw, hw)).astype(np.float32)
    y = rng.integers(0, classes, (steps, batch)).astype(np.int64)

    def run(fuse):
        monkeypatch.setenv("VKML_B200_FUSE", "1" if fuse else "0")
        b = vkml_b200.Backend(0)
        tape = Tape(b, program)
        tape.run_prologue(params)
        b.set_profiling(True)
        losses = []
        for s in range(steps):
            tape.step([np.ascontiguousarray(x[s]), np.ascontiguousarray(y[s])])
            losses.append(tape.downloads[0].view(np.float32)[0].copy())
        labels = [l for l, _ in b.last_profile()]
        b.set_profiling(False)
        tape.close()
        return np.array(losses, dtype=np.float32), labels

    plain, plain_labels = run(False)
    fused, fused_labels = run(True)
    assert not any(l.startswith("fused.") for l in plain_labels)
    assert "fused.log_softmax_backward" in fused_labels, sorted(set(fused_labels))
    # the loss's prologue, from its scalar fills to the one-hot mask and its product, is one launch
    assert "fused.loss_head" in fused_labels and "fused.scaled_add_group" in fused_labels, sorted(set(fused_labels))
    # the bias / mask / relu group appears in whichever form the span holds it
    assert any(l in ("fused.bias_mask_relu", "fused.bias_mask", "fused.bias_relu", "fused.mask") for l in fused_labels)
    assert len(fused_labels) <= len(plain_labels) - 12 * steps, (len(fused_labels), len(plain_labels))
    assert np.all(np.isfinite(plain))
    np.testing.assert_allclose(fused, plain, rtol=1e-6, atol=0)


def test_steps_on_resident_inputs_are_the_uploaded_ones():
    """The program whose inputs lie in the prologue gives the losses of the one that uploads the same batch every step."""
    import vkml_b200
    from vkml_b200.replay import load_program, with_resident_inputs
    from vkml_b200.tape import Tape
    program = load_program(os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "programs", "mlp_784_128_10_b64.json.gz"))
    meta, rng = program["meta"], np.random.default_rng(6)
    params = []
    for fin, fout in zip(meta["widths"][:-1], meta["widths"][1:]):
        params += [rng.uniform(-1, 1, s).astype(np.float32) / np.float32(np.sqrt(fin)) for s in ((fout, fin), (fout,))]
    x, y = rng.random((meta["batch"], meta["widths"][0]), dtype=np.float32), rng.integers(0, meta["widths"][-1], meta["batch"]).astype(np.int64)
    losses = []
    for resident in (False, True):
        tape = Tape(vkml_b200.Backend(0), with_resident_inputs(program) if resident else program)
        tape.run_prologue(params + ([x, y] if resident else []))
        losses.append([])
        for _ in range(8):
            tape.step([] if resident else [x, y])
            losses[-1].append(tape.downloads[0].view(np.float32)[0].copy())
        tape.close()
    assert np.array_equal(np.array(losses[0]).view(np.uint32), np.array(losses[1]).view(np.uint32)) and losses[0][-1] < losses[0][0]


def test_a_run_of_tiny_nodes_is_one_launch(monkeypatch):
    """The single-block chain, on a run that is no loss's prologue: every node's bits those of its own kernel."""
    import vkml_b200
    from vkml_b200 import DeviceTensor, DType, NodeDesc, Op, graph
    rng = np.random.default_rng(2)
    x, k = rng.standard_normal((37, 11), dtype=np.float32), rng.integers(-3, 40, 37)
    x[3, 4], x[5, 6], x[7] = np.inf, np.nan, -0.0

    def run(fuse):
        monkeypatch.setenv("VKML_B200_FUSE", fuse)
        b = vkml_b200.Backend(0)
        dx, dk, nodes, outs = DeviceTensor.from_host(b, x), DeviceTensor.from_host(b, k), [], []

        def node(op, dims, srcs=(), params=b"", dtype=DType.F32):
            outs.append(DeviceTensor.empty(b, dims, dtype))
            nodes.append(NodeDesc(int(op), outs[-1].desc, [s.desc for s in srcs], params))
            return outs[-1]

        wide = node(Op.CAST, (37,), [dk]).reshape((37, 1)).broadcast_to((37, 11))
        steps = node(Op.ARANGE, (11,), params=graph.arange_params(-0.5, 0.1)).broadcast_to((37, 11))
        t = node(Op.NEG, (37, 11), [node(Op.MUL, (37, 11), [wide, dx])])
        t = node(Op.DIV, (37, 11), [t, steps])
        node(Op.CAST, (37, 11), [node(Op.EQUAL, (37, 11), [t, wide], dtype=DType.BOOL)])
        node(Op.CONTIGUOUS, (11, 37), [t.transpose(0, 1)])
        b.set_profiling(True)
        b.compute(nodes)
        labels = [l for l, _ in b.last_profile()]
        b.set_profiling(False)
        return [o.numpy().view(np.uint8) for o in outs], labels

    plain, plain_labels = run("0")
    fused, fused_labels = run("1")
    assert fused_labels == ["fused.tiny_chain"] and len(plain_labels) == 8, (fused_labels, plain_labels)
    for i, (got, want) in enumerate(zip(fused, plain)):
        assert np.array_equal(got, want), i
