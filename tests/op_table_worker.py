"""One training step (or prediction) per case through the op table, by the host
program of perf/cases.py, against the numpy oracle in float64.  Run as a process
of its own (a process holds one enabled backend): cases as JSON on the command
line, one JSON line of errors per case on stdout."""
import ctypes
import importlib.util
import json
import os
import sys

import numpy as np

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, REPO)
os.chdir(REPO)
from oracle import vit_oracle as vo  # noqa: E402

spec = importlib.util.spec_from_file_location(
    "perf_cases", os.path.join(REPO, "perf", "cases.py"))
cases = importlib.util.module_from_spec(spec)
spec.loader.exec_module(cases)

# The oracle's names of the parameters.
NAMES = {"class_token": "cls_token", "positions": "positional"}
BLOCK = {"qkv": "query_key_value", "out": "attention_output", "fc1": "mlp_input",
         "fc2": "mlp_output", "norm1": "attention", "norm2": "mlp"}


def oracle_name(name):
    if "." not in name:
        return NAMES.get(name, name)
    layer, rest = name.split(".")
    head, _, tail = rest.partition("_")
    return f"{layer}.{BLOCK[head]}" + (f"_{tail}" if tail else "")


def larger(worst, error):
    """The larger of two errors; not a number if either is (max would drop it)."""
    return float(np.maximum(worst, error))


def batch_of(state, case, k):
    if state.resident is None:
        labels = state.labels[k].astype(int) if case["kind"] == "train" else None
        return state.images[k].astype(np.float64), labels
    images = np.empty((case["batch"], case["size"] ** 2), np.float32)
    labels = np.empty(case["batch"], np.uintp)
    state.resident.batch(33 + k * case["batch"], case["batch"],
                         images.ctypes.data_as(ctypes.c_void_p),
                         cases._label_pointer(labels))
    return images.astype(np.float64), labels.astype(int)


def augmentation_errors(case):
    """The batch against the oracle: largest difference, and whether the random
    stream ends where the oracle's does."""
    from oracle import augmentation_oracle as ao
    backend = cases._the_host().backend
    shape = (case["batch"], case["channels"], case["height"], case["width"])
    source = np.random.RandomState(5).rand(*shape).astype(np.float32)
    expected, expected_state = ao.apply(case["settings"], 77, source)
    status, out, state = backend.augment(case["settings"], 77, source)
    return {"status": status, "stream": int(state != expected_state),
            "pixel": float(np.abs(out - expected).max())}


def shared_allocations(case):
    """Weights at the front of an allocation that holds more: a step updates them like
    weights with one of their own and leaves the rest alone.  Returns how many of
    either differ."""
    rest = 1000
    states = [cases.prepare(case, 3) for _ in range(2)]
    for name, p in states[1].model.parameters.items():
        count = p.rows * p.cols
        memory = cases._Memory(count + rest)
        memory.array()[:count] = p.data.array()
        memory.array()[count:] = np.arange(rest)
        p.data, p.struct.data = memory, memory.address
    for _ in range(3):
        for state in states:
            state.train()
    plain, shared = (state.model.parameters for state in states)
    found = {"values": 0, "rest": 0}
    for name, p in plain.items():
        count = p.rows * p.cols
        found["values"] += int((shared[name].data.array()[:count] != p.data.array()).sum())
        found["rest"] += int((shared[name].data.array()[count:] != np.arange(rest)).sum())
    return found


def gelu_parameter_errors():
    """Two products of GELU outputs, the first of which is a parameter itself: its
    gradient is a pending definition that reads the first weights, the second weights
    have one too, and the optimiser gets them in the order (weights, GELU output,
    weights).  Largest error of each after the step, in learning rates."""
    rng = np.random.default_rng(11)
    host, n, k, m = cases._the_host(), 64, 32, 48
    host.configure({"precision": "fp32", "deferred": False})
    tensors = {name: cases._Tensor(*shape) for name, shape in (
        ("h1", (n, k)), ("h2", (n, k)), ("a2", (n, k)), ("y1", (n, m)), ("y2", (n, m)))}
    parameters = {name: cases._Parameter(*shape) for name, shape in (
        ("w1", (k, m)), ("a1", (n, k)), ("w2", (k, m)))}
    both = {**tensors, **parameters}
    values = {name: rng.standard_normal((t.rows, t.cols)).astype(np.float32)
              for name, t in both.items()}
    for name, t in both.items():
        t.array()[:] = values[name]
    for p in parameters.values():
        p.m.array()[:] = 0.0
        p.v.array()[:] = 0.0
        p.parameter.step = 1

    def op(slot, *arguments):
        assert host.ops[slot](host.table_context, *arguments) == 0, slot

    pointer = {name: t.pointer for name, t in both.items()}
    kept = cases._pointers(list(pointer.values()))
    op("zero_gradients", ctypes.addressof(kept), len(kept))
    for i in "12":
        op("gelu", pointer["h" + i], pointer["a" + i])
        op("gemm", pointer["a" + i], pointer["w" + i], pointer["y" + i])
    dy = {i: rng.standard_normal((n, m)).astype(np.float32) for i in "12"}
    for i in "12":
        tensors["y" + i].grad.array()[:] = dy[i].ravel()
        op("gemm_backward", pointer["a" + i], pointer["w" + i], pointer["y" + i])
        op("gelu_backward", pointer["h" + i], pointer["a" + i])
    table = cases._pointers([parameters[name].pointer for name in ("w1", "a1", "w2")])
    decays = (ctypes.c_float * 3)(0.0, 0.0, 0.0)
    op("adamw_step_parameters", ctypes.addressof(table), ctypes.addressof(decays), 3,
       cases.LEARNING_RATE, 0.9, 0.999, 1e-8, 0.0)
    host.synchronize()
    found = {}
    activated = {i: vo.gelu(values["h" + i].astype(np.float64)) for i in "12"}
    for name, value, gradient in (
            ("w1", values["w1"], activated["1"].T @ dy["1"]),
            ("a1", activated["1"], dy["1"].astype(np.float64) @ values["w1"].T),
            ("w2", values["w2"], activated["2"].T @ dy["2"])):
        want, _, _ = vo.adamw_update(value.astype(np.float64), gradient, 0.0 * gradient,
                                     0.0 * gradient, 1, cases.LEARNING_RATE, 0.0)
        found[name] = float(np.abs(parameters[name].array() - want).max()
                            / cases.LEARNING_RATE)
    return found


def slope_product_errors(case):
    """A product behind a GELU and a bias, backward, in FP32: the gradient before the
    GELU and its column sums, the weights' gradient and the skipped gradient, each
    against its largest entry."""
    rng = np.random.default_rng(case["m"])
    host, m, k, n = cases._the_host(), case["m"], case["k"], case["n"]
    host.configure({"precision": "fp32", "deferred": False})
    tensors = {name: cases._Tensor(*shape) for name, shape in (
        ("hidden", (m, k)), ("bias", (1, k)), ("activated", (m, k)), ("w", (k, n)),
        ("y", (m, n)))}
    pointer = {name: t.pointer for name, t in tensors.items()}

    def op(slot, *arguments):
        assert host.ops[slot](host.table_context, *arguments) == 0, slot

    kept = cases._pointers(list(pointer.values()))
    op("zero_gradients", ctypes.addressof(kept), len(kept))
    values = {name: rng.standard_normal((t.rows, t.cols)).astype(np.float32)
              for name, t in tensors.items()}
    for name in ("hidden", "w"):
        tensors[name].array()[:] = values[name]
    op("gelu", pointer["hidden"], pointer["activated"])
    op("gemm", pointer["activated"], pointer["w"], pointer["y"])
    tensors["y"].grad.array()[:] = values["y"].ravel()
    fused = host.backend.fusion_counters()["epilogues"]
    op("gemm_backward", pointer["activated"], pointer["w"], pointer["y"])
    if "read_under" in case:   # the product is still held back
        host.backend.set_gemm_precision(case["read_under"])
        host.options = None
        want = values["y"].astype(np.float64) @ values["w"].astype(np.float64).T
        got = tensors["activated"].grad.array().reshape(want.shape)
        return {"activated": float(np.abs(got - want).max() / np.abs(want).max())}
    op("gelu_backward", pointer["hidden"], pointer["activated"])
    op("bias_add_backward", pointer["hidden"], pointer["bias"])
    host.synchronize()
    found = {"fused": host.backend.fusion_counters()["epilogues"] - fused}
    hidden, w, dy = (values[name].astype(np.float64) for name in ("hidden", "w", "y"))
    skipped = dy @ w.T
    before = vo.gelu_backward(hidden, skipped)
    for name, want in (("hidden", before), ("bias", before.sum(axis=0, keepdims=True)),
                       ("w", vo.gelu(hidden).T @ dy), ("activated", skipped)):
        got = tensors[name].grad.array().reshape(want.shape)
        found[name] = float(np.abs(got - want).max() / np.abs(want).max())
    return found


def gradient_pair_errors(case):
    """Both gradients of a product, twice (the weights' add up, the input's starts from
    zero again): largest errors against the largest entry, and the kernels of the second
    pass."""
    rng = np.random.default_rng(case["m"])
    host, m, k, n = cases._the_host(), case["m"], case["k"], case["n"]
    host.configure({"precision": case["precision"], "deferred": False})
    tensors = {name: cases._Tensor(*shape) for name, shape in (
        ("x", (m, k)), ("w", (k, n)), ("y", (m, n)))}
    values = {name: rng.standard_normal((t.rows, t.cols)).astype(np.float32)
              for name, t in tensors.items()}
    pointer = {name: t.pointer for name, t in tensors.items()}

    def op(slot, *arguments):
        assert host.ops[slot](host.table_context, *arguments) == 0, slot

    for name in ("x", "w"):
        tensors[name].array()[:] = values[name]
    kept = cases._pointers([pointer["x"], pointer["w"]])
    op("zero_gradients", ctypes.addressof(kept), 2)
    tensors["y"].grad.array()[:] = values["y"].ravel()
    for _ in range(2):
        op("zero_gradient", pointer["x"])
        host.synchronize()
        launches = host.backend.kernel_launches()
        op("gemm_backward", pointer["x"], pointer["w"], pointer["y"])
        host.synchronize()
    found = {"kernels": host.backend.kernel_launches() - launches}
    x, w, dy = (values[name].astype(np.float64) for name in ("x", "w", "y"))
    for name, want in (("x", dy @ w.T), ("w", 2.0 * (x.T @ dy))):
        got = tensors[name].grad.array().reshape(want.shape)
        found[name] = float(np.abs(got - want).max() / np.abs(want).max())
    return found


def skipped_gradients(case):
    """The gradients of the GELU outputs, which no kernel stores, read after the
    optimiser has moved the weights they are defined by: largest error against
    dY W^T with the weights of before the step, and against those of after it; and how
    many definitions a block and step make, and the reads compute."""
    state = cases.prepare(case, 3)
    tensors, parameters = state.model.tensors, state.model.parameters
    counters = state.host.backend.elision_counters
    state.train()   # (the first step uploads)
    found = {"before": 0.0, "after": 0.0}
    old = {name: np.array(p.array(), np.float64) for name, p in parameters.items()}
    start = counters()
    state.train()
    end = counters()
    if "read_under" in case:   # another policy by the time they are read
        state.host.backend.set_gemm_precision(case["read_under"])
        state.host.options = None
    found["defined"] = (end["lazy_defined"] - start["lazy_defined"]) / case["layers"]
    for layer in range(case["layers"]):
        activated, branch = (
            tensors["%d.%s" % (layer, name)] for name in ("activated", "branch2"))
        dy = branch.grad.array().astype(np.float64).reshape(branch.rows, branch.cols)
        start = counters()
        dx = activated.grad.array().astype(np.float64).reshape(activated.rows, -1)
        found["computed"] = counters()["lazy_materialised"] - start["lazy_materialised"]
        name = "%d.fc2" % layer
        for key, w in (("before", old[name]), ("after", parameters[name].array())):
            want = dy @ w.astype(np.float64).T
            found[key] = larger(found[key], np.abs(dx - want).max() / np.abs(want).max())
    return found


def errors(case):
    if case["kind"] == "slope_product":
        return slope_product_errors(case)
    if case["kind"] == "gradient_pair":
        return gradient_pair_errors(case)
    if case["kind"] == "gelu_parameter":
        return gelu_parameter_errors()
    if case["kind"] == "augment":
        return augmentation_errors(case)
    if case.get("shared_allocations"):
        return shared_allocations(case)
    if case.get("skipped_gradients"):
        return skipped_gradients(case)
    state = cases.prepare(case, 3)
    model = state.model
    declined = state.host.backend.declined_ops()
    config = (case["channels"], case["size"], case["size"], case["patch"],
              case["width"], case["heads"], case["layers"], case["classes"])

    def double(memory, parameter):
        return memory.array().astype(np.float64).reshape(parameter.rows, parameter.cols)

    params = {oracle_name(n): double(p.data, p) for n, p in model.parameters.items()}
    first = {n: double(p.m, p) for n, p in model.parameters.items()}
    second = {n: double(p.v, p) for n, p in model.parameters.items()}
    micro = case.get("micro", 1)
    if case["kind"] == "predict":
        want, _ = vo.forward(params, config, batch_of(state, case, 0)[0])
        got = np.array(cases.run(state))
        return {"logits": float(np.abs(got - want).max() / np.abs(want).max())}
    weights = None
    if case["weights"]:
        weights = model.tensors["class_weights"].data.array().astype(np.float64)
    losses, grads = [], {}
    for k in range(micro):
        loss, g, _ = vo.loss_and_gradients(params, config, *batch_of(state, case, k),
                                           weights, cases.SMOOTHING)
        losses.append(float(loss))
        for name, value in g.items():
            grads[name] = grads.get(name, 0.0) + value / micro
    scale, _ = vo.clip_scale(list(grads.values()), cases.CLIP_NORM)
    got = cases.run(state)
    worst = {"loss": float(abs(got["loss"] - np.mean(losses))), "gradient": 0.0,
             "moment": 0.0, "value": 0.0}
    d = case["width"]
    for name, p in model.parameters.items():
        want = grads[oracle_name(name)] * float(scale)
        value, m, v = vo.adamw_update(
            params[oracle_name(name)], want, first[name], second[name],
            cases.STEPS_TAKEN + 1, cases.LEARNING_RATE,
            cases.WEIGHT_DECAY if cases._parameter_shapes(case)[name][2] else 0.0)
        # The gradient itself is zero again after the step; the first moment
        # holds a tenth of it.
        gradient = (double(p.m, p) - 0.9 * first[name]) / 0.1
        change = np.abs(got[name].reshape(value.shape) - value)
        moment = np.abs(double(p.v, p) - v)
        if name.endswith("qkv_bias"):
            # The key bias has no gradient: what is there is rounding.
            cut = np.s_[d:2 * d]
            gradient, want = np.delete(gradient, cut, 1), np.delete(want, cut, 1)
            change, moment, v = (np.delete(x, cut, 1) for x in (change, moment, v))
        largest = max(float(np.abs(want).max()), 1e-6)
        for key, error in (("gradient", np.abs(gradient - want).max() / largest),
                           ("moment", moment.max() / np.abs(v).max()),
                           ("value", change.max() / cases.LEARNING_RATE)):
            worst[key] = larger(worst[key], error)
    worst["declined"] = state.host.backend.declined_ops() - declined
    return worst


if __name__ == "__main__":
    for one in json.loads(sys.argv[1]):
        print(json.dumps(errors(one)), flush=True)
    os._exit(0)
