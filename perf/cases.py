"""Workloads of the quantized gradient aggregation path, for timing one build against another.

A case is a dict of plain values.  Its ``kind`` says which public entry points it goes through:

  matrix  one fp32 gradient matrix: quantize with error feedback, then unquantize (``qagg_quantize`` / ``qagg_unquantize``)
  double  the same for a double matrix (``qagg_quantize_f64`` / ``qagg_unquantize_f64``)
  step    one aggregation step of a whole gradient set on one rank (``Aggregator.step``)
  group   one aggregation step of K ranks in one process with peer-mapped windows, ending in the momentum-SGD update of
          every rank's parameters (``step_group`` with ``set_update``)
  host    one aggregation step of a gradient set held in pinned host memory (``HostAggregator.step``)

``shapes`` lists the tensors as ``rows x columns``, ``*n`` repeating one.  The ranges behind the listed cases, which draw()
samples: 1 to 20000 rows and 1 to 4096 columns of a single matrix (16 to 8 Mi values; double: 2 Mi), sets of 2 to 50 tensors
of 1 Ki to 16 Mi values with layer widths of 16 to 4096 and now and then an embedding of up to 40000 rows, 2 to 8 ranks,
1, 2, 4 or 8 bits, both 1-bit thresholds; half of the sizes are multiples of 8, the others are whatever they are.
"""
import math

import torch

from cntk_b200 import lib, workloads


def _pack(shapes):
    out, i = [], 0
    while i < len(shapes):
        j = i
        while j < len(shapes) and shapes[j] == shapes[i]:
            j += 1
        out.append("%dx%d" % shapes[i] + ("*%d" % (j - i) if j - i > 1 else ""))
        i = j
    return ",".join(out)


def _shapes(case):
    out = []
    for part in case["shapes"].split(","):
        dims, _, times = part.partition("*")
        m, n = dims.split("x")
        out += [(int(m), int(n))] * int(times or 1)
    return out


def _case(name, kind, shapes, bits=1, zero=True, ranks=1, dist="normal", scale=1e-3):
    c = {"kind": kind, "shapes": _pack(shapes), "bits": bits, "zero": zero, "ranks": ranks, "dist": dist, "scale": scale}
    if name:
        c["name"] = name
    return c


def listed():
    # feed-forward net 363:512:512:132 of the data-parallel speech tests: three weights, three biases
    small_dnn = [(512, 363), (512, 512), (132, 512), (512, 1), (512, 1), (132, 1)]
    return [
        # one bias vector: the smallest call a layer-by-layer user makes, nothing but latency
        _case("matrix_bias_512", "matrix", [(512, 1)], scale=0.01),
        # the 2048 x 2048 hidden-layer weight of the quantizer's round-trip configuration
        _case("matrix_2048", "matrix", [(2048, 2048)], scale=0.01),
        # a ragged matrix (no dimension a multiple of 4) with the column-mean threshold, the other 1-bit option
        _case("matrix_ragged_mean", "matrix", [(1001, 517)], zero=False, scale=0.01),
        # double precision, in which the end-to-end speech tests run: their 363 -> 512 layer
        _case("double_512x363", "double", [(512, 363)], scale=0.01),
        # a whole small net in one step: launches and host work count
        _case("step_small_dnn", "step", small_dnn),
        # the headline set: speech feed-forward DNN, 45 M values, 1 bit
        _case("step_speech_dnn", "step", workloads.speech_dnn()),
        # many tensors of very different sizes, 4 bits, heavy-tailed values: ResNet-50
        _case("step_resnet50", "step", workloads.resnet50(), bits=4, dist="laplace", scale=1e-4),
        # very tall and very wide matrices, most embedding columns zero: LSTM language model
        _case("step_lstm_lm", "step", workloads.lstm_lm(), dist="sparse", scale=5e-4),
        # one large matrix at 2 bits: the bandwidth sweep's 64 Mi values
        _case("step_sweep_64m", "step", workloads.sweep(3), bits=2),
        # four data-parallel ranks of the speech set, exchange and learner step included
        _case("group4_speech_dnn", "group", workloads.speech_dnn(), ranks=4),
        # the speech set in host memory: copies in, aggregation and copies out in one call
        _case("host_speech_dnn", "host", workloads.speech_dnn()),
    ]


def _log_int(rng, lo, hi):
    """Log-uniform integer of [lo, hi]; every other one rounded to a multiple of 8 where that stays in range."""
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    if rng.random() < 0.5 and v >= 8:
        v = v // 8 * 8
    return max(lo, min(hi, v))


def _draw_matrix(rng, most):
    while True:
        m, n = _log_int(rng, 1, 20000), _log_int(rng, 1, 4096)
        if 16 <= m * n <= most:
            return [(m, n)]


def _draw_set(rng, most):
    """A chain of layers (weight and bias each), now and then with an embedding in front."""
    while True:
        layers = rng.randint(1, 24)
        widths = [_log_int(rng, 16, 4096)]
        for _ in range(layers):
            # neighbouring layers are mostly of the same width, as in real nets
            widths.append(widths[-1] if rng.random() < 0.5 else _log_int(rng, 16, 4096))
        shapes = []
        if rng.random() < 0.25:
            shapes.append((_log_int(rng, 4096, 40000), _log_int(rng, 8, 256)))
        shapes += [(widths[i + 1], widths[i]) for i in range(layers)]
        shapes += [(widths[i + 1], 1) for i in range(layers)]
        if 1024 <= workloads.total_values(shapes) <= most:
            return shapes


def draw(rng):
    kind = rng.choices(["matrix", "double", "step", "group", "host"], [7, 2, 7, 3, 1])[0]
    bits = rng.choices([1, 2, 4, 8], [6, 1, 2, 1])[0]
    zero = bits > 1 or rng.random() < 0.85
    dist = rng.choice(["normal", "normal", "laplace", "sparse"])
    scale = 10.0 ** rng.uniform(-5, -1)
    if kind == "matrix":
        return _case(None, kind, _draw_matrix(rng, 8 << 20), bits, zero, 1, dist, scale)
    if kind == "double":
        return _case(None, kind, _draw_matrix(rng, 2 << 20), bits, zero, 1, dist, scale)
    if kind == "step":
        return _case(None, kind, _draw_set(rng, 16 << 20), bits, zero, 1, dist, scale)
    if kind == "group":
        return _case(None, kind, _draw_set(rng, 4 << 20), bits, zero, rng.randint(2, 8), dist, scale)
    return _case(None, kind, _draw_set(rng, 8 << 20), bits, zero, 1, dist, scale)


# ---- inputs and handles -------------------------------------------------------------------------------------------------


def _values(shapes, case, seed, dtype=torch.float32):
    """One flat gradient buffer on the GPU (every tensor 16-byte aligned in it) and each tensor's view, stored column by
    column as the library wants them."""
    offsets, total = [], 0
    for m, n in shapes:
        offsets.append(total)
        total += -(-m * n // 4) * 4
    gen = torch.Generator(device="cuda").manual_seed(seed)
    flat = torch.empty(total, dtype=dtype, device="cuda").normal_(0.0, case["scale"], generator=gen)
    if case["dist"] == "laplace":
        # the difference of two exponentials
        flat.exponential_(1.0, generator=gen)
        flat.sub_(torch.empty_like(flat).exponential_(1.0, generator=gen)).mul_(case["scale"])
    views = [flat[o:o + m * n].view(n, m) for o, (m, n) in zip(offsets, shapes)]
    if case["dist"] == "sparse":
        # nine of ten columns of the first tensor (an embedding) saw no sample of this minibatch
        n = shapes[0][1]
        views[0].mul_((torch.rand(n, 1, device="cuda", generator=gen) < 0.1).to(dtype))
    return flat, views


class _Owned:
    """Library handles that go away, in this order, with the state that holds them."""

    def __init__(self, *handles):
        self.handles = handles

    def __del__(self):
        torch.cuda.synchronize()
        for h in self.handles:
            h.destroy()


def _flags(case):
    return lib.SELF_QUANTIZED | (lib.ZERO_THRESHOLD if case["zero"] else 0)


def prepare(case, seed):
    shapes, bits = _shapes(case), case["bits"]
    kind = case["kind"]
    if kind in ("matrix", "double"):
        (m, n), = shapes
        double = kind == "double"
        flat, (grad,) = _values(shapes, case, seed, torch.float64 if double else torch.float32)
        size = lib.packed_bytes_f64(m, n, bits) if double else lib.packed_bytes(m, n, bits)
        # the packed matrix is kept as bytes: its words and its range headers are what travels
        return {"kind": kind, "m": m, "n": n, "bits": bits, "zero": case["zero"], "grad": grad, "residual": torch.zeros_like(grad),
                "packed": torch.zeros(size, dtype=torch.uint8, device="cuda"), "out": torch.zeros_like(grad)}
    if kind == "step":
        flat, views = _values(shapes, case, seed)
        comm = lib.Comm.create(None, 0, 1, 0)
        agg = lib.Aggregator(comm, shapes, bits, _flags(case))
        return {"kind": kind, "agg": agg, "grads": flat, "pointers": [v.data_ptr() for v in views], "owned": _Owned(agg, comm)}
    if kind == "host":
        flat, views = _values(shapes, case, seed)
        base = flat.data_ptr()
        host = torch.empty(flat.numel(), dtype=torch.float32, pin_memory=True)
        host.copy_(flat)
        comm = lib.Comm.create(None, 0, 1, 0)
        agg = lib.HostAggregator(comm, shapes, bits, _flags(case))
        return {"kind": kind, "agg": agg, "grads": host, "pointers": [host.data_ptr() + v.data_ptr() - base for v in views],
                "owned": _Owned(agg, comm)}
    K = case["ranks"]
    comms = lib.Comm.local_group(K, 0)
    aggs = [lib.Aggregator(c, shapes, bits, _flags(case)) for c in comms]
    handles = [a.peer_handle() for a in aggs]
    grads, params, smoothed, pointers = [], [], [], []
    for r, a in enumerate(aggs):
        a.enable_peer(handles)
        flat, views = _values(shapes, case, seed * 64 + r)
        # all ranks start from the same parameters
        gen = torch.Generator(device="cuda").manual_seed(seed)
        w = torch.empty_like(flat).normal_(0.0, 0.05, generator=gen)
        s = torch.zeros_like(flat)
        offsets = [v.data_ptr() - flat.data_ptr() for v in views]
        a.bind_update([w.data_ptr() + o for o in offsets], [s.data_ptr() + o for o in offsets])
        a.set_update(True, 0.02, 0.9, 0.1)
        grads.append(flat)
        params.append(w)
        smoothed.append(s)
        pointers.append([v.data_ptr() for v in views])
    return {"kind": kind, "aggs": aggs, "grads": grads, "params": params, "smoothed": smoothed, "pointers": pointers,
            "owned": _Owned(*aggs, *comms)}


def run(state):
    kind = state["kind"]
    if kind in ("matrix", "double"):
        quantize, unquantize = (lib.quantize_f64, lib.unquantize_f64) if kind == "double" else (lib.quantize, lib.unquantize)
        m, n, bits = state["m"], state["n"], state["bits"]
        residual, packed = state["residual"], state["packed"]
        stream = torch.cuda.current_stream().cuda_stream
        quantize(state["grad"].data_ptr(), residual.data_ptr(), residual.data_ptr(), packed.data_ptr(), m, n, bits, state["zero"], stream)
        unquantize(packed.data_ptr(), state["out"].data_ptr(), m, n, bits, False, stream)
        return {"packed": packed, "residual": residual, "out": state["out"]}
    if kind == "step":
        # the gradients come back aggregated in place; the residuals live inside the handle
        state["agg"].step(state["pointers"], torch.cuda.current_stream().cuda_stream)
        return state["grads"]
    if kind == "host":
        state["agg"].step(state["pointers"])
        return state["grads"]
    lib.step_group(state["aggs"], state["pointers"], torch.cuda.current_stream().cuda_stream)
    return {"params": state["params"], "smoothed": state["smoothed"]}


def work(case):
    shapes, K = _shapes(case), case["ranks"]
    V = workloads.total_values(shapes)
    if case["kind"] == "double":
        (m, n), = shapes
        # gradient, residual in and out, output; the packed matrix written and read
        return {"bytes": 32 * V + 2 * lib.packed_bytes_f64(m, n, case["bits"]), "flops": 6 * V}
    P = workloads.packed_bytes(shapes, case["bits"])
    if case["kind"] == "matrix":
        return {"bytes": 16 * V + 2 * P, "flops": 6 * V}
    if case["kind"] == "step":
        # gradient and residual read and written; the packed form need not leave the chip
        return {"bytes": 16 * V, "flops": 6 * V}
    if case["kind"] == "host":
        # every gradient value crosses the host link both ways
        return {"bytes": 8 * V, "flops": 6 * V}
    # per rank: gradient read, residual, parameter and smoothed gradient read and written, an owner's share of the stripe
    # residuals read and written; packed stripes written and read once in each half of the exchange
    return {"bytes": K * (28 * V + 8 * V / K + 4 * P), "flops": K * (12 * V + 4 * V)}


def tolerance(case):
    # every sum is taken in the reference's order with the reference's roundings: a correct build returns the same bits
    return "exact"
