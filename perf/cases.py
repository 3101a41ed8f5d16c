"""What a user of the backend has it do, as cases that can be timed and compared.

Four kinds of call, each through the public entry points (the C ABI, `CudaBackend`, `AotExecutor`):

  linear   one quantized Linear on device pointers, `fnn_cuda_qmatmul_ptr`, as an embedding program
           calls it between its own kernels
  mlp      a stack of (up, activation) and (down, residual add) pairs: a plan of `CallKernel`s dispatched
           once and then replayed as one captured graph, the way the executor replays a static plan
  decoder  the projections of decoder layers with the row kernels between them, replayed as one graph
  host     `AotExecutor.forward_pinned`: pinned host input to pinned host output

Weights are drawn on the GPU and packed there into the reference's rows with the quantization pass's
formulas (the host pass is a compile-time step and takes seconds on the largest layers); the `host` kind
goes through the whole compiler with the host pass.
"""
import ctypes
import math

import numpy as np
import torch

import fastnn_b200 as fnn
from fastnn_b200 import _lib as L

FORMATS = {"i8": L.FMT_I8, "i4": L.FMT_I4, "f8": L.FMT_F8, "f4": L.FMT_F4, "i4cb": L.FMT_I4CB}
BITS = {"i8": 8, "i4": 4, "f8": 8, "f4": 4, "i4cb": 4}
KERNELS = {"i8": "matmul_i8", "i4": "matmul_i4", "f8": "matmul_f8", "f4": "matmul_f4", "i4cb": "matmul_i4"}
ACTS = {"none": L.EPI_NONE, "relu": L.EPI_RELU, "gelu": L.EPI_GELU, "silu": L.EPI_SILU}


# ------------------------------------------------------------------------------ the cases


def listed():
    return [
        # the smallest call: one I4 layer with its bias for a batch of eight, where launches and latency count
        {"name": "linear_i4_m8", "kind": "linear", "fmt": "i4", "m": 8, "k": 4096, "n": 4096, "act": "none",
         "bias": True},
        # one request through the executor, host memory to host memory
        {"name": "host_i8_m1", "kind": "host", "fmt": "i8", "m": 1, "k": 4096, "n": 11008, "act": "silu",
         "bias": False},
        # single-stream decoding: I8 feed-forward blocks at one row, bound by the scan of the weights
        {"name": "mlp_i8_m1", "kind": "mlp", "fmt": "i8", "m": 1, "k": 4096, "n": 11008, "act": "silu", "pairs": 6},
        # the same blocks serving sixteen requests at once
        {"name": "mlp_i8_m16", "kind": "mlp", "fmt": "i8", "m": 16, "k": 4096, "n": 11008, "act": "silu",
         "pairs": 6},
        # prompt processing with I8 weights
        {"name": "linear_i8_m512", "kind": "linear", "fmt": "i8", "m": 512, "k": 4096, "n": 11008, "act": "silu",
         "bias": False},
        # a large FP8 layer at one row, and the largest call: the same layer on a long prompt
        {"name": "linear_f8_m1", "kind": "linear", "fmt": "f8", "m": 1, "k": 8192, "n": 28672, "act": "none",
         "bias": False},
        {"name": "linear_f8_m4096", "kind": "linear", "fmt": "f8", "m": 4096, "k": 8192, "n": 28672, "act": "none",
         "bias": False},
        # the FP4 layer for a few requests, and an FP4 layer of odd sizes on a prompt of odd length
        {"name": "linear_f4_m4", "kind": "linear", "fmt": "f4", "m": 4, "k": 8192, "n": 28672, "act": "none",
         "bias": False},
        {"name": "ragged_f4_m333", "kind": "linear", "fmt": "f4", "m": 333, "k": 5000, "n": 13001, "act": "gelu",
         "bias": True},
        # the codebook MLP stack at its batch of 64, and at one row
        {"name": "mlp_i4cb_m64", "kind": "mlp", "fmt": "i4cb", "m": 64, "k": 2048, "n": 8192, "act": "gelu",
         "pairs": 6},
        {"name": "mlp_i4cb_m1", "kind": "mlp", "fmt": "i4cb", "m": 1, "k": 2048, "n": 8192, "act": "gelu",
         "pairs": 6},
        # four decoder layers of the 8B dimensions, I4 weights, decoding a batch of 64
        {"name": "decoder_i4_m64", "kind": "decoder", "fmt": "i4", "m": 64, "k": 4096, "n": 14336, "act": "silu",
         "layers": 4},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng, lo, hi):
    """Log-uniform; half of the draws are layer-like multiples of 128 (of 16 when small), half are odd."""
    v = _log(rng, lo, hi)
    if rng.random() < 0.5:
        step = 128 if v >= 512 else 16
        return max(step, v // step * step)
    return max(lo, v | 1 if rng.random() < 0.5 else v)


def draw(rng):
    kind = rng.choice(["linear"] * 5 + ["mlp"] * 3 + ["decoder"] * 2 + ["host"])
    fmt = rng.choice(list(FORMATS))
    act = rng.choice(list(ACTS))
    if kind == "linear":
        m = _log(rng, 1, 4096)
        k, n = _size(rng, 192, 14336), _size(rng, 512, 28672)
        return {"kind": kind, "fmt": fmt, "m": m, "k": min(k, 8192) if m > 2048 else k, "n": n, "act": act,
                "bias": rng.random() < 0.5}
    if kind == "mlp":
        k = _size(rng, 512, 4096)
        n = int(k * rng.choice([2, 2.6875, 4]))
        return {"kind": kind, "fmt": fmt, "m": _log(rng, 1, 512), "k": k, "n": n,
                "act": rng.choice(["relu", "gelu", "silu"]), "pairs": rng.randint(2, 6)}
    if kind == "decoder":
        k = rng.choice([1024, 2048, 3072, 4096])
        return {"kind": kind, "fmt": fmt, "m": _log(rng, 1, 256), "k": k,
                "n": int(k * rng.choice([2.75, 3.5, 4])), "act": "silu", "layers": rng.randint(1, 4)}
    fmt = rng.choice(["i8", "i4", "f8", "f4"])   # the codebook's host pass takes seconds
    return {"kind": kind, "fmt": fmt, "m": _log(rng, 1, 64), "k": _size(rng, 512, 4096), "n": _size(rng, 1024, 11008),
            "act": act, "bias": rng.random() < 0.5}


def _layers(case):
    """(K, N) of every weight of one pass."""
    k, n = case["k"], case["n"]
    if case["kind"] == "mlp":
        return [(k, n), (n, k)] * case["pairs"]
    if case["kind"] == "decoder":   # q/k/v with grouped keys and values, output, gate/up, down
        return [(k, k + k // 2), (k, k), (k, 2 * n), (n, k)] * case["layers"]
    return [(k, n)]


def _sigma(case):
    return 0.015 if case["k"] >= 8192 else 0.02


def work(case):
    """Packed weights with their scales once, the input once, the output once; two operations per
    weight and row."""
    m, total, flops = case["m"], 0, 0
    for k, n in _layers(case):
        total += n * k * BITS[case["fmt"]] // 8
        total += {"i8": 8 * n, "i4": 8 * n, "f4": 8 * n, "f8": 4 * n, "i4cb": 4 * n * -(-k // 32)}[case["fmt"]]
        if case.get("bias") or case["kind"] == "mlp":
            total += 4 * n
        flops += 2 * m * k * n
    k_in = case["k"]
    n_out = case["n"] if case["kind"] in ("linear", "host") else case["k"]
    return {"bytes": total + 4 * m * (k_in + n_out), "flops": flops}


def tolerance(case):
    """About four times the relative error measured against the f32 row kernel on the same inputs.  f32
    activations reach the tensor cores as 15-bit fixed point (I8, I4, FP4 and the codebook at few rows:
    7e-5), as two e4m3 terms (FP8, FP4 from 128 rows: 6.4e-4) or three (1e-5), or as fp16 beside fp16 weights
    (codebook: 3e-4).  A stack adds its layers' errors up (six I8 pairs: 2.7e-4; four decoder layers: 3.3e-4)."""
    fmt, m = case["fmt"], case["m"]
    if fmt == "f8":
        one = 2.5e-3 if m >= 128 else 5e-5
    else:
        one = {"i8": 3e-4, "i4": 3e-4, "f4": 2.5e-3 if m >= 128 else 3e-4, "i4cb": 1.2e-3}[fmt]
    if case["kind"] in ("linear", "host"):
        return {"rel": one}
    depth = 2 * case["pairs"] if case["kind"] == "mlp" else 4 * case["layers"]
    return {"rel": one * math.sqrt(depth)}


# ------------------------------------------------------------------------------ weights on the GPU

_MAG4 = (0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0)
_BACKEND = None


def _backend():
    """One context for the process, as a serving program has."""
    global _BACKEND
    if _BACKEND is None:
        _BACKEND = fnn.CudaBackend(torch.cuda.current_device())
    return _BACKEND


def _align(v, a=256):
    return -(-v // a) * a


def _nearest(v, points):
    mid = (points[1:] + points[:-1]) / 2
    return torch.bucketize(v, mid)


def _codes(fmt, w):
    """Codes (uint8), scales, zeros and codebook of the f32 rows `w` [n, K] (one channel per row)."""
    none = torch.zeros(0, device=w.device)
    if fmt in ("i8", "i4"):
        levels = 255.0 if fmt == "i8" else 15.0
        lo, hi = w.amin(1), w.amax(1)
        step = (hi - lo) / levels
        lo, hi = lo - step, hi + step
        scale = (hi - lo) / levels
        half = 128.0 if fmt == "i8" else 8.0
        zero = lo + half * scale
        q = ((w - zero[:, None]) / scale[:, None]).round_().clamp_(-half, half - 1)
        return q.to(torch.int8).view(torch.uint8), scale, zero, None
    if fmt == "f8":
        scale = w.abs().amax(1) / 240.0
        return (w / scale[:, None]).to(torch.float8_e4m3fn).view(torch.uint8), scale, none, None
    if fmt == "f4":
        mean = w.mean(1)
        scale = (w - mean[:, None]).abs().amax(1) / 4.0
        v = (w - mean[:, None]) / scale[:, None]
        q = _nearest(v.abs(), torch.tensor(_MAG4, device=w.device))
        return torch.where((v < 0) & (q > 0), q + 8, q).to(torch.uint8), scale, mean, None
    n, k = w.shape   # codebook: absmax of every 32, one 16-entry table of the normalised values
    blocks = -(-k // 32)
    padded = torch.nn.functional.pad(w, (0, blocks * 32 - k)).view(n, blocks, 32)
    scale = padded.abs().amax(2)
    v = (padded / scale[:, :, None]).view(n, blocks * 32)[:, :k]
    table = torch.tensor([-0.95, -0.74, -0.58, -0.45, -0.34, -0.23, -0.135, -0.045, 0.045, 0.135, 0.23, 0.34, 0.45,
                          0.58, 0.74, 0.95], device=w.device)
    return _nearest(v, table).to(torch.uint8), scale.reshape(-1), none, table


def _packed_bytes(fmt, k, n):
    return int(L.load().fnn_quant_packed_bytes(FORMATS[fmt], n, k))


def _fill_weight(fmt, k, n, sigma, gen, slot):
    """Draws a weight and writes its packed rows into `slot` (bytes of the arena); returns its metadata."""
    per_word = 32 // BITS[fmt]
    words = -(-k // per_word)
    rows = slot[: n * words * 4].view(n, words * 4)
    scales, zeros, table = [], [], None
    step = max(1, (1 << 26) // k)
    for r in range(0, n, step):
        c = min(step, n - r)
        w = torch.randn((c, k), device=slot.device, generator=gen) * sigma
        q, s, z, table = _codes(fmt, w)
        q = torch.nn.functional.pad(q, (0, words * per_word - k))
        if per_word == 8:
            q = (q[:, 0::2] & 15) | (q[:, 1::2] << 4)
        rows[r:r + c].copy_(q)
        scales.append(s)
        zeros.append(z)
    zeros = torch.cat(zeros).cpu().numpy()
    return fnn.QuantizedWeightMeta(
        bit_width=BITS[fmt], scales=torch.cat(scales).cpu().numpy(), zero_points=zeros, shape=[n, k],
        quant_block_size=32 if fmt == "i4cb" else 0, codebooks=[table.cpu().numpy()] if fmt == "i4cb" else [],
        fmt=FORMATS[fmt])


class _Arena:
    """A plan's arena over one torch allocation: named slots, weights packed in place."""

    def __init__(self, sizes):
        self.slot, top = {}, 0
        for name, size in sizes:
            self.slot[name] = fnn.BufferSlice(top, size)
            top += _align(size)
        self.memory = torch.zeros(max(top, 256), dtype=torch.uint8, device="cuda")
        torch.cuda.synchronize()
        self.backend = _backend()
        self.buffer = self.backend.wrap_arena(self.memory.data_ptr(), self.memory.numel(), self.memory)

    def bytes(self, name):
        s = self.slot[name]
        return self.memory[s.offset: s.offset + s.size]

    def floats(self, name):
        return self.bytes(name).view(torch.float32)

    def ptr(self, name):
        return self.memory.data_ptr() + self.slot[name].offset


class _Graph:
    """Calls recorded once and replayed as one launch."""

    def __init__(self, backend, calls):
        self.backend, self.handle = backend, None
        lib = backend.lib
        calls()                        # first use: layouts, scratch
        backend.synchronize()
        _ok(lib.fnn_cuda_graph_begin(backend.ctx))
        g = ctypes.c_void_p()
        try:
            calls()
        finally:
            rc = lib.fnn_cuda_graph_end(backend.ctx, ctypes.byref(g))
        _ok(rc)
        self.handle = g.value

    def launch(self):
        _ok(self.backend.lib.fnn_cuda_graph_launch(self.backend.ctx, self.handle))

    def __del__(self):
        if self.handle:
            self.backend.lib.fnn_cuda_graph_free(self.handle)
            self.handle = None


def _ok(rc):
    if rc != L.FNN_OK:
        raise fnn.BackendError.from_status(rc)


# ------------------------------------------------------------------------------ prepare and run


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    state = {"linear": _prepare_linear, "mlp": _prepare_mlp, "decoder": _prepare_decoder,
             "host": _prepare_host}[case["kind"]](case, gen)
    torch.cuda.synchronize()
    return state


def run(state):
    return state["run"](state)


def _prepare_linear(case, gen):
    fmt, m, k, n = case["fmt"], case["m"], case["k"], case["n"]
    arena = _Arena([("w", _packed_bytes(fmt, k, n))])
    meta = _fill_weight(fmt, k, n, _sigma(case), gen, arena.bytes("w"))
    torch.cuda.synchronize()
    slot = arena.slot["w"]
    weight = arena.backend.upload_qweight(b"", meta, arena.buffer, slot.offset, slot.size)
    x = torch.randn((m, k), device="cuda", generator=gen)
    bias = torch.randn(n, device="cuda", generator=gen) * 0.01 if case["bias"] else None
    y = torch.empty((m, n), device="cuda")
    backend = arena.backend
    args = (backend.ctx, weight.handle, x.data_ptr(), y.data_ptr(), bias.data_ptr() if case["bias"] else None, m,
            ACTS[case["act"]], L.PATH_AUTO)
    return {"run": _run_linear, "call": backend.lib.fnn_cuda_qmatmul_ptr, "args": args, "y": y,
            "keep": (weight, arena, x, bias)}


def _run_linear(state):
    _ok(state["call"](*state["args"]))
    return state["y"]


def _prepare_mlp(case, gen):
    fmt, m, k, n = case["fmt"], case["m"], case["k"], case["n"]
    sizes = [("x", m * k * 4), ("h", m * n * 4), ("v", m * k * 4), ("r0", m * k * 4), ("r1", m * k * 4)]
    for i in range(case["pairs"]):
        sizes += [(f"up{i}", _packed_bytes(fmt, k, n)), (f"dn{i}", _packed_bytes(fmt, n, k)), (f"bu{i}", n * 4),
                  (f"bd{i}", k * 4)]
    arena = _Arena(sizes)
    plan, cur = [], "x"
    for i in range(case["pairs"]):
        out = f"r{i & 1}"
        for w, b, src, dst, kk, nn, act in ((f"up{i}", f"bu{i}", cur, "h", k, n, case["act"]),
                                            (f"dn{i}", f"bd{i}", "h", "v", n, k, "none")):
            meta = _fill_weight(fmt, kk, nn, 0.02, gen, arena.bytes(w))
            arena.floats(b).normal_(0.0, 0.01, generator=gen)
            plan.append(fnn.CallKernel(KERNELS[fmt], [arena.slot[src], arena.slot[w], arena.slot[b]],
                                       arena.slot[dst], [m, kk, nn, ACTS[act]], weight_meta=meta))
        plan.append(fnn.CallKernel("add_f32", [arena.slot["v"], arena.slot[cur]], arena.slot[out], []))
        cur = out
    arena.floats("x").normal_(generator=gen)
    torch.cuda.synchronize()
    backend = arena.backend
    plan = fnn.ExecutablePlan(plan, arena.memory.numel())
    graph = _Graph(backend, lambda: backend.dispatch(plan, arena.buffer, fnn.ShapeEnv()))
    return {"run": _run_graph, "graph": graph, "y": arena.floats(cur).view(m, k), "keep": arena}


def _run_graph(state):
    state["graph"].launch()
    return state["y"]


def _prepare_decoder(case, gen):
    """Per layer: a = (x Wqkv)[:, :d] (attention itself is not this backend's); r = a Wo + x; g = rms_norm(r) Wgu;
    h = silu(gate) * up; x' = h Wdn + r."""
    fmt, m, d, f = case["fmt"], case["m"], case["k"], case["n"]
    names = ("qkv", "o", "gu", "dn")
    sizes = [("x", d), ("qkv", d + d // 2), ("a", d), ("o", d), ("r", d), ("nrm", d), ("g", 2 * f), ("gate", f),
             ("up", f), ("dn", d), ("y0", d), ("y1", d)]
    sizes = [(s, m * cols * 4) for s, cols in sizes] + [("ones", d * 4)]
    shapes = dict(zip(names, _layers(case)[:4]))
    sizes += [(f"w{i}{name}", _packed_bytes(fmt, *shapes[name])) for i in range(case["layers"]) for name in names]
    arena = _Arena(sizes)
    backend, lib, ctx, buf = arena.backend, arena.backend.lib, arena.backend.ctx, arena.buffer.handle
    off = {name: s.offset for name, s in arena.slot.items()}
    weights = []
    for i in range(case["layers"]):
        for name in names:
            k, n = shapes[name]
            meta = _fill_weight(fmt, k, n, 0.02, gen, arena.bytes(f"w{i}{name}"))
            torch.cuda.synchronize()
            slot = arena.slot[f"w{i}{name}"]
            weights.append(backend.upload_qweight(b"", meta, arena.buffer, slot.offset, slot.size))
    arena.floats("x").normal_(generator=gen)
    arena.floats("ones").fill_(1.0)
    torch.cuda.synchronize()

    def matmul(w, src, dst):
        _ok(lib.fnn_cuda_qmatmul(ctx, w.handle, buf, off[src], off[dst], -1, m, L.EPI_NONE, L.PATH_AUTO))

    def binary(op, a, b, dst, cols):
        _ok(lib.fnn_cuda_elementwise(ctx, op, buf, off[a], m * cols, off[b], m * cols, off[dst], m * cols))

    def columns(src, first, pitch, cols, dst):
        _ok(lib.fnn_cuda_memcpy2d(ctx, buf, off[dst], cols * 4, off[src] + first * 4, pitch * 4, cols * 4, m))

    def calls():
        cur = "x"
        for i in range(case["layers"]):
            qkv, o, gu, dn = weights[4 * i: 4 * i + 4]
            matmul(qkv, cur, "qkv")
            columns("qkv", 0, d + d // 2, d, "a")
            matmul(o, "a", "o")
            binary(L.EW_ADD, "o", cur, "r", d)
            _ok(lib.fnn_cuda_rms_norm(ctx, buf, off["r"], m * d, off["ones"], d, d, 1e-5, off["nrm"]))
            matmul(gu, "nrm", "g")
            columns("g", 0, 2 * f, f, "gate")
            columns("g", f, 2 * f, f, "up")
            binary(L.EW_SILU, "gate", "gate", "gate", f)
            binary(L.EW_MUL, "gate", "up", "gate", f)
            matmul(dn, "gate", "dn")
            binary(L.EW_ADD, "dn", "r", f"y{i & 1}", d)
            cur = f"y{i & 1}"

    graph = _Graph(backend, calls)
    out = f"y{(case['layers'] - 1) & 1}"
    return {"run": _run_graph, "graph": graph, "y": arena.floats(out).view(m, d), "keep": (weights, arena)}


def _prepare_host(case, gen):
    m, k, n = case["m"], case["k"], case["n"]
    w = (torch.randn((k, n), device="cuda", generator=gen) * _sigma(case)).cpu().numpy()
    x = torch.randn((m, k), device="cuda", generator=gen).cpu().numpy()
    nodes = [{"op_type": "Gemm" if case["bias"] else "MatMul", "inputs": "[x, w, b]" if case["bias"] else "[x, w]",
              "outputs": "[h]"}]
    params = {"w": w}
    if case["bias"]:
        params["b"] = (torch.randn(n, device="cuda", generator=gen) * 0.01).cpu().numpy()
    out = "h"
    if case["act"] != "none":
        nodes.append({"op_type": case["act"].capitalize(), "inputs": "[h]", "outputs": "[y]"})
        out = "y"
    quantize = {"i8": 8, "i4": 4}.get(case["fmt"], case["fmt"])
    executor = fnn.AotExecutor(nodes, params, ["x"], [out], {"x": [m, k]}, quantize=quantize, backend=_backend())
    executor.forward({"x": x})     # constants written, layouts built
    executor.bind_pinned()
    return {"run": _run_host, "executor": executor, "x": np.ascontiguousarray(x), "out": out}


def _run_host(state):
    executor = state["executor"]
    executor.pinned_inputs["x"][...] = state["x"]
    return executor.forward_pinned()[state["out"]]
