"""The work that users have this framework do, as cases that can be timed.

Four kinds, all on one GPU and through the public entry points:

* ``rpc``: ``AxonRuntime.invoke`` of a device tensor whose handler returns it, between two runtimes of one
  process. One call or many in flight; dense tensors, tensors that start inside a larger buffer, row slices and
  transposed views; sent as they are or converted on the way (``wire_dtype``).
* ``push``: the transfer kernel as an op (``ops.tensor_xfer.push``): gather, handler and cast in one launch.
* ``gemm``: the remote GEMM in its three formats, as an Axon call (``serve_gemm`` / ``remote_gemm``) or as the op
  of the callee (``ops.remote_gemm``), with X in place or streamed into the staging buffer while the kernel runs.
* ``moe``: dispatch, identity expert and gate-weighted combine (``ops.moe.MoeAllToAll``).
"""
import asyncio
import math

import torch

from execution_ucx_b200 import axon
from execution_ucx_b200.ops import moe as moe_ops
from execution_ucx_b200.ops import remote_gemm as gemm_ops
from execution_ucx_b200.ops import tensor_xfer as tx
from execution_ucx_b200.parallel.peer import PeerGroup

DTYPES = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16, "e4m3": torch.float8_e4m3fn, "u8": torch.uint8}
OPS = {"none": tx.OP_NONE, "add": tx.OP_ADD, "mul": tx.OP_MUL}
KIB, MIB, GIB = 1 << 10, 1 << 20, 1 << 30


def listed():
    return [
        # one small activation or control tensor: the latency of a call
        {"name": "rpc_4KiB", "kind": "rpc", "calls": 1, "rows": 1, "cols": 2048, "dtype": "bf16", "layout": "dense", "wire": "none"},
        # small tensors of many callers at once, 256 B to 64 KiB each: the rate of calls
        {"name": "rpc_16_in_flight", "kind": "rpc", "calls": 16, "rows": 1, "cols": 16384, "dtype": "f32", "layout": "dense", "wire": "none"},
        # a matrix sent as its transposed view, in half the bytes: no copy is made by the caller
        {"name": "rpc_transposed_f32_as_bf16", "kind": "rpc", "calls": 1, "rows": 4099, "cols": 4096, "dtype": "f32", "layout": "transposed", "wire": "bf16"},
        # a shard of weights or of a cache: the bandwidth of a call
        {"name": "rpc_1GiB", "kind": "rpc", "calls": 1, "rows": 1, "cols": 1 << 29, "dtype": "bf16", "layout": "dense", "wire": "none"},
        # an activation scaled and cast to fp8 on its way into a peer's buffer
        {"name": "push_f32_to_e4m3", "kind": "push", "rows": 4096, "cols": 7168, "src": "f32", "dst": "e4m3", "layout": "dense", "op": "mul"},
        # a head-major view or a matrix transpose gathered on its way
        {"name": "push_transposed_bf16", "kind": "push", "rows": 8192, "cols": 8192, "src": "bf16", "dst": "bf16", "layout": "transposed", "op": "none"},
        # a large prefill product on another worker's weight, as a call
        {"name": "gemm_call_bf16_8192", "kind": "gemm", "fmt": "bf16", "via": "call", "x": "pulled", "m": 8192, "n": 8192, "k": 8192},
        # a decode batch: one row block against the whole weight
        {"name": "gemm_bf16_128_rows", "kind": "gemm", "fmt": "bf16", "via": "op", "x": "local", "m": 128, "n": 8192, "k": 8192},
        # block-scaled fp8 with arbitrary fp32 scales, tile counts that divide nothing
        {"name": "gemm_fp8_block_ragged", "kind": "gemm", "fmt": "fp8_block", "via": "op", "x": "local", "m": 1920, "n": 4608, "k": 7168},
        # MXFP8 with X streamed in while the kernel computes
        {"name": "gemm_mxfp8_pulled_4096", "kind": "gemm", "fmt": "mxfp8", "via": "op", "x": "pulled", "m": 4096, "n": 4096, "k": 4096},
        # tokens of a prefill batch to 256 experts and back
        {"name": "moe_bf16_prefill", "kind": "moe", "tokens": 4096, "hidden": 7168, "topk": 8, "experts": 256, "fp8": False},
        # tokens of a decode batch, fp8 rows
        {"name": "moe_fp8_decode", "kind": "moe", "tokens": 128, "hidden": 7168, "topk": 8, "experts": 256, "fp8": True},
    ]


def _spread(rng, low, high):
    """A whole number from low to high, spread over its logarithm."""
    return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    kind = rng.choice(["rpc", "rpc", "push", "push", "gemm", "gemm", "gemm", "moe", "moe"])
    if kind == "rpc":
        layout = rng.choice(["dense", "dense", "offset", "rows", "transposed"])
        dtype = rng.choice(["f32", "bf16", "f16"])
        size = 4 if dtype == "f32" else 2
        calls = rng.choice([1, 1, 1, _spread(rng, 2, 16)])
        if calls > 1:
            return {"kind": "rpc", "calls": calls, "rows": 1, "cols": _spread(rng, 64, 16384), "dtype": dtype, "layout": "dense", "wire": "none"}
        n = _spread(rng, 1024, (256 * MIB if layout == "dense" else 64 * MIB) // size)
        rows = 1 if layout in ("dense", "offset") else _spread(rng, 1, max(1, math.isqrt(n)))
        return {"kind": "rpc", "calls": 1, "rows": rows, "cols": n // rows, "dtype": dtype, "layout": layout,
                "wire": rng.choice(["none", "none", "bf16", "f32"])}
    if kind == "push":
        layout = rng.choice(["dense", "dense", "offset", "rows", "transposed"])
        src = rng.choice(["f32", "bf16", "f16", "e4m3", "u8"])
        dst = "u8" if src == "u8" else rng.choice([src, "f32", "bf16", "f16", "e4m3"])
        n = _spread(rng, 1024, 64 * MIB)
        rows = _spread(rng, 1, math.isqrt(n))
        return {"kind": "push", "rows": rows, "cols": n // rows, "src": src, "dst": dst, "layout": layout,
                "op": "none" if src == "u8" else rng.choice(["none", "none", "add", "mul"])}
    if kind == "gemm":
        fmt = rng.choice(["bf16", "fp8_block", "mxfp8"])
        step = 256 if fmt == "mxfp8" else 128
        m = step * _spread(rng, 1, 8192 // step)
        if rng.random() < 0.25:
            return {"kind": "gemm", "fmt": fmt, "via": "call", "x": "pulled", "m": m, "n": 8192, "k": 8192}
        return {"kind": "gemm", "fmt": fmt, "via": "op", "x": rng.choice(["local", "local", "pulled"]), "m": m,
                "n": 256 * _spread(rng, 2, 32), "k": 128 * _spread(rng, 4, 64)}
    topk = rng.choice([1, 2, 4, 6, 8, 8])
    return {"kind": "moe", "tokens": _spread(rng, 1, 4096), "hidden": 128 * _spread(rng, 4, 56), "topk": topk,
            "experts": rng.choice([8, 16, 64, 256]), "fp8": rng.random() < 0.5}


class Session:
    """Two runtimes of one process and the event loop that serves them, as a program keeps them for its lifetime."""

    _one = None

    @classmethod
    def get(cls):
        if cls._one is None:
            cls._one = cls()
        return cls._one

    def __init__(self):
        self.loop = asyncio.new_event_loop()
        asyncio.set_event_loop(self.loop)
        self.served = {}
        self.loop.run_until_complete(self._start())

    async def _start(self):
        self.server = axon.AxonRuntime("server", timeout=60000, device=axon.cuda(0))
        self.client = axon.AxonRuntime("client", timeout=60000, device=axon.cuda(0))
        for name in ("f32", "f16", "bf16"):
            async def echo(x: torch.Tensor) -> torch.Tensor:
                return x

            self.server.register_function(echo, function_name="echo_" + name, memory_policy=self.buffer(name))
        self.server.start_server()
        self.client.start_client()
        await self.client.connect_endpoint_async(self.server.get_local_address(), "server")

    @staticmethod
    def buffer(name):
        return lambda metas: torch.empty(tuple(metas[0].shape), dtype=DTYPES[name], device="cuda:0")

    def weight(self, fmt, n, k):
        """The id under which the server holds the weight of this format and shape: a worker's model is loaded once."""
        key = (fmt, n, k)
        if key not in self.served:
            g = torch.Generator(device="cuda").manual_seed(4321)
            w = (torch.randn(k, n, device="cuda", generator=g) * 0.02).to(torch.bfloat16)
            self.server.serve_gemm(len(self.served) + 1, w, fmt, max_m=8192)
            self.served[key] = len(self.served) + 1
        return self.served[key]


def _view(case, dtype, gen):
    """The tensor that a program sends: N(0, 1) values, in the case's layout."""
    rows, cols, layout = case["rows"], case["cols"], case["layout"]
    shape = {"dense": (rows, cols), "offset": (rows * cols + 1,), "rows": (rows, cols + cols // 3 + 1), "transposed": (cols, rows)}[layout]
    if dtype == torch.uint8:
        t = torch.randint(0, 256, shape, device="cuda", generator=gen, dtype=torch.uint8)
    elif dtype == torch.float8_e4m3fn:
        t = torch.randn(shape, device="cuda", generator=gen).to(dtype)
    else:
        t = torch.randn(shape, device="cuda", generator=gen, dtype=dtype)
    if layout == "offset":
        return t[1:].view(rows, cols)
    if layout == "rows":
        return t[:, :cols]
    return t.t() if layout == "transposed" else t


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    if kind == "rpc":
        s = Session.get()
        xs = [_view(case, DTYPES[case["dtype"]], gen) for _ in range(case["calls"])]
        wire = case["wire"] if case["wire"] != "none" else case["dtype"]
        return {"case": case, "session": s, "xs": xs, "function": "echo_" + wire, "policy": s.buffer(wire),
                "wire": None if case["wire"] == "none" else DTYPES[wire]}
    if kind == "push":
        x = _view(case, DTYPES[case["src"]], gen)
        return {"case": case, "x": x, "y": torch.empty(x.shape, dtype=DTYPES[case["dst"]], device="cuda"), "op": OPS[case["op"]]}
    if kind == "gemm":
        m, n, k, fmt = case["m"], case["n"], case["k"], case["fmt"]
        x = torch.randn(m, k, device="cuda", generator=gen)
        state = {"case": case, "y": torch.empty(m, n, dtype=torch.bfloat16, device="cuda"), "scale": None}
        if fmt == "bf16":
            state["x"] = x.to(torch.bfloat16)
        elif fmt == "fp8_block":
            state["x"], state["scale"] = gemm_ops.quantize_rows_1x128(x)
        else:
            state["x"], exponents = gemm_ops.quantize_mx(x)
            state["scale"] = gemm_ops.mx_scale_chunks(exponents, False)
        if case["via"] == "call":
            state["session"] = Session.get()
            state["weight"] = state["session"].weight(fmt, n, k)
        else:
            w = torch.randn(k, n, device="cuda", generator=gen) * 0.02
            make = {"bf16": gemm_ops.RemoteGemm, "fp8_block": gemm_ops.RemoteGemmFp8, "mxfp8": gemm_ops.RemoteGemmMx}[fmt]
            state["gemm"] = make(w.to(torch.bfloat16) if fmt == "bf16" else w, m)
        return state
    t, topk, experts = case["tokens"], case["topk"], case["experts"]
    a2a = moe_ops.MoeAllToAll(PeerGroup(0, 1), t, case["hidden"], topk, experts, fp8=case["fp8"])
    x = torch.randn(t, case["hidden"], device="cuda", generator=gen).to(torch.bfloat16)
    gates = torch.softmax(torch.randn(t, experts, device="cuda", generator=gen), dim=-1).topk(topk, dim=-1)
    return {"case": case, "a2a": a2a, "x": x, "idx": gates.indices.to(torch.int32), "w": gates.values.contiguous()}


async def _calls(s):
    invoke, policy, wire, fn = s["session"].client.invoke, s["policy"], s["wire"], s["function"]
    futures = [invoke(x, worker_name="server", session_id=1, function=fn, memory_policy=policy, wire_dtype=wire) for x in s["xs"]]
    return [await futures[0]] if len(futures) == 1 else await asyncio.gather(*futures)


async def _gemm_call(s):
    status = await s["session"].client.remote_gemm(s["x"], s["y"], worker_name="server", weight_id=s["weight"], x_scale=s["scale"])
    if status:
        raise RuntimeError(f"remote gemm status {status}")
    return s["y"]


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "rpc":
        return state["session"].loop.run_until_complete(_calls(state))
    if kind == "push":
        tx.push(state["x"], state["y"], op=state["op"], op_arg=0.5)
        return state["y"]
    if kind == "gemm":
        if case["via"] == "call":
            return state["session"].loop.run_until_complete(_gemm_call(state))
        x = [state["x"].data_ptr()] + ([state["scale"].data_ptr()] if state["scale"] is not None else [])
        state["gemm"](*x, case["m"], state["y"].data_ptr(), x_is_local=case["x"] == "local")
        return state["y"]
    a2a = state["a2a"]
    a2a.dispatch(state["x"], state["idx"], state["w"])
    a2a.expert_ready()
    return a2a.combine()


def work(case):
    size = lambda name: torch.empty((), dtype=DTYPES[name]).element_size()  # noqa: E731
    kind = case["kind"]
    if kind == "rpc":
        # the argument read once, the result written once
        n = case["calls"] * case["rows"] * case["cols"]
        return {"bytes": n * (size(case["dtype"]) + size(case["dtype"] if case["wire"] == "none" else case["wire"])), "flops": 0}
    if kind == "push":
        return {"bytes": case["rows"] * case["cols"] * (size(case["src"]) + size(case["dst"])), "flops": 0}
    if kind == "gemm":
        m, n, k = case["m"], case["n"], case["k"]
        per = {"bf16": 2, "fp8_block": 1, "mxfp8": 1 + 1 / 32}[case["fmt"]]
        scales = 4 * (m * k // 128 + (n // 128) * (k // 128)) if case["fmt"] == "fp8_block" else 0
        return {"bytes": (m * k + n * k) * per + scales + 2 * m * n, "flops": 2 * m * n * k}
    # the tokens are read, every routed row is written for its expert and read back, the result is written
    t, h = case["tokens"], case["hidden"]
    row = h + h // 128 * 4 if case["fp8"] else 2 * h
    return {"bytes": 2 * t * h * 2 + t * case["topk"] * (2 * row + 8), "flops": 2 * t * h * case["topk"]}


def tolerance(case):
    if case["kind"] in ("rpc", "push"):
        return "exact"  # bytes moved, or one rounding of one operation
    if case["kind"] == "gemm":
        # fp32 sums in any order, one rounding to bf16: against 64 bits 1.66e-3 in the 2-norm and 3.9e-3 at most in every format
        return {"rel": 6.6e-3, "max": 1.6e-2}
    if case["fp8"]:
        # as above (1.5e-3); the row's scale may be applied as a factor or as a quotient, and a value that lies between two
        # e4m3 numbers may then become the other one, 1/16 away at most
        return {"rel": 6.6e-3, "max": 7e-2}
    return {"rel": 6.6e-3, "max": 1.6e-2}


def _quantized(x, block):
    """x[R, K] as e4m3 values with one scale per `block` of K (the largest value of a block becomes 448), in 64 bits.
    The scales are arbitrary fp32 numbers for blocks of 128 and powers of two (MXFP8) for blocks of 32."""
    r, k = x.shape
    g = x.float().view(r, k // block, block)
    scale = g.abs().amax(-1, keepdim=True).clamp_min(2.0 ** -100) * (1.0 / 448.0)
    if block == 32:
        scale = torch.exp2(torch.ceil(torch.log2(scale)))
    return ((g * (1.0 / scale)).to(torch.float8_e4m3fn).double() * scale.double()).view(r, k)


def exact(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    if kind == "rpc":
        return [_view(case, DTYPES[case["dtype"]], gen).double() for _ in range(case["calls"])]
    if kind == "push":
        x = _view(case, DTYPES[case["src"]], gen)
        if case["src"] == "u8":
            return x
        return {"none": lambda v: v, "add": lambda v: v + 0.5, "mul": lambda v: v * 0.5}[case["op"]](x.double())
    if kind == "gemm":
        m, n, k, fmt = case["m"], case["n"], case["k"], case["fmt"]
        x = torch.randn(m, k, device="cuda", generator=gen)
        if case["via"] == "call":
            gen = torch.Generator(device="cuda").manual_seed(4321)
        w = torch.randn(k, n, device="cuda", generator=gen) * 0.02
        if case["via"] == "call" or fmt == "bf16":
            w = w.to(torch.bfloat16).float()
        if fmt == "bf16":
            return x.to(torch.bfloat16).double() @ w.double()
        if fmt == "mxfp8":
            return _quantized(x, 32) @ _quantized(w.t(), 32).t()
        # weights: one scale per 128 x 128 block
        blocks = w.t().reshape(n // 128, 128, k // 128, 128).transpose(1, 2).reshape(-1, 128 * 128)
        w_t = _quantized(blocks, 128 * 128).view(n // 128, k // 128, 128, 128).transpose(1, 2).reshape(n, k)
        return _quantized(x, 128) @ w_t.t()
    t, topk, experts = case["tokens"], case["topk"], case["experts"]
    x = torch.randn(t, case["hidden"], device="cuda", generator=gen).to(torch.bfloat16)
    gates = torch.softmax(torch.randn(t, experts, device="cuda", generator=gen), dim=-1).topk(topk, dim=-1)
    # an identity expert: every one of a token's copies comes back as its (quantised) row
    rows = _quantized(x, 128) if case["fp8"] else x.double()
    return rows * gates.values.double().sum(-1, keepdim=True)
