"""Work that users of this package have it do, through its public entry points, for timing.

Kinds of case:
  step   the projections of one forward step of `layers` layers of the 32-layer stack that bench.py and the tests use
         (hidden 2560; every fourth layer full attention: q, k, v, o; the others GDN in / out; each with a SwiGLU MLP of
         9216), for `m` tokens.  Every layer has weights of its own, so eight layers stream 0.4 GB, past L2, as a model does.
         `graph`: the step was captured once and is replayed, as a decode loop does after its warm-up; otherwise the calls
         are made one by one.  `rank` > 0: a LoRA adapter on every projection.
  mlp    gate+up with SwiGLU, then down, of one layer: what a prefill chunk spends most of its time in.
  proj   one projection call, optionally with per-column scales (`groupsize` -1) or a LoRA adapter.
  load   one weight that is on the GPU, quantised and packed (bf16, f32) or repacked (GPTQ) when a model is loaded.
  host   one f32 weight in host memory, quantised and packed on the CPU by the mirror of the reference's packer.
"""
import math

import numpy as np
import torch

import kiln_b200

HIDDEN, MIX, MLP = 2560, 4096, 9216  # of the 32-layer stack
MOST_FLOPS = 2.0 * 16384 * 9216 * 9216


def listed():
    return [
        # one token through the k projection of an attention layer: the smallest call there is, all latency
        {"name": "k_proj_m1", "kind": "proj", "m": 1, "k": 2560, "n": 512, "groupsize": 128, "rank": 0},
        # one user, one token: the decode loop's replayed step
        {"name": "decode_m1_graph", "kind": "step", "m": 1, "layers": 8, "graph": True, "rank": 0},
        # a small decode batch of odd size, called eagerly (batch sizes change from step to step: no captured graph)
        {"name": "decode_m13_eager", "kind": "step", "m": 13, "layers": 8, "graph": False, "rank": 0},
        # continuous batching, 64 sequences: the stack benchmark's configuration
        {"name": "batch_m64_graph", "kind": "step", "m": 64, "layers": 8, "graph": True, "rank": 0},
        # the same server with an adapter loaded and an odd number of sequences
        {"name": "lora_m37_eager", "kind": "step", "m": 37, "layers": 4, "graph": False, "rank": 64},
        # a per-column quantised output projection at a medium batch
        {"name": "per_column_m100", "kind": "proj", "m": 100, "k": 4096, "n": 2560, "groupsize": -1, "rank": 0},
        # a short prompt's chunk through a few layers
        {"name": "prefill_m512", "kind": "step", "m": 512, "layers": 4, "graph": False, "rank": 0},
        # a prompt of odd length through an MLP
        {"name": "prefill_mlp_m1789", "kind": "mlp", "m": 1789, "k": HIDDEN, "n": MLP},
        # the scheduler's whole token budget in one chunk
        {"name": "prefill_mlp_m8192", "kind": "mlp", "m": 8192, "k": HIDDEN, "n": MLP},
        # one GPU's share of the column-parallel configuration (N = 73728 over eight)
        {"name": "shard_m16384", "kind": "proj", "m": 16384, "k": 9216, "n": 9216, "groupsize": 128, "rank": 0},
        # a gate projection packed when the model is loaded
        {"name": "load_gate_bf16", "kind": "load", "source": "bf16", "k": 2560, "n": 9216, "groupsize": 128},
        # a q projection packed on the host
        {"name": "host_pack_q", "kind": "host", "k": 2560, "n": 4096, "groupsize": 128},
    ]


def _log(rng, lo, hi, step=1):
    """A multiple of `step` in [lo, hi], spread over the logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return int(min(hi, max(lo, round(v / step) * step)))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "proj", "proj", "proj", "mlp", "mlp", "load", "load", "host"])
    if kind == "step":
        m = _log(rng, 1, 512)
        rank = rng.choice([0, 0, 0, 8, 16, 64])
        return {"kind": "step", "m": m, "layers": 8 if m <= 128 and not rank else 4, "graph": rng.random() < 0.5, "rank": rank}
    if kind == "proj":
        k, n = _log(rng, 512, 9216, 128), _log(rng, 256, 18432, 256)
        groupsize = rng.choice([128, 128, 128, -1])
        rank = rng.choice([0, 0, 16, 64]) if groupsize == 128 else 0
        m = _log(rng, 1, min(16384, int(MOST_FLOPS / (2.0 * k * n))))
        return {"kind": "proj", "m": m, "k": k, "n": n, "groupsize": groupsize, "rank": rank}
    if kind == "mlp":
        return {"kind": "mlp", "m": _log(rng, 1, 8192), "k": _log(rng, 1024, 4096, 256), "n": _log(rng, 2048, 9216, 256)}
    if kind == "load":
        return {"kind": "load", "source": rng.choice(["bf16", "bf16", "f32", "gptq"]), "k": _log(rng, 512, 9216, 128),
                "n": _log(rng, 256, 9216, 256), "groupsize": rng.choice([128, 128, 128, -1])}
    return {"kind": "host", "k": _log(rng, 512, 2560, 128), "n": _log(rng, 256, 4096, 256), "groupsize": rng.choice([128, 128, -1])}


# ---- what a program has in hand -------------------------------------------------------------


class _Make:
    """Inputs on the GPU from one seed: int4 weights uniform in [-8, 7], scales 0.01 |N(0,1)| + 1e-3, activations N(0,1)."""

    def __init__(self, seed):
        self.dev = torch.device("cuda")
        self.gen = torch.Generator(device=self.dev)
        self.gen.manual_seed(seed)

    def normal(self, *shape, std=1.0, dtype=torch.bfloat16):
        return (torch.randn(shape, device=self.dev, generator=self.gen) * std).to(dtype)

    def words(self, rows, cols):
        return torch.randint(-2 ** 31, 2 ** 31 - 1, (rows, cols), dtype=torch.int32, device=self.dev, generator=self.gen)

    def scales(self, rows, n):
        return (0.01 * torch.randn((rows, n), device=self.dev, generator=self.gen).abs() + 1e-3).to(torch.float16)

    def proj(self, k, n, groupsize=128):
        g = k if groupsize == -1 else groupsize
        return kiln_b200.MarlinPackedProj(self.words(k // 16, 2 * n), self.scales(k // g, n), groupsize, k, n)

    def gate_up(self, k, n):
        return kiln_b200.interleave_gate_up(self.proj(k, n), self.proj(k, n))

    def adapter(self, rank, k, n):
        return (self.normal(rank, k, std=0.05), self.normal(n, rank, std=0.05), 2.0) if rank else None


def _prepare_step(case, make):
    m, rank, layers = case["m"], case["rank"], []
    for i in range(case["layers"]):
        shapes = {"in": (HIDDEN, 8192), "out": (MIX, HIDDEN)} if i % 4 != 3 else {
            "q": (HIDDEN, 4096), "k": (HIDDEN, 512), "v": (HIDDEN, 512), "o": (MIX, HIDDEN)}
        layer = {name: (make.proj(k, n), make.adapter(rank, k, n)) for name, (k, n) in shapes.items()}
        layer["gate_up"] = (make.gate_up(HIDDEN, MLP), make.adapter(rank, HIDDEN, 2 * MLP))
        layer["down"] = (make.proj(MLP, HIDDEN), make.adapter(rank, MLP, HIDDEN))
        # normalised residual before the mixer and before the MLP, and the mixer's own output
        layer["x"], layer["y"], layer["mixed"] = make.normal(m, HIDDEN), make.normal(m, HIDDEN), make.normal(m, MIX)
        layers.append(layer)
    return layers


def _linear(x, weight):
    proj, adapter = weight
    return kiln_b200.matmul_bf16_lora(x, proj, *adapter) if adapter else kiln_b200.matmul_bf16(x, proj)


def _swiglu(x, weight):
    proj, adapter = weight
    return kiln_b200.swiglu_gate_up(x, proj, *(adapter or ()))


def _step(layers):
    outs = []
    for layer in layers:
        x = layer["x"]
        if "in" in layer:
            outs += [_linear(x, layer["in"]), _linear(layer["mixed"], layer["out"])]
        else:
            siblings = [layer[name] for name in ("q", "k", "v")]
            if siblings[0][1] is None:
                outs += kiln_b200.grouped_matmul_bf16([x, x, x], [proj for proj, _ in siblings])
            else:
                outs += [_linear(x, w) for w in siblings]
            outs.append(_linear(layer["mixed"], layer["o"]))
        act = _swiglu(layer["y"], layer["gate_up"])
        outs += [act, _linear(act, layer["down"])]
    return outs


def prepare(case, seed):
    kind = case["kind"]
    if kind == "host":
        rng = np.random.default_rng(seed)
        return {"case": case, "w": rng.standard_normal((case["k"], case["n"]), dtype=np.float32) * np.float32(0.02)}
    make = _Make(seed)
    state = {"case": case}
    if kind == "step":
        state["layers"] = _prepare_step(case, make)
        if case["graph"]:
            stream = torch.cuda.Stream()
            stream.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(stream):
                _step(state["layers"])
            stream.synchronize()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=stream):
                state["outs"] = _step(state["layers"])
            state["graph"] = graph
    elif kind == "mlp":
        k, n = case["k"], case["n"]
        state.update(x=make.normal(case["m"], k), gate_up=make.gate_up(k, n), down=make.proj(n, k))
    elif kind == "proj":
        k, n = case["k"], case["n"]
        state.update(x=make.normal(1, case["m"], k), w=(make.proj(k, n, case["groupsize"]), make.adapter(case["rank"], k, n)))
    elif case["source"] == "gptq":
        k, n = case["k"], case["n"]
        g = k if case["groupsize"] == -1 else case["groupsize"]
        state.update(qweight=make.words(k // 8, n), scales=make.scales(k // g, n),
                     qzeros=torch.full((k // g, n // 8), -0x77777778, dtype=torch.int32, device=make.dev))  # every zero-point 8
    else:
        state["w"] = make.normal(case["k"], case["n"], std=0.02, dtype=torch.bfloat16 if case["source"] == "bf16" else torch.float32)
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "step":
        if case["graph"]:
            state["graph"].replay()
            return state["outs"]
        return _step(state["layers"])
    if kind == "mlp":
        act = kiln_b200.swiglu_gate_up(state["x"], state["gate_up"])
        return [act, kiln_b200.matmul_bf16(act, state["down"])]
    if kind == "proj":
        return _linear(state["x"], state["w"])
    if kind == "host":
        return kiln_b200.pack.quantize_and_pack(state["w"], case["k"], case["n"], case["groupsize"])
    if case["source"] == "gptq":
        proj = kiln_b200.pack_from_gptq(state["qweight"], state["qzeros"], state["scales"], case["groupsize"])
    else:
        proj = kiln_b200.pack_from_bf16(state["w"], case["groupsize"])
    return [proj.b_packed, proj.scales]


# ---- what the work cannot do without ----------------------------------------------------------


def _weight_bytes(k, n, groupsize=128):
    return k * n / 2 + (k // (k if groupsize == -1 else groupsize)) * n * 2


def _gemm(m, k, n, n_out, groupsize=128, rank=0, reads_x=True):
    """Bytes and operations of one projection of m rows; n_out: columns written (n/2 after SwiGLU)."""
    b = _weight_bytes(k, n, groupsize) + (2 * m * k if reads_x else 0) + 2 * m * n_out + 2 * rank * (k + n)
    return b, 2.0 * m * k * n + 2.0 * m * rank * (k + n)


def work(case):
    kind = case["kind"]
    if kind == "step":
        m, r, parts = case["m"], case["rank"], []
        for i in range(case["layers"]):
            if i % 4 != 3:
                parts += [_gemm(m, HIDDEN, 8192, 8192, rank=r), _gemm(m, MIX, HIDDEN, HIDDEN, rank=r)]
            else:
                parts += [_gemm(m, HIDDEN, 4096, 4096, rank=r), _gemm(m, HIDDEN, 512, 512, rank=r, reads_x=False),
                          _gemm(m, HIDDEN, 512, 512, rank=r, reads_x=False), _gemm(m, MIX, HIDDEN, HIDDEN, rank=r)]
            parts += [_gemm(m, HIDDEN, 2 * MLP, MLP, rank=r), _gemm(m, MLP, HIDDEN, HIDDEN, rank=r)]
    elif kind == "mlp":
        m, k, n = case["m"], case["k"], case["n"]
        parts = [_gemm(m, k, 2 * n, n), _gemm(m, n, k, k)]
    elif kind == "proj":
        parts = [_gemm(case["m"], case["k"], case["n"], case["n"], case["groupsize"], case["rank"])]
    else:
        k, n, out = case["k"], case["n"], _weight_bytes(case["k"], case["n"], case["groupsize"])
        if kind == "host":  # f32 in, packed words, scales and the f32 dequantised weight out
            parts = [(4.0 * k * n + out + 4.0 * k * n, 4.0 * k * n)]
        elif case["source"] == "gptq":  # zero-points are read as well
            parts = [(2 * out + (out - k * n / 2) / 4, 0.0)]
        else:
            parts = [((2.0 if case["source"] == "bf16" else 4.0) * k * n + out, 4.0 * k * n)]
    return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}


def tolerance(case):
    """Packing gives the same bytes.  Projections: bf16 results, and in the larger batches bf16 scales and weights, each
    rounded to 8 bits; `max` is the largest such error over millions of values, SwiGLU and down in sequence included."""
    if case["kind"] in ("load", "host"):
        return "exact"
    return {"rel": 1e-2, "max": 0.1}
