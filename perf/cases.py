"""The work that a user of this package has one GPU do, as cases that can be timed and compared.

Everything goes through the public entry points: ``torch.ops.tileccl.*`` (plans cached by operand layout, new
operands on every call), ``AgGemm`` (input written straight into the symmetric heap) and ``TpMlp`` (eager, and
replayed from a CUDA graph).  Shapes are those of the package's own configurations: the tensor-parallel pair of a
gated MLP with hidden 8192 and ffn 28672 (3584 per rank at tp = 8), the M sweep 512..32768 of the GEMM +
reduce-scatter at N = 8192, K = 1024 per rank, the 8192-cubed GEMM of the interference experiments, and the small
shapes of the tests.

Inputs: activations N(0, 1), weights N(0, 0.02) (the reduce-scatter's K shard takes N(0, 1) on both sides, as its
benchmark does), bf16, fp32 accumulation, bf16 results.
"""
import math
import weakref

import torch

import tileccl_b200 as tc
from tileccl_b200.models.tp_mlp import TpMlp
from tileccl_b200.ops.ag_gemm import AgGemm

HIDDEN, FFN = 8192, 28672
HEAP_BYTES = 12 << 30        # holds the symmetric buffers of ten states of the largest case


def listed():
    return [
        # The smallest call: one GEMM of the test-suite's size, where the launch and the host path are everything.
        {"name": "gemm_small", "op": "gemm", "m": 512, "n": 768, "k": 320},
        # One decode step's worth of rows against a down projection of the tp = 8 block: reading the weight counts.
        {"name": "gemm_decode", "op": "gemm", "m": 128, "n": HIDDEN, "k": FFN // 8},
        # A chunked-prefill batch with no round number in it: an odd count of 128-row and of 256-column tiles,
        # and a K that is not a multiple of the 64-element k-step.
        {"name": "gemm_ragged", "op": "gemm", "m": 1152, "n": 2816, "k": 1000},
        # The plain GEMM that runs beside the transports in the interference experiments.
        {"name": "gemm_8192", "op": "gemm", "m": 8192, "n": 8192, "k": 8192},
        # The two ends and an ordinary point of the GEMM + reduce-scatter M sweep (K of one of eight ranks).
        {"name": "gemm_rs_512", "op": "gemm_rs", "m": 512, "n": HIDDEN, "k": HIDDEN // 8},
        {"name": "gemm_rs_4096", "op": "gemm_rs", "m": 4096, "n": HIDDEN, "k": HIDDEN // 8},
        {"name": "gemm_rs_32768", "op": "gemm_rs", "m": 32768, "n": HIDDEN, "k": HIDDEN // 8},
        # All-gather + GEMM from an activation that lives outside the symmetric heap (one of eight ranks' columns).
        {"name": "ag_gemm_2048", "op": "ag_gemm", "m": 2048, "n": FFN // 8, "k": HIDDEN},
        # All-gather + GEMM of the headline benchmark, input already in the symmetric heap: the largest call.
        {"name": "ag_gemm_32768", "op": "ag_gemm_heap", "m": 32768, "n": FFN, "k": HIDDEN},
        # The MLP block of one of eight ranks: a prefill batch launched eagerly, a small batch replayed from a graph.
        {"name": "mlp_16384", "op": "mlp", "m": 16384, "hidden": HIDDEN, "ffn": FFN // 8, "graph": False},
        {"name": "mlp_graph_512", "op": "mlp", "m": 512, "hidden": HIDDEN, "ffn": FFN // 8, "graph": True},
        # The stand-alone activation of a block that keeps it apart from the GEMM.
        {"name": "silu_mul_16384", "op": "silu_mul", "m": 16384, "ffn": FFN // 8},
    ]


def draw(rng):
    """One more case of the same ranges: sizes spread over their logarithms, in the steps that the operations take
    (M by 128, for the MLP block by 256; N by 256; K by 8; ffn of the block by 128, of the activation by 8)."""
    def size(low, high, step):
        return min(high, max(low, round(math.exp(rng.uniform(math.log(low), math.log(high))) / step) * step))

    op = rng.choice(["gemm", "gemm", "gemm_rs", "ag_gemm", "ag_gemm_heap", "mlp", "silu_mul"])
    if op == "silu_mul":
        return {"op": op, "m": size(16, 32768, 1), "ffn": size(256, 14336, 8)}
    while True:
        if op == "mlp":
            case = {"op": op, "m": size(256, 16384, 256), "hidden": size(512, HIDDEN, 256), "ffn": size(512, FFN // 4, 128),
                    "graph": rng.random() < 0.5}
        else:
            case = {"op": op, "m": size(128, 32768, 128), "n": size(256, 14336, 256), "k": size(64, HIDDEN, 8)}
        if work(case)["flops"] <= 4e12:
            return case


def work(case):
    m = case["m"]
    if case["op"] == "silu_mul":
        return {"bytes": m * case["ffn"] * 2 * 3, "flops": 5 * m * case["ffn"]}
    if case["op"] == "mlp":
        h, f = case["hidden"], case["ffn"]
        return {"bytes": 2 * (m * h + 3 * h * f + m * h), "flops": 6 * m * h * f}
    n, k = case["n"], case["k"]
    return {"bytes": 2 * (m * k + n * k + m * n), "flops": 2 * m * n * k}


def tolerance(case):
    """bf16 results of fp32 sums: a result lies within half a bf16 step of the exact value, 1.7e-3 of it in the
    2-norm; the block rounds its activations as well, and the activation's exponential is a hardware approximation."""
    return {"rel": 8e-3 if case["op"] == "mlp" else 6e-3}


class _State:
    """What a program holds between calls; compared and hashed by identity."""

    def __init__(self, call, keep):
        self.call, self.keep = call, keep


_live = weakref.WeakSet()    # states whose buffers lie in the symmetric heap
_case = None                 # the case that the heap was set up for


def _heap(case):
    """One symmetric heap, as a process has: set up anew for another case, its space given back once no state is left."""
    global _case
    key = tuple(sorted((k, v) for k, v in case.items() if k != "name"))
    if not _live:
        if key != _case:
            tc.shutdown()
        elif case["op"] in ("ag_gemm_heap", "mlp"):
            tc.heap().reset()
    _case = key
    return tc.init(HEAP_BYTES)


def _normal(seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return lambda rows, cols, std=1.0: torch.empty(rows, cols, dtype=torch.bfloat16, device="cuda").normal_(0.0, std, generator=gen)


def _gemm_inputs(case, normal):
    return normal(case["m"], case["k"]), normal(case["n"], case["k"], 1.0 if case["op"] == "gemm_rs" else 0.02)


def _mlp_inputs(case, normal):
    """Activations, gate|up weight (128 gate rows, then the 128 up rows of the same features, and so on), down weight."""
    h, f = case["hidden"], case["ffn"]
    return normal(case["m"], h), normal(2 * f, h, 0.02), normal(h, f, 0.02)


def prepare(case, seed):
    op, m = case["op"], case["m"]
    normal = _normal(seed)
    if op == "silu_mul":
        gate_up = normal(m, 2 * case["ffn"])
        return _State(lambda: torch.ops.tileccl.silu_mul(gate_up), gate_up)
    heap = _heap(case)
    if op == "mlp":
        mlp = TpMlp(heap, m, case["hidden"], case["ffn"], seed=seed, graph=case["graph"])
        x, w_gate_up, w_down = _mlp_inputs(case, normal)
        mlp.x_shard.copy_(x)
        mlp.w_gate_up.copy_(w_gate_up)
        mlp.w_down.copy_(w_down)
        del x, w_gate_up, w_down
        if case["graph"]:
            mlp.capture()
        state = _State(mlp.replay if case["graph"] else mlp, mlp)
        _live.add(state)
        return state
    a, b_t = _gemm_inputs(case, normal)
    if op == "ag_gemm_heap":
        layer = AgGemm(heap, m, case["k"], b_t, cta_group=2 if m % 256 == 0 else 1)
        layer.a_shard.copy_(a)
        state = _State(layer, layer)
    else:
        call = getattr(torch.ops.tileccl, op)
        state = _State(lambda: call(a, b_t), (a, b_t))
    _live.add(state)
    return state


def run(state):
    return state.call()


def exact(case, seed):
    """The same pass in 64 bits, from the same inputs; none for results of over a gigabyte."""
    op, normal = case["op"], _normal(seed)
    if op == "silu_mul":
        if case["m"] * case["ffn"] > 1 << 27:
            return None
        gate, up = normal(case["m"], 2 * case["ffn"]).double().split(case["ffn"], dim=1)
        return gate * torch.sigmoid(gate) * up
    if case["m"] * (case["hidden"] if op == "mlp" else case["n"]) > 1 << 27:
        return None
    if op == "mlp":
        x, w_gate_up, w_down = _mlp_inputs(case, normal)
        h = (x.double() @ w_gate_up.double().t()).view(case["m"], -1, 2, 128)
        act = h[:, :, 0] * torch.sigmoid(h[:, :, 0]) * h[:, :, 1]
        return act.reshape(case["m"], -1) @ w_down.double().t()
    a, b_t = _gemm_inputs(case, normal)
    return a.double() @ b_t.double().t()
