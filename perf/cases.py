"""The work a user of this framework has it do, as timed cases.

Five kinds of call, each over the range of sizes it is used at:

  train    ``ragged_dot`` forward and backward (dlhs and drhs through autograd), 16-bit or float32
  decode   ``ragged_dot`` forward on few rows: inference, bound by the weights that are read
  e4m3     ``gmm_fp8_forward``: inference on 8-bit weights with one scale per expert
  moe      ``ragged_dot_permuted`` forward and backward: a mixture-of-experts layer on un-sorted tokens
  odd      ``ragged_dot`` forward and backward at small sizes whose rows are not multiples of 16 bytes

A case says everything that a call depends on: ``m`` rows, contraction ``k``, ``n`` columns, ``g``
groups, the ``dtype``, how unequal the groups are (``alpha``: multinomial over a Dirichlet(alpha)
draw; 0: uniform top-k routing of m / top_k tokens), the share of the rows that belong to a group
(``fill``), and the options of the entry point.
"""

import math

import numpy as np
import torch

import gpu_ragged_dot_b200 as rd
from gpu_ragged_dot_b200 import workloads

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "f32": torch.float32, "e4m3": torch.float8_e4m3fn}
BYTES = {"bf16": 2, "fp16": 2, "f32": 4, "e4m3": 1}
DEVICE = "cuda:0"


def _case(kind, m, k, n, g, dtype="bf16", alpha=1.0, fill=1.0, top_k=0, trans_rhs=False, precision="default", name=None):
    c = dict(kind=kind, m=m, k=k, n=n, g=g, dtype=dtype, alpha=alpha, fill=fill, top_k=top_k, trans_rhs=trans_rhs,
             precision=precision)
    return dict(c, name=name) if name else c


def listed():
    small, mixtral, deepseek = workloads.SMALL, workloads.MIXTRAL, workloads.DEEPSEEK_V3
    prefill, decode = workloads.EP_PREFILL, workloads.EP_DECODE
    return [
        # A point of the test grid: every size odd, 30 % of the rows in no group.  Small layers, unit tests.
        _case("odd", 171, 58, 77, 8, fill=0.7, name="odd_fwd_bwd_m171_k58_n77_g8"),
        # The small configuration: latency of the six kernels and of the host code around them.
        _case("train", small.m, small.k, small.n, small.g, name="small_fwd_bwd_m512_k256_n384_g8"),
        # One token, top-4: batch-1 decoding, four experts' weights are read.
        _case("decode", 4, decode.k, decode.n, decode.g, alpha=0, top_k=4, name="decode_fwd_m4_k4096_n1536_g64"),
        # 64 tokens, top-4: batched decoding, nearly every expert's weights are read.
        _case("decode", decode.m, decode.k, decode.n, decode.g, alpha=0, top_k=4, name="decode_fwd_m256_k4096_n1536_g64"),
        # The same with 8-bit weights.
        _case("e4m3", decode.m, decode.k, decode.n, decode.g, "e4m3", alpha=0, top_k=4, trans_rhs=True,
              name="decode_e4m3_m256_k4096_n1536_g64"),
        # Prompt processing with 8-bit weights.
        _case("e4m3", mixtral.m, mixtral.k, mixtral.n, mixtral.g, "e4m3", alpha=2.0, trans_rhs=True,
              name="prefill_e4m3_m8192_k4096_n14336_g8"),
        # One training step of an expert layer with 64 experts, uniform top-4 routing, fp16.
        _case("train", prefill.m, prefill.k, prefill.n, prefill.g, "fp16", alpha=0, top_k=4,
              name="train_fp16_m32768_k4096_n1536_g64"),
        # The benchmark's shape: few long groups, bound by the tensor cores.
        _case("train", mixtral.m, mixtral.k, mixtral.n, mixtral.g, alpha=2.0, name="train_m8192_k4096_n14336_g8"),
        # Many short, heavy-tailed groups, a fifth of them empty: bound by the weights and their gradient.
        _case("train", deepseek.m, deepseek.k, deepseek.n, deepseek.g, alpha=0.3, name="train_m32768_k7168_n2048_g256"),
        # float32 inputs, default precision, eight experts of the 64 (one of eight ranks).
        _case("train", 8192, prefill.k, prefill.n, 8, "f32", name="train_f32_m8192_k4096_n1536_g8"),
        # float32 inputs at nearly float32 accuracy.
        _case("train", 4096, prefill.k, prefill.n, 8, "f32", precision="highest", name="train_f32_highest_m4096_k4096_n1536_g8"),
        # The whole expert layer on un-sorted tokens: 4096 tokens, top-2 of 8 experts.
        _case("moe", mixtral.m, mixtral.k, mixtral.n, mixtral.g, alpha=0, top_k=2, name="moe_fwd_bwd_t4096_top2_k4096_n14336_g8"),
    ]


def draw(rng):
    def spread(lo, hi, mult=1):
        return max(1, round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / mult)) * mult

    kind = rng.choice(("train", "train", "train", "decode", "decode", "e4m3", "moe", "odd", "f32"))
    while True:
        if kind == "odd":
            return _case("odd", spread(100, 512), rng.randrange(33, 512, 2), rng.randrange(33, 512, 2), rng.choice((4, 8, 16)),
                         rng.choice(("bf16", "fp16")), fill=rng.choice((1.0, 0.7, 0.5)), trans_rhs=rng.random() < 0.3)
        k, n, g = spread(256, 14336, 8), spread(256, 14336, 8), spread(4, 256)
        alpha, fill = rng.choice((0.3, 1.0, 2.0)), rng.choice((1.0, 1.0, 0.9))
        if kind == "decode":
            c = _case("decode", spread(1, 512), k, n, g, rng.choice(("bf16", "bf16", "fp16")), alpha, 1.0, 0, rng.random() < 0.3)
        elif kind == "e4m3":
            c = _case("e4m3", spread(4, 32768), max(16, k // 16 * 16), n, g, "e4m3", alpha, fill, 0, True)
        elif kind == "moe":
            top_k = rng.choice((1, 2, 4, 8))
            c = _case("moe", spread(64, 4096) * top_k, k, n, max(g, top_k), rng.choice(("bf16", "fp16")), 0, 1.0, top_k)
        elif kind == "f32":
            c = _case("train", spread(256, 8192), k, n, spread(4, 64), "f32", alpha, fill, 0, rng.random() < 0.3,
                      rng.choice(("default", "default", "highest")))
        else:
            c = _case("train", spread(256, 32768), k, n, g, rng.choice(("bf16", "bf16", "fp16")), alpha, fill, 0, rng.random() < 0.3)
        # No drawn case costs more than the largest listed ones: 2.9e12 operations of 16-bit inputs
        # (a quarter of that as TF32, a twelfth in three passes), 7.5 GB of weights.
        limit = 2.8e12 / {"f32": 12 if c["precision"] == "highest" else 4}.get(c["dtype"], 1)
        products = 1 if kind in ("decode", "e4m3") else 3
        if products * 2.0 * c["m"] * c["k"] * c["n"] <= limit and c["g"] * c["k"] * c["n"] * max(2, BYTES[c["dtype"]]) <= 6e9:
            return c


def _routing(case, rng):
    tokens = max(1, case["m"] // case["top_k"])
    return np.argsort(rng.random((tokens, case["g"])), axis=1)[:, : case["top_k"]].astype(np.int32)


def _group_sizes(case, rng):
    if case["alpha"] == 0:
        return workloads.group_sizes_from_routing(_routing(case, rng), case["g"])
    p = rng.dirichlet(case["alpha"] * np.ones(case["g"]))
    return rng.multinomial(round(case["m"] * case["fill"]), p).astype(np.int32)


def _normal(shape, std, seed, dtype):
    return workloads.normal_tensor(shape, std, seed, DEVICE, dtype)


def prepare(case, seed):
    m, k, n, g, dtype = case["m"], case["k"], case["n"], case["g"], DTYPES[case["dtype"]]
    rng = np.random.default_rng(seed)
    weights = (g, n, k) if case["trans_rhs"] else (g, k, n)
    state = dict(case=case)
    if case["kind"] == "moe":
        routing = _routing(case, rng).reshape(-1)
        order = np.argsort(routing, kind="stable").astype(np.int32)
        state["gs"] = torch.from_numpy(workloads.group_sizes_from_routing(routing, g)).to(DEVICE)
        state["in_rows"] = torch.from_numpy(order // case["top_k"]).to(DEVICE)
        state["out_rows"] = torch.from_numpy(order).to(DEVICE)
        rows = m // case["top_k"]
    else:
        state["gs"] = torch.from_numpy(_group_sizes(case, rng)).to(DEVICE)
        rows = m
    if case["kind"] == "e4m3":
        # amax-scaled weights, as a quantised checkpoint has them: N(0, 1/k) = scale * e4m3
        state["x"] = _normal((rows, k), 1.0, 3 * seed + 1, torch.bfloat16).to(dtype)
        A = torch.empty(weights, dtype=dtype, device=DEVICE)
        for i in range(g):
            A[i] = _normal(weights[1:], 64.0, (3 * seed + 2) * 1009 + i, torch.bfloat16).to(dtype)
        state["A"] = A
        state["scale"] = torch.from_numpy((rng.uniform(0.9, 1.1, g) * k ** -0.5 / 64.0).astype(np.float32)).to(DEVICE)
        return state
    state["x"] = _normal((rows, k), 1.0, 3 * seed + 1, dtype)
    state["A"] = _normal(weights, k ** -0.5, 3 * seed + 2, dtype)
    if case["kind"] != "decode":
        state["dout"] = _normal((m, n), 1.0, 3 * seed + 3, dtype)
        state["x"].requires_grad_(True)
        state["A"].requires_grad_(True)
    return state


def run(state):
    case, x, A, gs = state["case"], state["x"], state["A"], state["gs"]
    if case["kind"] == "decode":
        return rd.ragged_dot(x, A, gs, trans_rhs=case["trans_rhs"])
    if case["kind"] == "e4m3":
        return rd.gmm_fp8_forward(x, A, gs, weight_scale=state["scale"])
    if case["kind"] == "moe":
        y = rd.ragged_dot_permuted(x, A, gs, in_rows=state["in_rows"], out_rows=state["out_rows"], y_rows=case["m"])
    else:
        precision = None if case["precision"] == "default" else case["precision"]
        y = rd.ragged_dot(x, A, gs, trans_rhs=case["trans_rhs"], precision=precision)
    dx, dA = torch.autograd.grad(y, (x, A), state["dout"])
    return {"y": y, "dx": dx, "dA": dA}


def work(case):
    """Each input read once and each output written once.  The forward reads x and the weights of the
    groups that have rows and writes y; the backward reads x, dout and those weights and writes dx and
    the whole weight gradient.  The expected number of groups with rows stands for the drawn one."""
    m, k, n, g, size = case["m"], case["k"], case["n"], case["g"], BYTES[case["dtype"]]
    if case["alpha"] == 0:
        live = g * (1.0 - (1.0 - min(1.0, case["top_k"] / g)) ** max(1, m // case["top_k"]))
    else:  # P(no row) of one component of a Dirichlet-multinomial
        a, rest, rows = case["alpha"], case["alpha"] * (g - 1), round(m * case["fill"])
        lg = math.lgamma
        live = g * (1.0 - math.exp(lg(a + rest) - lg(rest) + lg(rest + rows) - lg(a + rest + rows)))
    rows_in = m // case["top_k"] if case["kind"] == "moe" else m
    x, y, used, flops = rows_in * k, m * n, live * k * n, 2.0 * m * case["fill"] * k * n
    if case["kind"] == "decode":
        return {"bytes": size * (x + used + y), "flops": flops}
    if case["kind"] == "e4m3":
        return {"bytes": x + used + 2 * y, "flops": flops}
    return {"bytes": size * ((x + used + y) + (x + y + used + x + g * k * n)), "flops": 3 * flops}


def tolerance(case):
    """About four times the error of the present results against the same products in float64 (2-norm, and
    largest over the root mean square): the rounding of the 16-bit result (bf16 1.7e-3, fp16 2.1e-4; twice
    where rounded rows are summed per token), of float32 inputs to TF32 (7.8e-4), of float32 sums (1e-5)."""
    if case["dtype"] == "f32":
        return {"rel": 4e-5, "max": 2e-4} if case["precision"] == "highest" else {"rel": 3e-3, "max": 1.2e-2}
    rel, most = (8e-4, 2e-3) if case["dtype"] == "fp16" else (6.6e-3, 1.6e-2)
    return {"rel": 1.5 * rel, "max": 3 * most} if case["kind"] == "moe" else {"rel": rel, "max": most}
