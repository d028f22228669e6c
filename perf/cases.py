"""The work this library is used for, as timed cases.

Every case goes through the public entry points of `rlx_b200`: the device-pointer calls on torch tensors
(`matmul`, `matmul_chain`, `grouped_matmul`, `gguf_tied_lm_argmax`, `gguf_tied_lm_topk`), a decode step captured in
a CUDA graph, and a compiled session with host arrays in and out.  Weights are raw GGUF blocks with the value
distributions the benchmark uses; activations are ~N(0, 1).  Shapes are those of the benchmark configurations and
tests (7B, 8B and 70B feed-forward layers, a 128 k vocabulary, 8-expert stacks) and their neighbourhood.
"""
import math

import numpy as np
import torch

import rlx_b200 as R

SCHEME = {"q4_0": R.QuantScheme.GgufQ4_0, "q8_0": R.QuantScheme.GgufQ8_0, "q4_k": R.QuantScheme.GgufQ4K,
          "q5_k": R.QuantScheme.GgufQ5K, "q6_k": R.QuantScheme.GgufQ6K}
GEOM = {"q4_0": (32, 18), "q8_0": (32, 34), "q4_k": (256, 144), "q5_k": (256, 176), "q6_k": (256, 210)}
DT = {"f32": torch.float32, "bf16": torch.bfloat16}
MAX_WEIGHTS = 8192 * 28672            # elements of the largest single matrix
MAX_MACS = 4096 * 8192 * 28672        # multiply-adds of the largest call


def listed():
    return [
        # the smallest call: one token through a square projection, called eagerly with the loop's own buffers
        {"name": "decode_q8_0_4096_m1", "kind": "linear", "scheme": "q8_0", "m": 1, "k": 4096, "n": 4096, "x": "f32", "y": "f32"},
        # a token's up / down pair, captured once in a CUDA graph and replayed every step
        {"name": "step_q4_0_7b_ffn_m1", "kind": "step", "scheme": "q4_0", "m": 1, "d": 4096, "f": 11008, "x": "f32"},
        # four sequences decoded together
        {"name": "decode_q4_k_8b_up_m4", "kind": "linear", "scheme": "q4_k", "m": 4, "k": 4096, "n": 14336, "x": "bf16", "y": "f32"},
        # rows that are no whole number of 256 weights and an odd output width (small models keep such layers in Q8_0)
        {"name": "decode_q8_0_odd_m3", "kind": "linear", "scheme": "q8_0", "m": 3, "k": 2080, "n": 5003, "x": "f32", "y": "f32"},
        # a prompt of 512 tokens
        {"name": "prefill_q4_k_8b_up_m512", "kind": "linear", "scheme": "q4_k", "m": 512, "k": 4096, "n": 14336, "x": "bf16", "y": "bf16"},
        # a ragged prompt with f32 activations through a 7B down projection kept in Q6_K, as mixed Q4_K / Q6_K files do
        {"name": "prefill_q6_k_7b_down_m300", "kind": "linear", "scheme": "q6_k", "m": 300, "k": 11008, "n": 4096, "x": "f32", "y": "f32"},
        # the largest call: a long prompt through a 70B up projection
        {"name": "prefill_q8_0_70b_up_m4096", "kind": "linear", "scheme": "q8_0", "m": 4096, "k": 8192, "n": 28672, "x": "bf16", "y": "bf16"},
        # a token's SwiGLU feed-forward block at 70B size: stacked gate / up, then down
        {"name": "swiglu_q4_k_70b_m1", "kind": "swiglu", "scheme": "q4_k", "m": 1, "d": 8192, "f": 28672, "x": "bf16"},
        # one token routed to two of eight experts
        {"name": "moe_q4_k_8x_decode", "kind": "moe", "scheme": "q4_k", "tokens": 1, "k": 4096, "n": 14336, "experts": 8, "x": "f32", "y": "f32"},
        # a prompt of 512 tokens, each routed to two of eight experts
        {"name": "moe_q4_k_8x_prefill", "kind": "moe", "scheme": "q4_k", "tokens": 512, "k": 4096, "n": 14336, "experts": 8, "x": "bf16", "y": "bf16"},
        # greedy choice of the next token over a tied 128 k embedding
        {"name": "lm_head_q4_k_128k_greedy", "kind": "lm", "scheme": "q4_k", "k": 4096, "n": 128256, "cap": 1, "x": "bf16"},
        # the graph / session API with host arrays: a mixed Q4_K / Q6_K feed-forward block at 8B size, one token a run
        {"name": "session_q4_k_q6_k_8b_ffn_m1", "kind": "session", "scheme": "q4_k", "down": "q6_k", "m": 1, "d": 4096, "f": 14336},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _to(v, step):
    return max(step, int(round(v / step)) * step)


def _width(rng, lo, hi):
    """An output width: mostly a multiple of 64, one in four whatever comes."""
    v = _log(rng, lo, hi)
    return int(v) | 1 if rng.random() < 0.25 else _to(v, 64)


def _depth(rng, scheme, lo, hi):
    """A row length: a multiple of 256, one in five of the 32-weight formats' only a multiple of 32."""
    return _to(_log(rng, lo, hi), 32 if GEOM[scheme][0] == 32 and rng.random() < 0.2 else 256)


def draw(rng):
    kind = rng.choices(["decode", "prefill", "step", "swiglu", "moe", "lm", "session"], [24, 24, 10, 10, 14, 8, 10])[0]
    scheme = rng.choice(sorted(SCHEME))
    x = rng.choice(["f32", "bf16"])
    if kind in ("decode", "prefill"):
        k, n = _depth(rng, scheme, 512, 16384), _width(rng, 256, 32768)
        if k * n > MAX_WEIGHTS:
            n = MAX_WEIGHTS // k
        if kind == "decode":
            m = rng.choice([1, 1, 1, 2, 3, 4, 5, 6, 7, 8])
            return {"kind": "linear", "scheme": scheme, "m": m, "k": k, "n": n, "x": x, "y": "f32"}
        m = min(int(_log(rng, 9, 4096)), MAX_MACS // (k * n))
        return {"kind": "linear", "scheme": scheme, "m": m, "k": k, "n": n, "x": x, "y": x}
    if kind in ("step", "swiglu"):
        d = _to(_log(rng, 1024, 8192), 256)
        f = _to(d * rng.uniform(2.5, 3.6), 256)
        if kind == "step":
            return {"kind": kind, "scheme": scheme, "m": rng.choice([1, 1, 2, 4, 8]), "d": d, "f": f, "x": x}
        m = rng.choice([1, 1, 2, 4, 8, int(_log(rng, 9, 512))])
        return {"kind": kind, "scheme": scheme, "m": m, "d": d, "f": f, "x": x}
    if kind == "moe":
        k, n, e = _to(_log(rng, 1024, 8192), 256), _to(_log(rng, 512, 14336), 64), rng.choice([4, 8, 16, 32])
        while e * k * n > 2 * MAX_WEIGHTS:
            e //= 2
        return {"kind": kind, "scheme": scheme, "tokens": rng.choice([1, 2, 4, int(_log(rng, 5, 1024)), int(_log(rng, 5, 1024))]),
                "k": k, "n": n, "experts": max(e, 2), "x": x, "y": x}
    if kind == "lm":
        k = _to(_log(rng, 1024, 6144), 256)
        return {"kind": kind, "scheme": scheme, "k": k, "n": int(_log(rng, 32000, 131072)), "cap": rng.choice([1, 1, 8, 40]), "x": x}
    d = _to(_log(rng, 512, 4096), 256)
    return {"kind": "session", "scheme": scheme, "down": rng.choice([scheme, "q6_k"]), "m": rng.choice([1, 1, 1, 2, 4, 8, 16]),
            "d": d, "f": _to(d * rng.uniform(2.5, 3.6), 256)}


# ------------------------------------------------------------------------------------------------ inputs
def _bytes(g, blocks, count):
    return torch.randint(0, 256, (blocks, count), dtype=torch.uint8, device="cuda", generator=g)


def _scales(g, blocks, count=1):
    """fp16 block scales uniform in [1e-3, 1e-2], as bytes."""
    return torch.empty((blocks, count), device="cuda").uniform_(1e-3, 1e-2, generator=g).half().view(torch.uint8)


def _weights(g, scheme, k, n):
    """Packed W[n, k]: raw blocks with uniform quants and scales."""
    elems, size = GEOM[scheme]
    b = k // elems * n
    if scheme == "q4_0":                       # d | 16 bytes of nibbles
        w = torch.cat([_scales(g, b), _bytes(g, b, 16)], 1)
    elif scheme == "q8_0":                     # d | 32 int8 in [-127, 127]
        q = torch.randint(-127, 128, (b, 32), dtype=torch.int8, device="cuda", generator=g)
        w = torch.cat([_scales(g, b), q.view(torch.uint8)], 1)
    elif scheme in ("q4_k", "q5_k"):           # d, dmin | 12 bytes of 6-bit scales and mins | (high bits) nibbles
        w = torch.cat([_scales(g, b, 2), _bytes(g, b, size - 4)], 1)
    else:                                      # q6_k: low nibbles | high bits | 16 int8 in [-64, 63] | d
        s = torch.randint(-64, 64, (b, 16), dtype=torch.int8, device="cuda", generator=g)
        w = torch.cat([_bytes(g, b, 192), s.view(torch.uint8), _scales(g, b)], 1)
    return w.view(-1)


def _normal(g, m, k, dtype):
    return torch.randn((m, k), device="cuda", generator=g).to(dtype)


def _workspace(size):
    return torch.empty(max(size, 256), dtype=torch.uint8, device="cuda")


def prepare(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    kind, s = case["kind"], SCHEME[case["scheme"]]
    st = dict(case)
    if kind == "linear":
        m, k, n = case["m"], case["k"], case["n"]
        st["w"] = _weights(g, case["scheme"], k, n)
        st["xd"] = _normal(g, m, k, DT[case["x"]])
        if m <= 8:                             # a decode loop keeps its output and scratch; a prompt's come with its length
            st["out"] = torch.empty((m, n), dtype=DT[case["y"]], device="cuda")
            st["ws"] = _workspace(R.workspace_bytes(s, m, k, n, int(case["x"] == "bf16"), int(case["y"] == "bf16")))
    elif kind == "step":
        m, d, f = case["m"], case["d"], case["f"]
        up, down = _weights(g, case["scheme"], d, f), _weights(g, case["scheme"], f, d)
        xd = _normal(g, m, d, DT[case["x"]])
        h, out = torch.empty((m, f), device="cuda"), torch.empty((m, d), device="cuda")
        ws = _workspace(max(R.workspace_bytes(s, m, d, f, int(case["x"] == "bf16")), R.workspace_bytes(s, m, f, d)))

        def step():
            R.matmul(xd, up, s, f, out=h, workspace=ws)
            R.matmul(h, down, s, d, out=out, workspace=ws)
        step()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            step()
        st.update(graph=graph, out=out, keep=(up, down, xd, h, ws))
    elif kind == "swiglu":
        m, d, f = case["m"], case["d"], case["f"]
        st["layers"] = [(_weights(g, case["scheme"], d, 2 * f), 2 * f), (_weights(g, case["scheme"], f, d), d, True)]
        st["xd"] = _normal(g, m, d, DT[case["x"]])
        st["ws"] = _workspace(R.chain_workspace_bytes(s, [(d, 2 * f, False), (f, d, True)], m, int(case["x"] == "bf16")))
    elif kind == "moe":
        k, n, e, t = case["k"], case["n"], case["experts"], case["tokens"]
        st["w"] = _weights(g, case["scheme"], k, n * e)
        st["xd"] = _normal(g, t, k, DT[case["x"]]).repeat_interleave(2, 0)          # every token once per chosen expert
        st["route"] = torch.rand((t, e), device="cuda", generator=g).topk(2, 1).indices.float().view(-1)
    elif kind == "lm":
        st["w"] = _weights(g, case["scheme"], case["k"], case["n"])
        st["xd"] = _normal(g, 1, case["k"], DT[case["x"]]).view(-1)
        st["ws"] = _workspace(R.lm_head_workspace_bytes(s, case["k"], case["n"], int(case["x"] == "bf16"), case["cap"]))
    else:
        m, d, f = case["m"], case["d"], case["f"]
        down = SCHEME[case["down"]]
        gr = R.Graph("ffn")
        xi = gr.input("x", [m, d])
        params = [("gate", case["scheme"], d, f), ("up", case["scheme"], d, f), ("down", case["down"], f, d)]
        gate, up, dn = (gr.param(name, [R.packed_bytes(SCHEME[sch], k, n)]) for name, sch, k, n in params)
        h = gr.swiglu_mul(gr.dequant_matmul_packed(xi, gate, s, f), gr.dequant_matmul_packed(xi, up, s, f))
        gr.set_outputs([gr.dequant_matmul_packed(h, dn, down, d)])
        st["graph"] = R.Session(R.Device.Cuda).compile(gr)
        for name, sch, k, n in params:
            st["graph"].set_param_typed(name, _weights(g, sch, k, n).cpu().numpy())
        st["xh"] = np.random.RandomState(seed % (1 << 32)).standard_normal((m, d)).astype(np.float32)
    return st


# ------------------------------------------------------------------------------------------------ one pass
def run(st):
    kind, s = st["kind"], SCHEME[st["scheme"]]
    if kind == "linear":
        if "out" in st:
            return R.matmul(st["xd"], st["w"], s, st["n"], out=st["out"], workspace=st["ws"])
        return R.matmul(st["xd"], st["w"], s, st["n"], out_dtype=DT[st["y"]])
    if kind == "step":
        st["graph"].replay()
        return st["out"]
    if kind == "swiglu":
        return R.matmul_chain(st["xd"], st["layers"], s, workspace=st["ws"])
    if kind == "moe":
        return R.grouped_matmul(st["xd"], st["w"], st["route"], s, st["n"], st["experts"], out_dtype=DT[st["y"]])
    if kind == "lm":
        if st["cap"] == 1:
            return R.gguf_tied_lm_argmax(st["xd"], st["w"], st["k"], st["n"], s, workspace=st["ws"])
        return R.gguf_tied_lm_topk(st["xd"], st["w"], st["k"], st["n"], s, st["cap"], workspace=st["ws"])
    return st["graph"].run([("x", st["xh"])], (st["m"], st["d"]))


# ------------------------------------------------------------------------------------------------ what it costs, how close
def work(case):
    kind = case["kind"]
    xb = 2 if case.get("x") == "bf16" else 4

    def packed(scheme, k, n):
        return k // GEOM[scheme][0] * GEOM[scheme][1] * n
    if kind == "linear":
        m, k, n = case["m"], case["k"], case["n"]
        return {"bytes": packed(case["scheme"], k, n) + m * k * xb + m * n * (2 if case["y"] == "bf16" else 4), "flops": 2 * m * k * n}
    if kind in ("step", "swiglu", "session"):
        m, d, f = case["m"], case["d"], case["f"]
        g = 1 if kind == "step" else 2
        return {"bytes": packed(case["scheme"], d, g * f) + packed(case.get("down", case["scheme"]), f, d) + m * d * xb + m * d * 4,
                "flops": 2 * m * d * f * (g + 1)}
    if kind == "moe":
        t, k, n, e = case["tokens"], case["k"], case["n"], case["experts"]
        used = e * (1 - (1 - 2 / e) ** t)                                            # experts that a batch meets
        return {"bytes": used * packed(case["scheme"], k, n) + 2 * t * k * xb + 2 * t * n * (2 if case["y"] == "bf16" else 4),
                "flops": 4 * t * k * n}
    return {"bytes": packed(case["scheme"], case["k"], case["n"]) + case["k"] * xb + 8 * case["cap"], "flops": 2 * case["k"] * case["n"]}


def tolerance(case):
    kind = case["kind"]
    if kind == "lm":
        return "exact"                          # logits re-evaluated in one fixed order of f32 additions
    rows = 2 * case["tokens"] if kind == "moe" else case["m"]
    if case.get("y") == "bf16":
        return {"rel": 6e-3}                    # bf16 results
    if rows > 8:
        return {"rel": 6e-3}                    # weights rounded to bf16 for the tensor cores
    return {"rel": 3e-4}                        # activations as 15-bit integers per 32 values
