"""The work that a user of this package has it do, as measurable cases: proofs and verdicts through the public entry points,
from the smallest calls to the largest.  Shapes are the ones of the repository's benchmark and tests; weights and inputs are
seeded random integers (int8 range embedded in the field where they stand for weights and activations, the whole field for
polynomials and sumcheck tables).

A case is a dict with a "kind":
  sumcheck   one sumcheck over tables on the GPU (n variables; proto: base-field or extension tables, two or three of them)
  mlp        an op list of linears and ReLUs, base-field challenges, host input in, proof bytes out
  gpt2       an op list of GPT-2-shaped blocks at one position (LayerNorm, linears, GELU lookups, residuals)
  qwen       forward pass + the layer proofs of a stack of Qwen3.5-shaped layers (three GatedDeltaNet-structure layers, then one
             grouped-query attention layer, and so on), with a weight binding; "verify": the proofs of that stack are checked
  attention  row attention over heads x positions; "verify": its proof is checked
  basefold   Basefold commitment and opening of one polynomial
  batch      one batch-Basefold proof over polynomials of different sizes that were committed at load time
"""
import math

import numpy as np
import torch

import zklm_compile_b200 as zk
from zklm_compile_b200 import attention, oplist, pcs, qwen, tables

P = (1 << 31) - 1
LABEL = b"structured-ml-proof"
PROTOS = {  # proto -> (entry point, words per element of each table)
    "product": (zk.prove_product, (1, 1)),
    "triple": (zk.prove_triple, (1, 1, 1)),
    "product_ef": (zk.prove_product_ef, (1, 1)),
    "product_ef_full": (zk.prove_product_ef_full, (4, 4)),
    "triple_ef_full": (zk.prove_triple_ef_full, (4, 4, 4)),
}


def listed():
    return [
        # a sumcheck of an activation vector's length (a 4096-wide layer): nothing but latency
        {"name": "sumcheck small", "kind": "sumcheck", "proto": "product_ef", "n": 12},
        # the three-table sumcheck that norms and gated products reduce to, at a size where rounds still fill the GPU
        {"name": "sumcheck triple", "kind": "sumcheck", "proto": "triple_ef_full", "n": 20},
        # the isolated product sumcheck at the largest size of the microbenchmark
        {"name": "sumcheck large", "kind": "sumcheck", "proto": "product_ef", "n": 28},
        # the MLP of the published comparison: 1024 -> 2048 -> 1024 -> 10
        {"name": "mlp dense-4m", "kind": "mlp", "dims": "1024,2048,1024,10"},
        # a whole small language model in op-list mode: 182 ops on one transcript
        {"name": "gpt2 124m", "kind": "gpt2", "d": 768, "layers": 12, "vocab": 50257},
        # one GPU's share of the 32-layer 4B-shape model when eight GPUs prove it: three GDN layers and one GQA layer
        {"name": "qwen 4b prove", "kind": "qwen", "d_model": 2560, "d_ff": 9728, "unit": 128, "layers": 4, "binding": 0, "node": 0, "verify": False},
        # the same proofs on the receiving side
        {"name": "qwen 4b verify", "kind": "qwen", "d_model": 2560, "d_ff": 9728, "unit": 128, "layers": 4, "binding": 0, "node": 0, "verify": True},
        # a layer of the 9B shape whose every weight matrix is bound by a full Basefold opening
        {"name": "qwen 9b pcs-full", "kind": "qwen", "d_model": 4096, "d_ff": 12288, "unit": 128, "layers": 1, "binding": 2, "node": 0, "verify": False},
        # attention over a prompt of 128 positions at GPT-2's head shape, the caller keeping its own transcript
        {"name": "attention prove", "kind": "attention", "heads": 12, "kv": 0, "seq": 128, "d": 64, "own_transcript": False, "verify": False},
        # a grouped-query attention proof over a ragged prompt, checked on the receiving side, transcript included
        {"name": "attention verify", "kind": "attention", "heads": 16, "kv": 4, "seq": 77, "d": 128, "own_transcript": True, "verify": True},
        # commitment and opening of a polynomial at the microbenchmark's size
        {"name": "basefold 2^24", "kind": "basefold", "coeffs": 1 << 24, "node": 0},
        # one proof over a layer's matrices of different sizes, with the node hash of the reference's ARM build
        {"name": "batch basefold aes", "kind": "batch", "sizes": "2621440,655360,655360,2621440,1000003,300,4097", "node": 1},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("sumcheck", "sumcheck", "mlp", "gpt2", "qwen", "qwen", "attention", "attention", "basefold", "batch"))
    if kind == "sumcheck":
        proto = rng.choice(sorted(PROTOS))
        return {"kind": kind, "proto": proto, "n": rng.randint(8, 24 if proto.endswith("full") else 27)}
    if kind == "mlp":
        return {"kind": kind, "dims": ",".join(str(_log(rng, 10, 4096)) for _ in range(rng.randint(3, 5)))}
    if kind == "gpt2":
        return {"kind": kind, "d": 4 * _log(rng, 24, 256), "layers": rng.randint(1, 6), "vocab": _log(rng, 1000, 50257)}
    if kind == "qwen":
        binding = rng.choice((0, 0, 1, 2))
        d = _log(rng, 320, 1600 if binding == 2 else 4096)
        return {"kind": kind, "d_model": d, "d_ff": int(d * rng.uniform(2.5, 4)), "unit": max(8, d // 20), "layers": rng.randint(1, 4),
                "binding": binding, "node": rng.randint(0, 1), "verify": rng.random() < 0.4}
    if kind == "attention":
        kv = rng.choice((0, 0, 1, 2, 4))
        return {"kind": kind, "heads": rng.randint(1, 12) if kv == 0 else kv * rng.randint(1, 4), "kv": kv, "seq": _log(rng, 3, 140),
                "d": _log(rng, 16, 128), "own_transcript": rng.random() < 0.5, "verify": rng.random() < 0.4}
    if kind == "basefold":
        return {"kind": kind, "coeffs": _log(rng, 1 << 10, 1 << 24), "node": rng.randint(0, 1)}
    return {"kind": kind, "sizes": ",".join(str(_log(rng, 256, 1 << 22)) for _ in range(rng.randint(2, 8))), "node": rng.randint(0, 1)}


# ---- inputs -------------------------------------------------------------------------------------
class _Inputs:
    """Seeded values, made on the GPU."""

    def __init__(self, seed):
        self.g = torch.Generator(device="cuda")
        self.g.manual_seed(seed)

    def field(self, n):
        """n elements uniform in the field, as a tensor on the GPU."""
        return torch.randint(0, P, (n,), generator=self.g, device="cuda", dtype=torch.int32)

    def small(self, n, most=127):
        """n integers uniform in [-most, most] embedded in the field, on the host."""
        a = torch.randint(-most, most + 1, (n,), generator=self.g, device="cuda", dtype=torch.int32)
        return torch.where(a < 0, a + P, a).cpu().numpy().view(np.uint32)


class _Buffers:
    """Tensors on the GPU as the package's device buffers (the tensors stay alive with this object)."""

    def __init__(self, ctx, tensors):
        self.tensors = tensors
        self.bufs = [zk.DeviceBuffer.wrap(ctx, t.data_ptr(), t.numel()) for t in tensors]


def _layer_config(case, i):
    u = case["unit"]
    c = dict(d_model=case["d_model"], d_ff=case["d_ff"], d_head=u)
    if i % 4 == 3:
        return dict(c, num_q_heads=32 if u >= 128 else 8, num_kv_heads=8 if u >= 128 else 2, v_num_heads=0, v_d_head=0)
    return dict(c, num_q_heads=16 if u >= 128 else 4, num_kv_heads=16 if u >= 128 else 4, v_num_heads=32 if u >= 128 else 8, v_d_head=u)


def _layer_sizes(c):
    q, k = c["num_q_heads"] * c["d_head"], c["num_kv_heads"] * c["d_head"]
    v = (c["v_num_heads"] or c["num_kv_heads"]) * (c["v_d_head"] or c["d_head"])
    o = q if c["num_q_heads"] != c["num_kv_heads"] else v
    dm, ff = c["d_model"], c["d_ff"]
    return dict(norm1_gamma=dm, w_q=q * dm, w_k=k * dm, w_v=v * dm, w_o=dm * o, w_g_proj=o * dm, norm2_gamma=dm, w_gate=ff * dm, w_up=ff * dm,
                w_down=dm * ff)


def _gpt2(ctx, inp, case):
    d, f, v = case["d"], 4 * case["d"], case["vocab"]
    gelu = ctx.upload(tables.build_gelu_table(1000))
    p = oplist.OpList(ctx, d)
    for i in range(case["layers"]):
        if i:
            p.set_input_requant("layer_%d_a" % i)
        p.save("save_res1_%d" % i, "res1_%d" % i)
        p.layernorm("ln1_%d" % i, inp.small(d), inp.small(d))
        p.linear("c_attn_%d" % i, inp.small(3 * d * d), inp.small(3 * d), 3 * d, d)
        p.attention_seq1("attn_%d" % i)
        p.linear("c_proj_%d" % i, inp.small(d * d), inp.small(d), d, d)
        p.add_saved("add_res1_%d" % i, "res1_%d" % i)
        p.set_input_requant("mlp_fc_%d" % i)
        p.save("save_res2_%d" % i, "res2_%d" % i)
        p.layernorm("ln2_%d" % i, inp.small(d), inp.small(d))
        p.linear("mlp_fc_%d" % i, inp.small(f * d), inp.small(f), f, d)
        p.gelu("gelu_%d" % i, gelu)
        p.set_input_requant("mlp_proj_%d" % i)
        p.linear("mlp_proj_%d" % i, inp.small(d * f), inp.small(d), d, f)
        p.add_saved("add_res2_%d" % i, "res2_%d" % i)
    p.set_input_requant("lm_head")
    p.layernorm("final_ln", inp.small(d), inp.small(d))
    p.linear("lm_head", inp.small(v * d), np.zeros(v, np.uint32), v, d)
    return p


class _Qwen:
    """A model with its input, and its proofs where they are to be verified."""

    def __init__(self, inp, case):
        configs = [_layer_config(case, i) for i in range(case["layers"])]
        weights = lambda i: {k: inp.small(n) for k, n in _layer_sizes(configs[i]).items()}
        self.model = qwen.QwenModel(0, configs, weights, tables.build_silu_table(1000), tables.build_sigmoid_table(1000))
        for layer in self.model.layers:
            layer.set_binding(case["binding"], case["node"])
        self.x = inp.small(case["d_model"])
        self.proofs = self.y = None
        if case["verify"]:
            self.proofs = self.model.forward_and_prove(self.x)
            self.y = self.model.output()

    def __del__(self):
        self.model.close()


def prepare(case, seed):
    inp, kind, s = _Inputs(seed), case["kind"], {"case": case}
    if kind == "qwen":
        s["qwen"] = _Qwen(inp, case)
        return s
    ctx = s["ctx"] = zk.Context(0)
    if kind == "sumcheck":
        s["tables"] = _Buffers(ctx, [inp.field(w << case["n"]) for w in PROTOS[case["proto"]][1]])
    elif kind == "mlp":
        dims = [int(d) for d in case["dims"].split(",")]
        s["list"] = oplist.OpList(ctx, dims[0])
        for i in range(len(dims) - 1):
            s["list"].linear("fc%d" % i, inp.small(dims[i + 1] * dims[i]), inp.small(dims[i + 1]), dims[i + 1], dims[i])
            if i + 2 < len(dims):
                s["list"].relu("relu%d" % i)
        s["x"] = inp.small(dims[0])
    elif kind == "gpt2":
        s["list"], s["x"] = _gpt2(ctx, inp, case), inp.small(case["d"])
    elif kind == "attention":
        # q and k in {-1, 0, 1}, so that every score is an input of the exp table; v from the whole field
        h, kv, n, d = case["heads"], case["kv"], case["seq"], case["d"]
        s["q"], s["k"] = inp.small(h * n * d, 1), inp.small((kv or h) * n * d, 1)
        s["v"] = inp.field((kv or h) * n * d).cpu().numpy().view(np.uint32)
        s["table"] = tables.build_exp_table(100)
        if case["verify"]:
            s["proof"] = attention.prove_row_attention(s["q"], s["k"], s["v"], h, n, d, s["table"], zk.Transcript(ctx, LABEL), num_kv_heads=kv)
    elif kind == "basefold":
        n = case["coeffs"]
        s["poly"] = _Buffers(ctx, [inp.field(n), inp.field(max(1, (n - 1).bit_length()))])
    elif kind == "batch":
        sizes = [int(n) for n in case["sizes"].split(",")]
        s["polys"] = _Buffers(ctx, [inp.field(n) for n in sizes])
        torch.cuda.synchronize()
        s["batch"] = pcs.BasefoldBatch(ctx, s["polys"].bufs, [max(1, (n - 1).bit_length()) for n in sizes], case["node"])
    return s


def _bytes(proof):
    return np.frombuffer(proof, np.uint8)


def _opening_bound(n):
    """Most bytes of a Basefold opening of n coefficients: 24 queries a round, two trees, paths without a node in common."""
    log_n = max(1, (n - 1).bit_length())
    return 1024 + sum(24 * 2 * (16 * (h + 1) + 32) for h in range(1, log_n + 2))


def _kept(state, i, bound, proof):
    """Proofs with Basefold openings differ in length with the positions that the queries meet: they are kept in a buffer of
    the most that they can take, zero behind the proof, as a program that sends them on would."""
    bufs = state.setdefault("kept", {})
    if i not in bufs:
        bufs[i] = np.zeros(bound, np.uint8)
    bufs[i][:len(proof)] = np.frombuffer(proof, np.uint8)
    bufs[i][len(proof):] = 0
    return {"bytes": len(proof), "proof": bufs[i]}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "qwen":
        q = state["qwen"]
        if case["verify"]:
            ok = q.model.forward_and_verify(q.x, q.proofs, y_expected=q.y)
            return {"ok": ok, "y": q.model.output()}
        proofs = q.model.forward_and_prove(q.x)
        if case["binding"] == 2:
            bounds = [sum(_opening_bound(n) for n in _layer_sizes(_layer_config(case, i)).values()) + (1 << 18) for i in range(case["layers"])][::-1]
            return {"proofs": [_kept(state, i, bounds[i], p) for i, p in enumerate(proofs)], "y": q.model.output()}
        return {"proofs": [_bytes(p) for p in proofs], "y": q.model.output()}
    ctx = state["ctx"]
    if kind == "sumcheck":
        proof, *finals = PROTOS[case["proto"]][0](*state["tables"].bufs, case["n"], zk.Transcript(ctx, LABEL))
        return {"polys": proof.round_polys, "challenges": proof.challenges, "finals": [np.asarray(v, np.uint32) for v in finals]}
    if kind in ("mlp", "gpt2"):
        return _bytes(state["list"].prove(state["x"]))
    if kind == "attention":
        shape = (case["heads"], case["seq"], case["d"])
        tr = zk.Transcript(ctx, LABEL) if case["own_transcript"] else None
        if case["verify"]:
            ok = attention.verify_row_attention(state["proof"], state["k"], state["v"], *shape, tr or ctx, num_kv_heads=case["kv"])
            out = {"ok": ok, "v": state["v"]}
        else:
            proof, y = attention.prove_row_attention(state["q"], state["k"], state["v"], *shape, state["table"], tr or ctx, want_output=True,
                                                     num_kv_heads=case["kv"])
            out = {"proof": _bytes(proof), "y": y}
        if tr:      # the protocol goes on with the caller's transcript
            out["challenge"] = tr.squeeze_ef()
        return out
    tr = zk.Transcript(ctx, LABEL)
    if kind == "basefold":
        return _kept(state, 0, _opening_bound(case["coeffs"]), pcs.basefold_commit_and_prove(ctx, tr, *state["poly"].bufs, case["node"]))
    return _kept(state, 0, 2 * sum(_opening_bound(int(n)) for n in case["sizes"].split(",")), state["batch"].prove(tr))


# ---- what a pass cannot do without -----------------------------------------------------------------
SHA_OPS = 2600          # 32-bit operations of one SHA-256 compression (64 rounds and the message schedule, a rotation counted as one)
NODE_OPS = 700          # of one Merkle node
EF_MUL = 32             # of one extension-field product: sixteen multiply-adds


def _sumcheck_work(n, widths):
    elements = float(1 << n)
    return sum(widths) * elements * 4, 2 * elements * len(widths) * 3 * EF_MUL + n * 5 * SHA_OPS


def _basefold_work(n):
    log_n = max(1, (n - 1).bit_length())
    code = 2.0 * (1 << log_n)
    return 4.0 * n + 4 * code, 4 * code * log_n / 2 + 2 * code * NODE_OPS + log_n * 26 * SHA_OPS


def work(case):
    kind = case["kind"]
    if kind == "sumcheck":
        b, f = _sumcheck_work(case["n"], PROTOS[case["proto"]][1])
    elif kind in ("mlp", "gpt2"):
        if kind == "mlp":
            dims = [int(d) for d in case["dims"].split(",")]
            pairs = list(zip(dims[1:], dims))
        else:
            d = case["d"]
            pairs = [(3 * d, d), (d, d), (4 * d, d), (d, 4 * d)] * case["layers"] + [(case["vocab"], d)]
        words = float(sum(m * n for m, n in pairs))
        vectors = float(sum(m + n for m, n in pairs))
        # weights once; forward and fold two operations a weight each; every vector absorbed once (sixteen words a compression), 26 rounds a linear
        b, f = 4 * words, 4 * words + (vectors / 16 + 150 * len(pairs)) * SHA_OPS
    elif kind == "qwen":
        sizes = [_layer_sizes(_layer_config(case, i)) for i in range(case["layers"])]
        words = float(sum(sum(s.values()) for s in sizes))
        b, f = 4 * words, 10 * words + len(sizes) * 6000 * SHA_OPS
        if case["binding"] == 2:
            for s in sizes:
                for k, n in s.items():
                    if k.startswith("w_"):
                        wb, wf = _basefold_work(n)
                        b, f = b + wb, f + wf
    elif kind == "attention":
        h, kv, n, d = case["heads"], case["kv"] or case["heads"], case["seq"], case["d"]
        rows = h * n
        b = 4.0 * (h + 2 * kv) * n * d + rows * 4.0 * (6 * n + d)
        f = rows * (8.0 * n * d + (150 + n / 4) * SHA_OPS)
    else:
        sizes = [case["coeffs"]] if kind == "basefold" else [int(n) for n in case["sizes"].split(",")]
        parts = [_basefold_work(n) for n in sizes]
        # a batch proof reads the committed codewords and builds one chain of trees
        b = sum(p[0] for p in parts)
        f = max(p[1] for p in parts)
    return {"bytes": b, "flops": f}


def tolerance(case):
    """All arithmetic is exact: proofs, verdicts and challenges are the same bytes whatever the implementation."""
    return "exact"
