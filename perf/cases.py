"""The workloads this framework's speed is judged by: decode steps, their projections, and prefill-sized norms and appends.

Every case goes through the public entry points (``ops``, ``w4a16``, ``chain``) the way a serving program calls them:
eagerly, or -- ``graph: True`` -- as a step captured once with ``timing.capture`` and replayed, which is how a decode
loop runs.  A pass walks several layers' weights where one layer's would stay in the 126 MB L2 of the previous pass.

``listed()`` are the fixed cases, ``draw(rng)`` one more of the same ranges, ``exact`` the results in 64-bit arithmetic.
"""

from __future__ import annotations

import math

import torch

from cross_dsl_kernels_b200 import workloads as wl
from cross_dsl_kernels_b200.chain import ChainConfig, DecodeLayerChain
from cross_dsl_kernels_b200.ops import (decode_linear, fused_residual_rmsnorm, paged_decode_attention,
                                        rope_gqa_paged_kv_append)
from cross_dsl_kernels_b200.timing import capture
from cross_dsl_kernels_b200.w4a16 import w4a16_linear

_DTYPES = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}
_EPS = 1e-6


def listed() -> list[dict]:
    return [
        # The smallest call of the path: the norm in front of one decode step, called eagerly.  All launch and host cost.
        dict(name="norm_bf16_16x4096", kind="norm", rows=16, hidden=4096, dtype="bf16"),
        # A prefill-sized norm: 4096 rows, the largest of the norm sizes this repository measures.
        dict(name="norm_bf16_4096x4096", kind="norm", rows=4096, hidden=4096, dtype="bf16"),
        # FP32 projections of single-sequence decode, weights as [K, N]; three layers' output projections.
        dict(name="linear_kn_m1_n4096", kind="linear", m=1, k=4096, n=4096, layout="KN", layers=3),
        # A ragged small batch on an odd width: neither M nor N fits a tile.
        dict(name="linear_kn_m6_n11012", kind="linear", m=6, k=4096, n=11012, layout="KN", layers=2),
        # The widest FP32 projection at the full decode batch, weights as [N, K]; two layers.
        dict(name="linear_nk_m16_n14336", kind="linear", m=16, k=4096, n=14336, layout="NK", layers=2),
        # A batch of more than sixteen sequences (or several draft tokens for each): the upper end of M.
        dict(name="linear_nk_m64_n4096", kind="linear", m=64, k=4096, n=4096, layout="NK", layers=3),
        # The INT4 down projection of an MLP (long K), captured over four layers.
        dict(name="int4_m16_k14336_n4096", kind="int4", m=16, k=14336, n=4096, group=128, bias=True, layers=4, graph=True),
        # Rotation and cache append of a prefill chunk: 4096 tokens, half of each head rotated.
        dict(name="append_bf16_hnd_4096", kind="append", tokens=4096, q_heads=32, kv_heads=8, head_dim=128, rope_dim=64,
             page_size=16, layout="HND", interleaved=False, dtype="bf16"),
        # Attention read of a larger batch with contexts of every length up to 2048.
        dict(name="attend_bf16_64x2048", kind="attend", tokens=64, q_heads=32, kv_heads=8, head_dim=128, context=2048,
             page_size=16, layout="HND", dtype="bf16"),
        # A decode step of one sequence with a long context: four layers, captured, dependent launches.
        dict(name="step_t1_ctx8192", kind="step", tokens=1, hidden=4096, head_dim=128, kv_heads=8, mlp=14336, context=8192,
             page_size=16, layers=4, graph=True, dependent=True),
        # A decode step of a small batch called eagerly: two layers of the narrower MLP, short context.
        dict(name="step_t4_ctx1024_eager", kind="step", tokens=4, hidden=4096, head_dim=128, kv_heads=8, mlp=11008, context=1024,
             page_size=16, layers=2, graph=False, dependent=False),
        # The full decode batch with long contexts: four layers, captured, dependent launches.
        dict(name="step_t16_ctx8192", kind="step", tokens=16, hidden=4096, head_dim=128, kv_heads=8, mlp=14336, context=8192,
             page_size=16, layers=4, graph=True, dependent=True),
    ]


def _log_int(rng, lo: int, hi: int, multiple: int = 1) -> int:
    """An integer spread evenly over its logarithm in [lo, hi], a multiple of ``multiple``."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(lo, min(hi, int(round(v / multiple)) * multiple))


def draw(rng) -> dict:
    kind = rng.choice(["norm", "linear", "linear", "int4", "int4", "append", "attend", "step", "step"])
    if kind == "norm":
        hidden = _log_int(rng, 1024, 8192, rng.choice([8, 128, 1024]))
        return dict(kind=kind, rows=_log_int(rng, 1, 4096), hidden=hidden, dtype=rng.choice(["f32", "bf16", "f16"]))
    if kind == "linear":
        m, k = _log_int(rng, 1, 64), _log_int(rng, 1024, 14336, rng.choice([4, 64, 512]))
        n, layout = _log_int(rng, 1024, 14336, rng.choice([4, 32])), rng.choice(["KN", "NK"])
        layers = max(1, min(4, int(240e6 / (4 * k * n)), int(900e6 / (4 * k * n * -(-m // 16)))))
        return dict(kind=kind, m=m, k=k, n=n, layout=layout, layers=layers)
    if kind == "int4":
        m, k = _log_int(rng, 1, 16), _log_int(rng, 1024, 14336, rng.choice([256, 512, 1024]))
        n, group = _log_int(rng, 1024, 28672, rng.choice([8, 16, 128])), rng.choice([64, 128, 128])
        return dict(kind=kind, m=m, k=k, n=n, group=group, bias=rng.random() < 0.5, layers=rng.choice([2, 4]), graph=rng.random() < 0.7)
    head_dim = rng.choice([64, 128, 128])
    kv_heads, group = rng.choice([2, 4, 8]), rng.choice([2, 4, 4, 8])
    if kind == "append":
        return dict(kind=kind, tokens=_log_int(rng, 1, 4096), q_heads=kv_heads * group, kv_heads=kv_heads, head_dim=head_dim,
                    rope_dim=head_dim // rng.choice([1, 1, 2]), page_size=rng.choice([16, 32, 64]), layout=rng.choice(["NHD", "HND"]),
                    interleaved=rng.random() < 0.3, dtype=rng.choice(["f32", "bf16", "f16"]))
    if kind == "attend":
        tokens = _log_int(rng, 1, 64)
        return dict(kind=kind, tokens=tokens, q_heads=kv_heads * group, kv_heads=kv_heads, head_dim=head_dim,
                    context=_log_int(rng, 128, min(8192, 131072 // tokens)), page_size=rng.choice([16, 32, 64]),
                    layout=rng.choice(["NHD", "HND"]), dtype=rng.choice(["bf16", "f16", "f16", "f32"]))
    hidden = rng.choice([1024, 2048, 3072, 4096, 4096])
    q_heads = hidden // head_dim
    kv_heads = q_heads // rng.choice([1, 2, 4, 4, 8])
    page_size = rng.choice([16, 32, 64])
    graph = rng.random() < 0.75
    return dict(kind=kind, tokens=_log_int(rng, 1, 16), hidden=hidden, head_dim=head_dim, kv_heads=kv_heads,
                mlp=_log_int(rng, 2048, 14336, rng.choice([8, 256])), context=_log_int(rng, 256, 8192, 64), page_size=page_size,
                layers=rng.choice([2, 3, 4]), graph=graph, dependent=graph and rng.random() < 0.8)


def _config(case: dict) -> ChainConfig:
    return ChainConfig(tokens=case["tokens"], hidden=case["hidden"], q_heads=case["hidden"] // case["head_dim"],
                       kv_heads=case["kv_heads"], head_dim=case["head_dim"], mlp=case["mlp"], context=case["context"],
                       page_size=case["page_size"])


def _paged(case: dict, gen: torch.Generator, context: int) -> dict:
    """Caches and index tensors of ``tokens`` sequences whose pages are one random permutation."""
    dtype, tokens, page = _DTYPES[case["dtype"]], case["tokens"], case["page_size"]
    per_seq = -(-context // page)
    inner = (page, case["kv_heads"]) if case["layout"] == "NHD" else (case["kv_heads"], page)
    shape = (tokens * per_seq, *inner, case["head_dim"])
    return dict(k_cache=torch.randn(shape, generator=gen, device="cuda", dtype=dtype),
                v_cache=torch.randn(shape, generator=gen, device="cuda", dtype=dtype),
                positions=torch.randint(0, context, (tokens,), generator=gen, device="cuda"),
                page_table=torch.randperm(tokens * per_seq, generator=gen, device="cuda").reshape(tokens, per_seq),
                sequence_ids=torch.arange(tokens, device="cuda"))


def prepare(case: dict, seed: int) -> dict:
    gen = torch.Generator(device="cuda").manual_seed(seed)

    def normal(*shape, dtype=torch.float32):
        return torch.randn(*shape, generator=gen, device="cuda", dtype=dtype)

    kind = case["kind"]
    st = dict(case=case)
    if kind == "norm":
        dtype = _DTYPES[case["dtype"]]
        rows, hidden = case["rows"], case["hidden"]
        st.update(x=normal(rows, hidden, dtype=dtype), residual=normal(rows, hidden, dtype=dtype),
                  weight=(1 + 0.1 * normal(hidden)).to(dtype))
    elif kind == "linear":
        m, k, n = case["m"], case["k"], case["n"]
        shape = (k, n) if case["layout"] == "KN" else (n, k)
        st.update(x=normal(m, k), weights=[normal(*shape).div_(k ** 0.5) for _ in range(case["layers"])],
                  biases=[0.02 * normal(n) for _ in range(case["layers"])])
    elif kind == "int4":
        m, k, n = case["m"], case["k"], case["n"]
        layers = range(case["layers"])
        st.update(x=normal(m, k, dtype=torch.float16),
                  packed=[torch.randint(0, 256, (n, (k + 1) // 2), generator=gen, device="cuda", dtype=torch.uint8) for _ in layers],
                  scales=[(0.005 + 0.015 * torch.rand(n, -(-k // case["group"]), generator=gen, device="cuda")).half() for _ in layers],
                  biases=[(0.02 * normal(n)).half() if case["bias"] else None for _ in layers])
    elif kind == "append":
        tokens, dim, rope = case["tokens"], case["head_dim"], case["rope_dim"]
        dtype = _DTYPES[case["dtype"]]
        per_seq = 256  # positions a sequence may reach; one page table row per token
        st.update(_paged(dict(case, tokens=max(1, tokens // 64)), gen, per_seq))
        # a prefill chunk: runs of consecutive positions, at most 64 tokens of a sequence
        run_of = torch.arange(tokens, device="cuda")
        seqs = st["page_table"].shape[0]
        st["sequence_ids"] = run_of % seqs
        start = torch.randint(0, per_seq - (tokens - 1) // seqs, (seqs,), generator=gen, device="cuda")
        st["positions"] = start[st["sequence_ids"]] + run_of // seqs
        inv_freq = 10000.0 ** (-torch.arange(0, rope, 2, device="cuda").float() / rope)
        angle = torch.arange(per_seq, device="cuda").float()[:, None] * inv_freq[None, :]
        st.update(q=normal(tokens, case["q_heads"], dim, dtype=dtype), k=normal(tokens, case["kv_heads"], dim, dtype=dtype),
                  v=normal(tokens, case["kv_heads"], dim, dtype=dtype), cos=angle.cos(), sin=angle.sin())
    elif kind == "attend":
        st.update(_paged(case, gen, case["context"]))
        st["q"] = normal(case["tokens"], case["q_heads"], case["head_dim"], dtype=_DTYPES[case["dtype"]])
    else:
        chain = DecodeLayerChain(_config(case), layers=case["layers"], seed=seed, dependent_launch=case["dependent"], attention=True)
        chain.k_cache.normal_(generator=gen)
        chain.v_cache.normal_(generator=gen)
        st["chain"] = chain
    if case.get("graph"):
        outputs: list = []
        st["replay"] = capture([lambda: _call(st)], outputs=outputs)
        st["outputs"] = outputs[0]
    return st


def _call(st: dict):
    case = st["case"]
    kind = case["kind"]
    if kind == "norm":
        return fused_residual_rmsnorm(st["x"], st["residual"], st["weight"], _EPS)
    if kind == "linear":
        return [decode_linear(st["x"], w, b, weight_layout=case["layout"]) for w, b in zip(st["weights"], st["biases"])]
    if kind == "int4":
        return [w4a16_linear(st["x"], p, s, b, group_size=case["group"])
                for p, s, b in zip(st["packed"], st["scales"], st["biases"])]
    if kind == "append":
        q_out = rope_gqa_paged_kv_append(st["q"], st["k"], st["v"], st["cos"], st["sin"], st["positions"], st["page_table"],
                                         st["sequence_ids"], st["k_cache"], st["v_cache"], page_size=case["page_size"],
                                         rope_dim=case["rope_dim"], interleaved=case["interleaved"], kv_layout=case["layout"])
        return q_out, st["k_cache"], st["v_cache"]
    if kind == "attend":
        return paged_decode_attention(st["q"], st["k_cache"], st["v_cache"], st["positions"], st["page_table"], st["sequence_ids"],
                                      page_size=case["page_size"], kv_layout=case["layout"], context_hint=case["context"])
    out = st["chain"].run_layers()
    return {**out, "k_cache": st["chain"].k_cache, "v_cache": st["chain"].v_cache}


def run(st: dict):
    if "replay" in st:
        st["replay"].replay()
        return st["outputs"]
    return _call(st)


def work(case: dict) -> dict:
    """Bytes: every operand read once, every result written once.  Contexts are uniform in [1, context]."""
    kind = case["kind"]
    if kind == "norm":
        return dict(bytes=wl.rmsnorm_bytes(case["rows"], case["hidden"], _DTYPES[case["dtype"]]), flops=0)
    if kind == "linear":
        m, k, n, layers = case["m"], case["k"], case["n"], case["layers"]
        return dict(bytes=layers * wl.projection_bytes(m, k, n, True), flops=2 * layers * m * k * n)
    if kind == "int4":
        m, k, n, layers = case["m"], case["k"], case["n"], case["layers"]
        return dict(bytes=layers * wl.w4a16_bytes(m, k, n, case["group"], case["bias"]), flops=2 * layers * m * k * n)
    if kind == "append":
        return dict(bytes=wl.rope_bytes(case["tokens"], case["q_heads"], case["kv_heads"], case["head_dim"], case["rope_dim"],
                                        _DTYPES[case["dtype"]]), flops=0)

    def attention(tokens, q_heads, kv_heads, dim, elt):
        positions = tokens * (case["context"] + 1) / 2
        return 2 * positions * kv_heads * dim * elt + 2 * tokens * q_heads * dim * elt, 4 * positions * q_heads * dim

    if kind == "attend":
        nbytes, flops = attention(case["tokens"], case["q_heads"], case["kv_heads"], case["head_dim"], _DTYPES[case["dtype"]].itemsize)
        return dict(bytes=nbytes, flops=flops)
    c = _config(case)
    nbytes, flops = attention(c.tokens, c.q_heads, c.kv_heads, c.head_dim, 2)
    nbytes += c.algorithmic_bytes() + 3 * 2 * c.tokens * c.mlp
    flops += 2 * c.tokens * c.hidden * (c.qkv_cols + 2 * c.mlp)
    return dict(bytes=case["layers"] * nbytes, flops=case["layers"] * flops)


def tolerance(case: dict):
    """About four times what a 64-bit computation of the same path differs from the results by: the rounding of the output
    type for one op; for a step, FP16 roundings of every stage carried through the layers."""
    kind = case["kind"]
    if kind == "append":
        return "exact"  # separately rounded FP32 operations: every byte is defined
    if kind == "linear":
        return {"rel": 1e-5}
    if kind == "step":
        return {"rel": 1e-2}
    dtype = case.get("dtype", "f16")
    return {"rel": {"f32": 1e-5 if kind == "attend" else 2e-6, "f16": 1e-3, "bf16": 7e-3}[dtype]}


def _norm64(x, residual, weight):
    s = x + residual
    return s / (s.square().mean(-1, keepdim=True) + _EPS).sqrt() * weight, s


def _int4_64(x, packed, scales, bias, group):
    """x [M, K] times the weights the format defines: half(q * scale), low nibble first."""
    k = x.shape[1]
    codes = torch.stack((packed & 15, packed >> 4), dim=2).flatten(1)[:, :k].float() - 8
    w = (codes * scales.float().repeat_interleave(group, dim=1)[:, :k]).half()
    y = x @ w.double().t()
    return y if bias is None else y + bias.double()


def _rotate64(x, cos, sin, rope, interleaved):
    """The first ``rope`` dims of each head of x [tokens, heads, dim] turned by the angles of cos, sin [tokens, rope / 2]."""
    out, half = x.clone(), rope // 2
    one, two = (slice(0, rope, 2), slice(1, rope, 2)) if interleaved else (slice(0, half), slice(half, rope))
    a, b, c, s = x[..., one], x[..., two], cos.double()[:, None, :half], sin.double()[:, None, :half]
    out[..., one], out[..., two] = a * c - b * s, a * s + b * c
    return out


def _slots(positions, page_table, sequence_ids, page):
    return page_table[sequence_ids, positions // page], positions % page


def _attend64(q, k_cache, v_cache, positions, page_table, sequence_ids, page, layout):
    out = torch.empty_like(q, dtype=torch.float64)
    for t in range(q.shape[0]):
        js = torch.arange(int(positions[t]) + 1, device=q.device)
        pages, offs = _slots(js, page_table, sequence_ids[t].expand(js.numel()), page)
        k, v = ((c[pages, offs] if layout == "NHD" else c[pages, :, offs]).double() for c in (k_cache, v_cache))
        heads = q[t].double().reshape(k.shape[1], -1, q.shape[2])  # [kv_heads, group, dim]
        p = torch.softmax(torch.einsum("hgd,jhd->hgj", heads, k) * q.shape[2] ** -0.5, dim=-1)
        out[t] = torch.einsum("hgj,jhd->hgd", p, v).reshape(q.shape[1:])
    return out


def exact(case: dict, seed: int):
    """What ``run`` returns for these inputs, every operation in 64 bits and nothing rounded between them."""
    kind = case["kind"]
    st = prepare(dict(case, graph=False), seed)
    if kind == "norm":
        return _norm64(st["x"].double(), st["residual"].double(), st["weight"].double())
    if kind == "linear":
        ws = (w if case["layout"] == "KN" else w.t() for w in st["weights"])
        return [st["x"].double() @ w.double() + b.double() for w, b in zip(ws, st["biases"])]
    if kind == "int4":
        return [_int4_64(st["x"].double(), p, s, b, case["group"]) for p, s, b in zip(st["packed"], st["scales"], st["biases"])]
    if kind == "append":
        pos, rope = st["positions"], case["rope_dim"]
        pages, offs = _slots(pos, st["page_table"], st["sequence_ids"], case["page_size"])
        at = (pages, offs) if case["layout"] == "NHD" else (pages, slice(None), offs)
        turn = [_rotate64(st[n].double(), st["cos"][pos], st["sin"][pos], rope, case["interleaved"]) for n in ("q", "k")]
        k_cache, v_cache = st["k_cache"].double(), st["v_cache"].double()
        k_cache[at], v_cache[at] = turn[1], st["v"].double()
        return turn[0], k_cache, v_cache
    if kind == "attend":
        return _attend64(st["q"], st["k_cache"], st["v_cache"], st["positions"], st["page_table"], st["sequence_ids"],
                         case["page_size"], case["layout"])
    chain, c = st["chain"], _config(case)
    pos, table, seqs = (chain.dev[n] for n in ("positions", "page_table", "sequence_ids"))
    k_cache, v_cache = chain.k_cache.double(), chain.v_cache.double()
    at = _slots(pos, table, seqs, c.page_size)
    h, res, out = chain.dev["h"].double(), chain.dev["res"].double(), {}
    for layer in chain.layers:
        n1, r1 = _norm64(h, res, layer["w1"].double())
        qkv = _int4_64(n1, layer["qkv_packed"], layer["qkv_scales"], None, c.group)
        heads = qkv.view(c.tokens, -1, c.head_dim)
        cos, sin = chain.dev["cos"][pos], chain.dev["sin"][pos]
        q_rot = _rotate64(heads[:, :c.q_heads], cos, sin, c.head_dim, False)
        k_cache[at] = _rotate64(heads[:, c.q_heads:c.q_heads + c.kv_heads], cos, sin, c.head_dim, False)
        v_cache[at] = heads[:, c.q_heads + c.kv_heads:]
        attn = _attend64(q_rot, k_cache, v_cache, pos, table, seqs, c.page_size, "NHD").view(c.tokens, c.hidden)
        n2, r2 = _norm64(attn, r1, layer["w2"].double())
        up = _int4_64(n2, layer["up_packed"], layer["up_scales"], None, c.group)
        act = torch.nn.functional.silu(up[:, c.mlp:]) * up[:, :c.mlp]
        out = dict(n1=n1, r1=r1, qkv=qkv, q_rot=q_rot, attn=attn, n2=n2, r2=r2, up=up, up_all=up, act=act)
        h, res = n2, r2
    return {**out, "k_cache": k_cache, "v_cache": v_cache}
