"""Performance cases of frink_b200: what its users have it do, through its public entry points.

  host      frink-core's decode matvec on host buffers (`gpu.launch_<kind>_matvec`): x up, y down, weights resident
  matvec    one projection of every layer in turn on device tensors (`device.gemv`), called one by one or from a CUDA graph
  gemm      a prompt's projection (`device.gemm`, `device.gemm_q8k`)
  moe       one routed layer (`device.moe_layer`): a few decode rows, or the rows of a prompt
  prompt    a prompt through a resident decoder (`Decoder.forward`)
  generate  prompt + greedy decode from the captured graph, one sequence or a batch (`Decoder.replay`, `replay_seqs`)

Weights are random matrices quantized to GGUF blocks on the GPU (simple min / max quantizers: every block has real scales,
mins and codes); activations are N(0, 1).  Shapes are those of the benchmark's three models (Llama-3.2-3B, Qwen3-30B-A3B,
gpt-oss-20b) with fewer layers, and their neighbourhood."""
import math

import torch

from frink_b200 import device, gpu
from frink_b200.decoder import Decoder, DecoderConfig, LayerWeights
from frink_b200.prefill import RoutedLayer

TAG = {"q8_0": 8, "q4_k": 12, "q5_k": 13, "q6_k": 14, "bf16": 30, "mxfp4": 39}
BLOCK = {"q8_0": (32, 34), "q4_k": (256, 144), "q5_k": (256, 176), "q6_k": (256, 210), "bf16": (1, 2), "mxfp4": (32, 17)}


# ---- the cases ----------------------------------------------------------------
def listed():
    return [
        # the call frink-core makes per projection and token: the smallest one, latency is all there is
        dict(name="host q4_k 3072x3072", op="host", kind="q4_k", rows=3072, cols=3072),
        # one decode matvec on device tensors, the benchmark's headline shape
        dict(name="matvec q4_k 8192x3072", op="matvec", kind="q4_k", rows=8192, cols=3072, batch=1, mats=1, graph=False),
        # a token's down projections, layer after layer out of HBM, replayed from a graph as a serving loop does
        dict(name="matvecs q4_k 3072x8192 graph", op="matvec", kind="q4_k", rows=3072, cols=8192, batch=1, mats=28, graph=True),
        # the same for a batch of eight sequences in the larger K-quant
        dict(name="matvecs q6_k 8192x3072 b8 graph", op="matvec", kind="q6_k", rows=8192, cols=3072, batch=8, mats=12, graph=True),
        # a 512-token prompt's largest projection, decode's activation rule
        dict(name="gemm q4_k 8192x3072 m512", op="gemm", kind="q4_k", rows=8192, cols=3072, m=512, acts="q8_1"),
        # a short ragged prompt
        dict(name="gemm q6_k 3072x8192 m77", op="gemm", kind="q6_k", rows=3072, cols=8192, m=77, acts="q8_1"),
        # a long prompt on the CPU activation rule
        dict(name="gemm q4_k 8192x3072 m2048 q8_k", op="gemm", kind="q4_k", rows=8192, cols=3072, m=2048, acts="q8_k"),
        # Qwen3-MoE's routed layer for one token
        dict(name="moe q4_k 128x8 row", op="moe", kind="q4_k", experts=128, k=8, hidden=2048, ffn=768, rows=1, biased=False),
        # gpt-oss's routed layer for a 512-token prompt
        dict(name="moe mxfp4 32x4 prompt", op="moe", kind="mxfp4", experts=32, k=4, hidden=2880, ffn=2880, rows=512, biased=True),
        # 512 prompt tokens through Llama-3.2-3B's layers
        dict(name="prompt llama 512", op="prompt", model="dense", layers=4, hidden=3072, heads=24, kv=8, head_dim=128, ffn=8192, experts=0, k=0,
             vocab=128256, prompt=512, new=0, seqs=1, acts="q8_k"),
        # chat with one user: Llama-3.2-3B's layers, 128 prompt tokens, 32 new ones
        dict(name="generate llama", op="generate", model="dense", layers=4, hidden=3072, heads=24, kv=8, head_dim=128, ffn=8192, experts=0, k=0,
             vocab=128256, prompt=128, new=32, seqs=1, acts="q8_1"),
        # serving eight users: Qwen3-MoE's layers
        dict(name="generate qwen3moe b8", op="generate", model="routed", layers=2, hidden=2048, heads=32, kv=4, head_dim=128, ffn=768,
             experts=128, k=8, vocab=151936, prompt=16, new=48, seqs=8, acts="q8_1"),
    ]


def _lg(rng, lo, hi, step=1):
    """A whole number of [lo, hi], log-uniform, a multiple of step."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return int(min(hi // step * step, max(-(-lo // step) * step, round(v / step) * step)))


def draw(rng):
    op = rng.choice(["host", "matvec", "matvec", "matvec", "gemm", "gemm", "gemm", "moe", "moe", "prompt", "generate", "generate"])
    if op == "host":
        kind = rng.choice(["q4_k", "q4_k", "q5_k", "q6_k", "q8_0", "mxfp4"])
        return dict(op=op, kind=kind, rows=_lg(rng, 512, 16384), cols=_lg(rng, 512, 8192, BLOCK[kind][0]))
    if op == "matvec":
        kind = rng.choice(["q4_k", "q4_k", "q6_k", "q6_k", "q8_0", "mxfp4", "q5_k", "bf16"])
        rows, cols = _lg(rng, 512, 16384), _lg(rng, 512, 8192, max(32, BLOCK[kind][0]))
        graph = rng.random() < 0.6
        most = max(1, int(400e6 / (rows * _row_bytes(kind, cols))))
        mats = min(most, _lg(rng, 4, 28) if graph else _lg(rng, 1, 8))
        return dict(op=op, kind=kind, rows=rows, cols=cols, batch=rng.choice([1, 1, 1, 2, 3, 4, 5, 6, 7, 8]), mats=mats, graph=graph)
    if op == "gemm":
        kind = rng.choice(["q4_k", "q4_k", "q6_k", "q8_0", "mxfp4"])
        return dict(op=op, kind=kind, rows=_lg(rng, 256, 8192), cols=_lg(rng, 512, 4096, BLOCK[kind][0]), m=_lg(rng, 9, 2048),
                    acts=rng.choice(["q8_1", "q8_k"]) if kind == "q4_k" else "q8_1")
    if op == "moe":
        kind = rng.choice(["q4_k", "q4_k", "q8_0", "mxfp4", "mxfp4"])
        step = BLOCK[kind][0]
        experts = _lg(rng, 8, 128)
        hidden = _lg(rng, 512, 2880, step)
        ffn = _lg(rng, 256, min(2880, int(3.2e8 / (experts * hidden))), step)
        return dict(op=op, kind=kind, experts=experts, k=rng.randint(1, 8), hidden=hidden, ffn=ffn,
                    rows=rng.choice([1, 1, rng.randint(2, 8), _lg(rng, 9, 512), _lg(rng, 9, 512)]), biased=kind == "mxfp4")
    model = rng.choice(["dense", "dense", "routed", "oai"])
    head_dim = 64 if model == "oai" else 128
    kv = rng.choice([2, 4, 8])
    heads = kv * rng.choice([2, 3, 4, 8] if model != "oai" else [4, 8])
    heads = min(heads, 32 if model != "oai" else 64) // kv * kv
    hidden = 2880 if model == "oai" else _lg(rng, 1024, 3072, 256)
    c = dict(op=op, model=model, layers=rng.randint(1, 3), hidden=hidden, heads=heads, kv=kv, head_dim=head_dim, vocab=_lg(rng, 32000, 128256))
    if model == "dense":
        c.update(ffn=_lg(rng, 2048, 8192, 256), experts=0, k=0)
    elif model == "routed":
        c.update(ffn=_lg(rng, 512, 1024, 256), experts=_lg(rng, 16, 128), k=rng.randint(2, 8))
    else:
        c.update(ffn=2880, experts=_lg(rng, 8, 32), k=4)
    acts = rng.choice(["q8_1", "q8_k"]) if model == "dense" else "q8_1"
    if op == "prompt":
        return dict(c, prompt=_lg(rng, 9, 512), new=0, seqs=1, acts=acts)
    seqs = rng.choice([1, 1, rng.randint(2, 8)])
    return dict(c, prompt=_lg(rng, 9, 200) if seqs == 1 else _lg(rng, 9, 24), new=_lg(rng, 8, 32), seqs=seqs, acts=acts)


# ---- GGUF blocks of random weights, made on the GPU --------------------------------
def _row_bytes(kind, cols):
    return cols // BLOCK[kind][0] * BLOCK[kind][1]


def _half_bytes(v):
    """f32 [n] -> (the f16 rounding as f32, its two bytes [n, 2])."""
    h = v.to(torch.float16)
    return h.float(), h.view(torch.uint8).view(-1, 2)


def _safe_div(a, b):
    return torch.where(b != 0, a / torch.where(b != 0, b, torch.ones_like(b)), torch.zeros_like(a))


def _encode_k45(w, high):
    """Q4_K (high: Q5_K) blocks of w [n, 256]: sub-blocks of 32 with a 6-bit scale and a 6-bit min each."""
    s = w.view(-1, 8, 32)
    top = 31 if high else 15
    mn = (-s.amin(-1)).clamp_min(0)
    sc = (s.amax(-1) + mn) / top
    d, db = _half_bytes(sc.amax(-1) / 63)
    dm, mb = _half_bytes(mn.amax(-1) / 63)
    qs = _safe_div(sc, d[:, None]).round().clamp(0, 63)
    qm = _safe_div(mn, dm[:, None]).round().clamp(0, 63)
    q = _safe_div(s + (dm[:, None] * qm)[..., None], (d[:, None] * qs)[..., None]).round().clamp(0, top).to(torch.uint8)
    a, b = qs.to(torch.uint8), qm.to(torch.uint8)
    packed = torch.cat([a[:, :4] | ((a[:, 4:] >> 4) << 6), b[:, :4] | ((b[:, 4:] >> 4) << 6), (a[:, 4:] & 15) | ((b[:, 4:] & 15) << 4)], 1)
    lo = q & 15
    quants = (lo[:, 0::2] | (lo[:, 1::2] << 4)).reshape(-1, 128)
    parts = [db, mb, packed]
    if high:
        bit = torch.arange(8, device=w.device, dtype=torch.uint8)[None, :, None]
        parts.append(((q >> 4) << bit).sum(1, dtype=torch.uint8))
    return torch.cat(parts + [quants], 1)


def _encode_q6_k(w):
    s = w.view(-1, 16, 16)
    sc = s.abs().amax(-1) / 31
    d, db = _half_bytes(sc.amax(-1) / 127)
    qs = _safe_div(sc, d[:, None]).round().clamp(0, 127)
    q = (_safe_div(s, (d[:, None] * qs)[..., None]).round().clamp(-32, 31) + 32).to(torch.uint8).view(-1, 2, 4, 32)
    lo, hi = q & 15, q >> 4
    ql = torch.cat([lo[:, :, 0] | (lo[:, :, 2] << 4), lo[:, :, 1] | (lo[:, :, 3] << 4)], -1).reshape(-1, 128)
    qh = (hi[:, :, 0] | (hi[:, :, 1] << 2) | (hi[:, :, 2] << 4) | (hi[:, :, 3] << 6)).reshape(-1, 64)
    return torch.cat([ql, qh, qs.to(torch.uint8), db], 1)


def _encode_q8_0(w):
    s = w.view(-1, 32)
    d, db = _half_bytes(s.abs().amax(-1) / 127)
    q = _safe_div(s, d[:, None].expand_as(s)).round().clamp(-127, 127).to(torch.int8)
    return torch.cat([db, q.view(torch.uint8)], 1)


def _encode_mxfp4(w):
    s = w.view(-1, 32)
    e = (torch.floor(torch.log2(s.abs().amax(-1).clamp_min(1e-30))) - 2 + 127).clamp(1, 254)
    edges = torch.tensor([0.25, 0.75, 1.25, 1.75, 2.5, 3.5, 5.0], device=w.device)
    code = torch.bucketize(s.abs() * torch.exp2(127 - e)[:, None], edges).to(torch.uint8) | ((s < 0).to(torch.uint8) << 3)
    return torch.cat([e.to(torch.uint8)[:, None], code[:, :16] | (code[:, 16:] << 4)], 1)


def _encode(kind, w):
    w = w.reshape(-1, BLOCK[kind][0])
    if kind == "bf16":
        return w.to(torch.bfloat16).view(torch.uint8).reshape(-1)
    fn = {"q4_k": lambda v: _encode_k45(v, False), "q5_k": lambda v: _encode_k45(v, True), "q6_k": _encode_q6_k, "q8_0": _encode_q8_0,
          "mxfp4": _encode_mxfp4}[kind]
    return fn(w).reshape(-1)


def _matrix(gen, kind, rows, cols, std=0.02, near=None):
    """GGUF bytes of a random [rows, cols] matrix (plus near(lo, hi) for its rows lo .. hi - 1), a slab of rows at a time."""
    slab, out = max(1, (1 << 26) // cols), []
    for lo in range(0, rows, slab):
        hi = min(rows, lo + slab)
        w = torch.randn((hi - lo, cols), generator=gen, device="cuda") * std
        out.append(_encode(kind, w if near is None else w + near(lo, hi)))
    return torch.cat(out)


# ---- what a user's program holds before the call ---------------------------------
def _decoder(case, gen):
    H, hd, F, E = case["hidden"], case["head_dim"], case["ffn"], case["experts"]
    hq, hkv = case["heads"] * hd, case["kv"] * hd
    model, V = case["model"], case["vocab"]
    oai, routed = model == "oai", model != "dense"
    cfg = DecoderConfig(
        n_layers=case["layers"], hidden=H, n_heads=case["heads"], n_kv=case["kv"], head_dim=hd, ffn=F, vocab=V,
        rope_theta={"dense": 500000.0, "routed": 1000000.0, "oai": 150000.0}[model], eps=1e-6 if model == "routed" else 1e-5, neox=routed,
        qk_norm=model == "routed", n_experts=E, top_k=case["k"], oai=oai, sliding_window=128 if oai else 0, swa_period=2 if oai else 0)
    rnd = lambda *n: torch.randn(n, generator=gen, device="cuda")
    host = lambda t: t.cpu().numpy()
    norm = lambda n: host(1 + 0.1 * rnd(n))
    raw = lambda kind, r, c, std=0.02: host(_matrix(gen, kind, r, c, std))

    def layers():       # one at a time: a layer's host bytes live until they are uploaded
        for i in range(case["layers"]):
            if oai:
                kd = dict(wq="bf16", wk="bf16", wv="bf16", wo="bf16", experts="mxfp4")
            elif routed:
                kd = dict(wq="q8_0", wk="q8_0", wv="q8_0", wo="q8_0", experts="q4_k")
            else:       # the Q4_K_M mix: every other layer keeps v and down in Q6_K
                hi = "q6_k" if i % 2 else "q4_k"
                kd = dict(wq="q4_k", wk="q4_k", wv=hi, wo="q4_k", gate="q4_k", up="q4_k", down=hi)
            L = LayerWeights(attn_norm=norm(H), wq=raw(kd["wq"], hq, H), wk=raw(kd["wk"], hkv, H), wv=raw(kd["wv"], hkv, H),
                             wo=raw(kd["wo"], H, hq), ffn_norm=norm(H), kinds={n: TAG[k] for n, k in kd.items()})
            ek, n = (kd["experts"], E) if routed else (kd["gate"], 1)
            L.gate, L.up = raw(ek, n * F, H), raw(ek, n * F, H)
            L.down = raw(ek if routed else kd["down"], n * H, F)
            if routed:
                L.router = host(0.02 * rnd(E, H))
            if model == "routed":
                L.q_norm, L.k_norm = 0.3 * norm(hd), 0.3 * norm(hd)
            if oai:
                L.sinks, L.router_bias = host(rnd(case["heads"])), host(0.1 * rnd(E))
                L.bq, L.bk, L.bv, L.bo = (host(0.02 * rnd(n)) for n in (hq, hkv, hkv, H))
                L.gate_b, L.up_b, L.down_b = (host(0.02 * rnd(E, n)) for n in (F, F, H))
            yield L

    # A random head's logits are nearly flat, a trained one's are not: each token has a successor whose head row leans
    # towards the token's embedding, so the greedy continuation has a clear winner at every step.
    kind = "bf16" if oai else "q6_k"
    succ = torch.randperm(V, generator=gen, device="cuda")
    emb = rnd(V, H)
    tok = host(_encode(kind, emb) if V * H < 1 << 26 else torch.cat([_encode(kind, e) for e in emb.split((1 << 26) // H)]))
    head = host(_matrix(gen, kind, V, H, 0.5, near=lambda lo, hi: 0.5 * emb[succ[lo:hi]]))
    del emb
    return Decoder(cfg, layers(), tok, TAG[kind], norm(H), output=head, output_kind=TAG[kind],
                   max_seq=case["prompt"] + case["new"] + 8, prefill_acts=case["acts"])


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    rnd = lambda *n: torch.randn(n, generator=gen, device="cuda")
    op = case["op"]
    s = dict(case=case)
    if op == "host":
        s["w"] = _matrix(gen, case["kind"], case["rows"], case["cols"]).cpu().numpy()
        s["x"] = rnd(case["cols"]).cpu().numpy()
        s["call"] = getattr(gpu, "launch_%s_matvec" % case["kind"])
    elif op in ("matvec", "gemm"):
        kind, rows, cols = case["kind"], case["rows"], case["cols"]
        s["w"] = [device.Weights(_matrix(gen, kind, rows, cols), TAG[kind], rows, cols) for _ in range(case.get("mats", 1))]
        s["x"] = rnd(case["batch"] if op == "matvec" else case["m"], cols)
        if case.get("graph"):
            stack = lambda: [device.gemv(w, s["x"]) for w in s["w"]]
            stack()
            torch.cuda.synchronize()
            s["g"] = torch.cuda.CUDAGraph()
            with torch.cuda.graph(s["g"]):
                s["y"] = stack()
    elif op == "moe":
        E, H, F, kind = case["experts"], case["hidden"], case["ffn"], case["kind"]
        mk = lambda r, c: device.Weights(_matrix(gen, kind, E * r, c), TAG[kind], r, c, n_mats=E)
        s["layer"] = RoutedLayer(0.05 * rnd(E, H), mk(F, H), mk(F, H), mk(H, F), k=case["k"], mode=1, act=1 if case["biased"] else 0,
                                 router_bias=0.1 * rnd(E) if case["biased"] else None)
        s["biases"] = (0.02 * rnd(E, F), 0.02 * rnd(E, F), 0.02 * rnd(E, H)) if case["biased"] else None
        s["x"] = rnd(case["rows"], H)
    else:
        dec = s["dec"] = _decoder(case, gen)
        V, n = case["vocab"], case["seqs"]
        s["prompts"] = list(torch.randint(0, V, (n, case["prompt"]), generator=gen, device="cuda", dtype=torch.int32))
        if op == "generate" and n == 1:
            s["cur"] = dec.prefill(s["prompts"][0]).clone()
            s["out"] = dec.capture_decode(s["cur"])[1]
        elif op == "generate":
            dec.alloc_seqs(n)
            s["cur"] = torch.cat([dec.prefill_seq(i, p) for i, p in enumerate(s["prompts"])])
            s["out"] = dec.capture_decode_seqs(s["cur"])[1]
    return s


def run(s):
    case = s["case"]
    op = case["op"]
    if op == "host":
        return s["call"](s["w"], s["x"], case["rows"], _row_bytes(case["kind"], case["cols"]), case["cols"] // BLOCK[case["kind"]][0])
    if op == "matvec":
        if case["graph"]:
            s["g"].replay()
            return s["y"]
        return [device.gemv(w, s["x"]) for w in s["w"]]
    if op == "gemm":
        return (device.gemm_q8k if case["acts"] == "q8_k" else device.gemm)(s["w"][0], s["x"])
    if op == "moe":
        return device.moe_layer(s["layer"], s["x"], biases=s["biases"])
    dec = s["dec"]
    if op == "prompt":
        dec.reset()
        return dec.forward(s["prompts"][0]), [(L["k"], L["v"]) for L in dec.layers]
    cur, out = s["cur"], s["out"]
    if case["seqs"] == 1:
        dec.reset()
        cur.copy_(dec.prefill(s["prompts"][0]))
        step, caches = dec.replay, [(L["k"], L["v"]) for L in dec.layers]
    else:
        for i, p in enumerate(s["prompts"]):
            cur[i:i + 1].copy_(dec.prefill_seq(i, p))
        step, caches = dec.replay_seqs, [(L["ks"], L["vs"]) for L in dec.layers]
    toks = [cur.clone()]
    for _ in range(case["new"] - 1):
        step()
        cur.copy_(out)
        toks.append(out.clone())
    return torch.stack(toks), caches


# ---- what a pass cannot do without ------------------------------------------------
def _routed_share(case, rows):
    """Experts that `rows` tokens reach, on average, when the router spreads them evenly."""
    return case["experts"] * (1 - (1 - case["k"] / case["experts"]) ** rows)


def work(case):
    op = case["op"]
    if op in ("host", "matvec", "gemm"):
        r, c = case["rows"], case["cols"]
        n, mats = case.get("batch", case.get("m", 1)), case.get("mats", 1)
        return {"bytes": mats * (r * _row_bytes(case["kind"], c) + 4 * n * r) + 4 * n * c, "flops": 2 * mats * n * r * c}
    if op == "moe":
        E, H, F, n = case["experts"], case["hidden"], case["ffn"], case["rows"]
        expert = 2 * F * _row_bytes(case["kind"], H) + H * _row_bytes(case["kind"], F)
        return {"bytes": _routed_share(case, n) * expert + 4 * E * H + 8 * n * H, "flops": 6 * n * case["k"] * H * F + 2 * n * E * H}
    H, F = case["hidden"], case["ffn"]
    hq, hkv, dense = case["heads"] * case["head_dim"], case["kv"] * case["head_dim"], case["model"] == "dense"
    ak = {"dense": "q4_k", "routed": "q8_0", "oai": "bf16"}[case["model"]]
    fk = {"dense": "q4_k", "routed": "q4_k", "oai": "mxfp4"}[case["model"]]
    vk = "bf16" if case["model"] == "oai" else "q6_k"
    attn = (hq + 2 * hkv) * _row_bytes(ak, H) + H * _row_bytes(ak, hq)
    ffn = 2 * F * _row_bytes(fk, H) + H * _row_bytes(fk, F)
    head = case["vocab"] * _row_bytes(vk, H)
    experts = lambda rows: ffn * (1 if dense else _routed_share(case, rows))
    per_token = 2 * case["layers"] * (H * (2 * hq + 2 * hkv) + 3 * H * F * (1 if dense else case["k"]))
    P, N, S = case["prompt"], max(0, case["new"] - 1), case["seqs"]
    ctx = sum(P + i for i in range(N))      # cached rows that the decode steps read
    byte = S * (case["layers"] * (attn + experts(P)) + head) + N * (case["layers"] * (attn + experts(S)) + head) + S * case["layers"] * 8 * hkv * (P + ctx)
    pairs = S * case["layers"] * 4 * hq * (P * P / 2 + ctx)
    return {"bytes": byte, "flops": S * (P + N) * per_token + pairs + S * (1 + N) * 2 * case["vocab"] * H}


def tolerance(case):
    if case["op"] in ("host", "matvec", "gemm"):
        return {"rel": 1e-5}            # exact integers per run of 32, their scaled sum in f32
    if case["op"] == "moe":
        return {"rel": 1e-3}            # an ulp in gate / up moves a value over a rounding step of the down projection's 8-bit input
    return {"rel": 2e-2, "max": 0.9}    # the same in every projection of a stack of layers; the tokens have clear margins and stay
