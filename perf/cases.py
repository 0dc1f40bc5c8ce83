"""The calls whose speed matters to a user of this engine, each through a public entry point of `llmq_b200`.

A worker spends its time in decode steps (one token for every running sequence) and prompt steps (portions of up to a step's
token budget).  Both are made of a few operations: projections, gated feed-forwards, attention over the paged cache for single
tokens and for portions, the head with the sampler, and, in the routed designs, the experts.  A case is one of these at sizes of
the built-in models, or a whole forward step.  All tensors are made on the GPU from the seed; activations and cached rows are
unit normal, matrices are scaled to keep them so, contexts are spread evenly over a range (ragged), pages are scattered."""
import ctypes as C
import dataclasses
import math

import torch

from llmq_b200 import lib as L
from llmq_b200.model import BUILTIN_SPECS, NativeModel, interleave_gate_up

PAGE = 16
BF = torch.bfloat16
MODELS = ("llama-3-8b", "llama-3.2-1b", "gemma-2-9b", "gemma-2-2b")


def listed():
    return [
        # one user, one token: the query / key / value product of the small model, the smallest call there is
        {"name": "qkv 1b 1 row", "kind": "linear", "model": "llama-3.2-1b", "part": "qkv", "rows": 1},
        # the common serving batch of about a hundred sequences: the product with the longest reduction
        {"name": "down 8b 100 rows", "kind": "linear", "model": "llama-3-8b", "part": "down", "rows": 100},
        # steady state of the offline batch job (4608 sequences in flight): the feed-forward of a decode step
        {"name": "mlp 8b 4608 rows", "kind": "mlp", "model": "llama-3-8b", "rows": 4608},
        # the number of sequences that the reference's production scripts set, on the translation model
        {"name": "mlp gemma 9b 750 rows", "kind": "mlp", "model": "gemma-2-9b", "rows": 750},
        # the same steady state, 128 tokens in and 128 out: contexts between 129 and 256
        {"name": "decode 8b 4608 seqs", "kind": "decode", "model": "llama-3-8b", "seqs": 4608, "lo": 129, "hi": 256},
        # a handful of users with long documents on the small model
        {"name": "decode 1b 6 long seqs", "kind": "decode", "model": "llama-3.2-1b", "seqs": 6, "lo": 3000, "hi": 8100},
        # mixed lengths on the model with the large heads, soft cap and sliding window
        {"name": "decode gemma 9b 100 seqs", "kind": "decode", "model": "gemma-2-9b", "seqs": 100, "lo": 33, "hi": 2560},
        # prompts of the offline batch job: a full step of 36 prompts of 128 tokens
        {"name": "prompts 8b 36 x 128", "kind": "portion", "model": "llama-3-8b", "prompts": 36, "lo": 128, "hi": 128, "past": 0},
        # long and ragged prompts on the model with the large heads, soft cap and sliding window
        {"name": "prompts gemma 9b 3 long", "kind": "portion", "model": "gemma-2-9b", "prompts": 3, "lo": 333, "hi": 2048, "past": 0},
        # the end of a decode step: last norm, rows, vocabulary product, sampling at the default temperature
        {"name": "head 8b 128 rows", "kind": "head", "model": "llama-3-8b", "rows": 128, "temperature": 0.7},
        # a whole decode step at the small model's widths, replayed from a graph as the engine does (four layers: behind more of them two
        # correct orders of the same sums are further apart than a comparison could allow)
        {"name": "step 1b 48 seqs", "kind": "step", "model": "llama-3.2-1b", "layers": 4, "seqs": 48, "lo": 100, "hi": 900, "prompts": 0,
         "prompt": 0},
        # the routed feed-forward of a decode step
        {"name": "experts 128 rows", "kind": "experts", "width": 2048, "ff": 1024, "experts": 16, "top": 4, "groups": 4, "keep": 2,
         "rows": 128},
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(("linear", "linear", "mlp", "mlp", "decode", "decode", "portion", "portion", "head", "step", "experts"))
    model = rng.choice(MODELS)
    spec = BUILTIN_SPECS[model]
    if kind == "linear":
        return {"kind": kind, "model": model, "part": rng.choice(("qkv", "o", "down")), "rows": _log(rng, 1, 4608)}
    if kind == "mlp":
        return {"kind": kind, "model": model, "rows": _log(rng, 1, 4608)}
    if kind == "decode":
        hi = _log(rng, 64, 8000)
        most = int(2.0e9 / (4.0 * spec.n_kv_heads * spec.head_dim * hi))   # 2 GB of cached rows
        return {"kind": kind, "model": model, "seqs": _log(rng, 1, max(2, min(4608, most))), "lo": rng.randint(1, hi), "hi": hi}
    if kind == "portion":
        hi = _log(rng, 8, 6000)
        return {"kind": kind, "model": model, "prompts": _log(rng, 1, max(1, 8192 // hi)), "lo": rng.randint(max(1, hi // 4), hi), "hi": hi,
                "past": rng.choice((0, 0, 0, rng.randint(1, 1500)))}
    if kind == "head":
        return {"kind": kind, "model": model, "rows": _log(rng, 1, 1024), "temperature": rng.choice((0.0, 0.7))}
    if kind == "step":
        model, layers = rng.choice((("llama-3.2-1b", 4), ("llama-3-8b", 4)))
        prompts = rng.choice((0, 0, rng.randint(1, 8)))
        lo = rng.randint(16, 600)
        return {"kind": kind, "model": model, "layers": layers, "seqs": _log(rng, 1, 256), "lo": lo, "hi": lo + rng.randint(0, 900),
                "prompts": prompts, "prompt": rng.randint(5, 256) if prompts else 0}
    width = rng.choice((2048, 3072))
    experts, top = rng.choice(((16, 4), (32, 6)))
    return {"kind": kind, "width": width, "ff": width // 2, "experts": experts, "top": top, "groups": 4, "keep": 2,
            "rows": _log(rng, 1, 4096)}


# ---- inputs ----------------------------------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _normal(g, *shape, scale=1.0, dtype=BF):
    return (torch.randn(*shape, generator=g, device="cuda", dtype=torch.float32) * scale).to(dtype)


def _spread(case, n, lo, hi):
    """n lengths spread evenly over [lo, hi]"""
    return [hi if n == 1 else lo + (hi - lo) * i // (n - 1) for i in range(n)]


def _lengths(case, seed):
    n = case["seqs"] if case["kind"] in ("decode", "step") else case["prompts"]
    lens = _spread(case, n, case["lo"], case["hi"])
    order = torch.randperm(n, generator=torch.Generator().manual_seed(int(seed))).tolist()
    return [lens[i] for i in order]


def _pages(g, needs, extra=3):
    """a block table over a scattered pool for sequences that need so many pages each: (table int32 [n, stride], pool size)"""
    total = sum(needs) + extra
    stride = (max(needs) + 7) // 8 * 8
    perm = torch.randperm(total, generator=g, device="cuda").to(torch.int32).tolist()
    table, at = [], 0
    for k in needs:
        table.append(perm[at:at + k] + [0] * (stride - k))
        at += k
    return torch.tensor(table, dtype=torch.int32, device="cuda"), total


def _cache(g, blocks, n_kv, D, layers=None):
    shape = (blocks, 2, n_kv, PAGE, D)
    if layers is None:
        return torch.randn(*shape, generator=g, device="cuda", dtype=BF)
    return torch.randn(layers, *shape, generator=g, device="cuda", dtype=BF)


def _window(spec):
    return spec.sliding_window if spec.arch == "gemma2" else 0


def _linear_shape(case):
    s = BUILTIN_SPECS[case["model"]]
    q = s.n_q_heads * s.head_dim
    return {"qkv": (s.qkv_dim, s.hidden), "o": (s.hidden, q), "down": (s.hidden, s.intermediate)}[case["part"]]


def _portion_tiles(lens, past):
    tiles, row = [], 0
    for i, n in enumerate(lens):
        tiles += [[i, row + j, min(16, n - j), past + j] for j in range(0, n, 16)]
        row += n
    return tiles, row


def _step_spec(case):
    return dataclasses.replace(BUILTIN_SPECS[case["model"]], n_layers=case["layers"])


def _step_weights(spec, g):
    """matrices scaled by the width they reduce over: activations keep the size they have in a trained model"""
    H, I, q = spec.hidden, spec.intermediate, spec.n_q_heads * spec.head_dim
    norm = lambda: (1.0 + 0.1 * torch.randn(1, H, generator=g, device="cuda")).to(BF)
    w = {"embed": _normal(g, spec.vocab, H, scale=H ** -0.5), "final_norm": norm()}
    if not spec.tie_embeddings:
        w["lm_head"] = _normal(g, spec.vocab, H, scale=H ** -0.5)
    for i in range(spec.n_layers):
        p = f"layers.{i}."
        w[p + "input_norm"], w[p + "post_norm"] = norm(), norm()
        w[p + "qkv"], w[p + "o"] = _normal(g, spec.qkv_dim, H, scale=H ** -0.5), _normal(g, H, q, scale=0.3 * q ** -0.5)
        w[p + "gate"], w[p + "up"] = _normal(g, I, H, scale=H ** -0.5), _normal(g, I, H, scale=H ** -0.5)
        w[p + "down"] = _normal(g, H, I, scale=0.3 * I ** -0.5)
    return w


def _step_inputs(case, seed):
    spec, g = _step_spec(case), _gen(seed)
    weights = _step_weights(spec, g)
    B, P, n = case["seqs"], case["prompts"], case["prompt"]
    ctx = _lengths(case, seed)
    needs = [(c + PAGE - 1) // PAGE for c in ctx] + [(n + PAGE - 1) // PAGE] * P
    table, blocks = _pages(g, needs)
    T = B + P * n
    tab = table.tolist()
    pos = [c - 1 for c in ctx] + [j for _ in range(P) for j in range(n)]
    seq = list(range(B)) + [B + i for i in range(P) for _ in range(n)]
    slots = [tab[s][p // PAGE] * PAGE + p % PAGE for s, p in zip(seq, pos)]
    tiles = [[B + i, B + i * n + j, min(16, n - j), j] for i in range(P) for j in range(0, n, 16)]
    rows = list(range(B)) + [B + (i + 1) * n - 1 for i in range(P)]
    ints = lambda v: torch.tensor(v, dtype=torch.int32, device="cuda")
    meta = {"tok": torch.randint(0, spec.vocab, (T,), generator=g, device="cuda", dtype=torch.int32), "pos": ints(pos), "slot": ints(slots),
            "bt": table, "ctx": ints(ctx), "tiles": ints(tiles or [[0, 0, 0, 0]]), "rows": ints(rows)}
    kv = _cache(g, blocks, spec.n_kv_heads, spec.head_dim, spec.n_layers)
    return spec, weights, meta, kv, ctx, len(tiles)


def prepare(case, seed):
    k, g = case["kind"], _gen(seed)
    st = {"case": case}
    if k == "linear":
        N, K = _linear_shape(case)
        st["a"], st["w"] = _normal(g, case["rows"], K), _normal(g, N, K, scale=K ** -0.5)
        st["c"] = torch.empty(case["rows"], N, dtype=BF, device="cuda")
    elif k == "mlp":
        s = BUILTIN_SPECS[case["model"]]
        H, I, M = s.hidden, s.intermediate, case["rows"]
        st["a"] = _normal(g, M, H)
        st["gate_up"] = interleave_gate_up(_normal(g, I, H, scale=H ** -0.5), _normal(g, I, H, scale=H ** -0.5)).contiguous()
        st["down"] = _normal(g, H, I, scale=I ** -0.5)
        st["act"], st["out"] = torch.empty(M, I, dtype=BF, device="cuda"), torch.empty(M, H, dtype=BF, device="cuda")
        st["gated"] = L.gemm_geglu_bf16 if s.arch == "gemma2" else L.gemm_swiglu_bf16
    elif k in ("decode", "portion"):
        s = BUILTIN_SPECS[case["model"]]
        past = case.get("past", 0)
        lens = _lengths(case, seed)
        st["bt"], blocks = _pages(g, [(past + n + PAGE - 1) // PAGE for n in lens])
        st["kv"] = _cache(g, blocks, s.n_kv_heads, s.head_dim)
        st["lens"], T = lens, len(lens)
        if k == "portion":
            tiles, T = _portion_tiles(lens, past)
            st["tiles"] = torch.tensor(tiles, dtype=torch.int32, device="cuda")
        else:
            st["ctx"] = torch.tensor(lens, dtype=torch.int32, device="cuda")
        st["qkv"] = _normal(g, T, s.qkv_dim)
        st["out"] = torch.empty(T, s.n_q_heads * s.head_dim, dtype=BF, device="cuda")
        st["args"] = (s.n_q_heads, s.n_kv_heads, s.head_dim, PAGE, s.attn_scale)
        st["options"] = {"softcap": s.attn_softcap, "window": _window(s)}
    elif k == "head":
        s = BUILTIN_SPECS[case["model"]]
        M = case["rows"]
        st["x"], st["norm"] = _normal(g, M, s.hidden), (1.0 + 0.1 * torch.randn(s.hidden, generator=g, device="cuda")).to(BF)
        st["w"] = _normal(g, s.vocab, s.hidden, scale=s.hidden ** -0.5)
        st["rows"] = torch.arange(M, dtype=torch.int32, device="cuda")
        st["y"], st["sel"] = torch.empty_like(st["x"]), torch.empty_like(st["x"])
        st["logits"], st["ids"] = torch.empty(M, s.vocab, dtype=BF, device="cuda"), torch.empty(M, dtype=torch.int32, device="cuda")
        st["eps"], st["cap"] = s.rms_eps, s.final_softcap
        params = torch.zeros(M, 4, dtype=torch.int32)
        params[:, 0] = torch.tensor([case["temperature"]], dtype=torch.float32).view(torch.int32)
        params[:, 1], params[:, 3] = torch.arange(M) + int(seed) % 100003, torch.arange(M) + 128
        st["params"] = params.cuda()
    elif k == "step":
        spec, weights, meta, kv, ctx, n_tiles = _step_inputs(case, seed)

        def engine_layout():
            for name, t in weights.items():
                if name.endswith(".gate"):
                    yield name[:-4] + "gate_up", interleave_gate_up(t, weights[name[:-4] + "up"])
                elif not name.endswith(".up"):
                    yield name, t
        T, B, P = meta["tok"].numel(), case["seqs"], case["prompts"]
        model = NativeModel(spec, engine_layout(), max_tokens=T, max_seqs=B + P, max_model_len=2048, num_blocks=kv.shape[1])
        model.kv.copy_(kv)
        ids = torch.empty(B + P, dtype=torch.int32, device="cuda")
        p = {n: t.data_ptr() for n, t in meta.items()}
        batch = L.Batch(T=T, n_dec=B, n_tiles=n_tiles, n_sample=B + P, bt_stride=meta["bt"].shape[1], token_ids=p["tok"], positions=p["pos"],
                        slot_mapping=p["slot"], block_table=p["bt"], ctx_lens=p["ctx"], tiles=p["tiles"], sample_rows=p["rows"],
                        out_ids=ids.data_ptr())
        st.update(model=model, batch=batch, meta=meta, ids=ids, logits=model.logits_view(B + P), graph=None)
        if not P:  # steps of single tokens are replayed from a graph
            _forward(st)
            torch.cuda.synchronize()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                _forward(st)
            st["graph"] = graph
    else:
        T, W, F, E, top = case["rows"], case["width"], case["ff"], case["experts"], case["top"]
        P = T * top
        st["h"], st["x0"] = _normal(g, T, W), _normal(g, T, W, dtype=torch.float32)
        st["scores"], st["corr"] = _normal(g, T, E, dtype=torch.float32), _normal(g, E, scale=0.2, dtype=torch.float32)
        st["up"], st["down"] = _normal(g, E * 2 * F, W, scale=W ** -0.5), _normal(g, E * W, F, scale=F ** -0.5)
        ints = lambda n: torch.empty(n, dtype=torch.int32, device="cuda")
        bf = lambda *s: torch.empty(*s, dtype=BF, device="cuda")
        st.update(idx=ints(P), wts=torch.empty(P, device="cuda"), off=ints(E + 1), perm=ints(P), pair=ints(P), tab=ints((P // 128 + E) * 4),
                  nt=ints(1), src=bf(P, W), gu=bf(P, 2 * F), act=bf(P, F), eo=bf(P, W), x=torch.empty(T, W, device="cuda"))
    return st


# ---- passes ----------------------------------------------------------------------------------------------------------
def _forward(st):
    L.check(st["model"].lib.b200q_model_forward(st["model"].handle, C.byref(st["batch"]), torch.cuda.current_stream().cuda_stream))


def run(st):
    case = st["case"]
    k = case["kind"]
    if k == "linear":
        L.gemm_bf16(st["a"], st["w"], st["c"])
        return st["c"]
    if k == "mlp":
        st["gated"](st["a"], st["gate_up"], st["act"])
        L.gemm_bf16(st["act"], st["down"], st["out"])
        return {"act": st["act"], "out": st["out"]}
    if k == "decode":
        L.decode_attn(st["qkv"], st["out"], st["kv"], st["bt"], st["ctx"], *st["args"], **st["options"])
        return st["out"]
    if k == "portion":
        L.prefill_attn(st["qkv"], st["out"], st["kv"], st["bt"], st["tiles"], *st["args"], **st["options"])
        return st["out"]
    if k == "head":
        L.rmsnorm(st["x"], st["norm"], st["y"], st["eps"])
        L.gather_rows(st["y"], st["rows"], st["sel"])
        L.gemm_bf16(st["sel"], st["w"], st["logits"])
        if st["cap"]:
            L.softcap_bf16(st["logits"], st["cap"])
        L.sample_bf16(st["logits"], st["params"], st["ids"])
        return {"logits": st["logits"], "ids": st["ids"]}
    if k == "step":
        if st["graph"] is not None:
            st["graph"].replay()
        else:
            _forward(st)
        return {"logits": st["logits"]}   # (the greedy ids are the places of the largest of these)
    T, W, F, E, top = case["rows"], case["width"], case["ff"], case["experts"], case["top"]
    P, lib, s = T * top, L.load(), torch.cuda.current_stream().cuda_stream
    p = {n: t.data_ptr() for n, t in st.items() if isinstance(t, torch.Tensor)}
    L.check(lib.b200q_copy_f32(p["x0"], p["x"], T * W, s))
    L.check(lib.b200q_moe_route_gated(p["scores"], E, p["corr"], T, E, top, case["groups"], case["keep"], 0, p["idx"], p["wts"], p["off"],
                                      p["perm"], p["pair"], p["tab"], p["nt"], s))
    L.check(lib.b200q_gather_rows(p["h"], p["perm"], p["src"], P, W, s))
    L.check(lib.b200q_linear_grouped(p["src"], W, None, p["up"], 2 * F * W, p["gu"], 2 * F, p["off"], E, P, 2 * F, W, L.DTYPE_BF16, p["tab"],
                                     p["nt"], s))
    L.check(lib.b200q_silu_glu(p["gu"], p["act"], P, F, L.DTYPE_BF16, s))
    L.check(lib.b200q_linear_grouped(p["act"], F, None, p["down"], W * F, p["eo"], W, p["off"], E, P, W, F, L.DTYPE_BF16, p["tab"], p["nt"],
                                     s))
    L.check(lib.b200q_residual_add_routed(p["x"], p["eo"], p["pair"], p["idx"], p["wts"], top, E, p["h"], T, W, L.DTYPE_BF16, s))
    return st["x"]


# ---- what a pass cannot do without -----------------------------------------------------------------------------------
def _pairs(spec, n, past):
    """(query, key) pairs of a portion of n tokens behind `past` cached ones, under the window"""
    w = _window(spec)
    return sum(min(p + 1, w) if w else p + 1 for p in range(past, past + n))


def work(case):
    k = case["kind"]
    if k == "linear":
        N, K = _linear_shape(case)
        M = case["rows"]
        return {"bytes": 2 * (M * K + N * K + M * N), "flops": 2 * M * N * K}
    if k == "experts":
        T, W, F, E, top = case["rows"], case["width"], case["ff"], case["experts"], case["top"]
        used = min(E, T * top)
        return {"bytes": 2 * (used * 3 * W * F + T * W) + 8 * T * W + 4 * T * E, "flops": 6 * T * top * W * F}
    s = _step_spec(case) if k == "step" else BUILTIN_SPECS[case["model"]]
    H, I, q, kvrow = s.hidden, s.intermediate, s.n_q_heads * s.head_dim, 4 * s.n_kv_heads * s.head_dim
    if k == "mlp":
        M = case["rows"]
        return {"bytes": 2 * (3 * H * I + 2 * M * H + M * I), "flops": 6 * M * H * I}
    if k == "decode":
        lens = _spread(case, case["seqs"], case["lo"], case["hi"])
        seen = sum(min(c, _window(s)) if _window(s) else c for c in lens)
        return {"bytes": seen * kvrow + 4 * len(lens) * q, "flops": 4 * seen * q}
    if k == "portion":
        lens = _spread(case, case["prompts"], case["lo"], case["hi"])
        return {"bytes": sum(case["past"] + n for n in lens) * kvrow + 4 * sum(lens) * q,
                "flops": 4 * q * sum(_pairs(s, n, case["past"]) for n in lens)}
    if k == "head":
        M = case["rows"]
        return {"bytes": 2 * (s.vocab * H + M * H + M * s.vocab), "flops": 2 * M * H * s.vocab}
    T, rows = case["seqs"] + case["prompts"] * case["prompt"], case["seqs"] + case["prompts"]
    ctx = _spread(case, case["seqs"], case["lo"], case["hi"])
    pairs = sum(ctx) + case["prompts"] * _pairs(s, case["prompt"], 0)
    layer = s.qkv_dim * H + H * q + 3 * H * I
    return {"bytes": 2 * (s.n_layers * layer + s.vocab * H + rows * s.vocab) + s.n_layers * kvrow * (sum(ctx) + T),
            "flops": 2 * (T * s.n_layers * layer + rows * s.vocab * H) + 4 * s.n_layers * q * pairs}


def tolerance(case):
    """about four times what another order of the same sums (other splits of the reduction, the other decode kernel) was seen to change,
    for a whole step twice that: 1.5e-2 is as far as two roundings of four layers of bf16 activations get apart"""
    k = case["kind"]
    if k == "step":
        return {"rel": 0.03, "max": 0.4}
    if k == "head":      # a logit that rounds the other way may change which of two near equals is drawn
        return {"rel": 0.002, "max": 0.05, "differ": 0.01}
    if k in ("decode", "portion"):   # probabilities are rounded to bf16 against whatever maximum was known: 2.6e-3
        return {"rel": 0.01, "max": 0.1}
    if k == "linear":    # 2.5e-4
        return {"rel": 0.002, "max": 0.05}
    return {"rel": 0.004, "max": 0.05}


# ---- the same in 64 bits, in plain torch ------------------------------------------------------------------------------
def _unswizzle(pages):
    """[..., PAGE, D] as the cache stores it (16-byte piece c of row t at c ^ (t & 7)) -> logical rows"""
    D = pages.shape[-1]
    t, d = torch.arange(PAGE, device="cuda")[:, None], torch.arange(D, device="cuda")[None]
    return torch.gather(pages, -1, (((d // 8) ^ (t & 7)) * 8 + d % 8).expand(pages.shape))


def _keys_values(kv, table_row, n):
    """the first n cached rows of a sequence: fp64 [n, n_kv, D] twice"""
    pages = _unswizzle(kv[table_row[: (n + PAGE - 1) // PAGE].long()]).double()   # [pages, 2, n_kv, PAGE, D]
    rows = pages.permute(1, 0, 3, 2, 4).flatten(1, 2)[:, :n]
    return rows[0], rows[1]


def _attend(q, k, v, pos, scale, cap, window):
    """q [T, n_q, D] at absolute positions pos over k, v [n, n_kv, D]: [T, n_q * D]"""
    T, n_q, D = q.shape
    G = n_q // k.shape[1]
    out = torch.empty_like(q)
    j = torch.arange(k.shape[0], device="cuda")
    for h in range(n_q):
        for a in range(0, T, 2048):
            p = pos[a:a + 2048, None]
            s = (q[a:a + 2048, h] @ k[:, h // G].t()) * scale
            s = cap * torch.tanh(s / cap) if cap else s
            hide = j[None] > p
            hide = hide | (j[None] <= p - window) if window else hide
            out[a:a + 2048, h] = torch.softmax(s.masked_fill(hide, -math.inf), -1) @ v[:, h // G]
    return out.reshape(T, n_q * D)


def _attend_one(q, kv, table, ctx, spec):
    """one query per sequence; sequences in groups of like length: q [B, n_q, D] -> [B, n_q * D]"""
    B, n_q, D = q.shape
    G, w = n_q // spec.n_kv_heads, _window(spec)
    out = torch.empty(B, n_q * D, dtype=torch.float64, device="cuda")
    order = sorted(range(B), key=lambda i: ctx[i])
    step = max(1, int(2e8 // (max(ctx) * spec.n_kv_heads * D * 2)))
    for a in range(0, B, step):
        at = order[a:a + step]
        n = max(ctx[i] for i in at)
        np_ = (n + PAGE - 1) // PAGE
        rows = _unswizzle(kv[table[at][:, :np_].long()]).double()            # [b, pages, 2, n_kv, PAGE, D]
        rows = rows.permute(2, 0, 3, 1, 4, 5).flatten(3, 4)                  # [2, b, n_kv, n, D]
        s = torch.einsum("bhgd,bhnd->bhgn", q[at].view(len(at), spec.n_kv_heads, G, D), rows[0]) * spec.attn_scale
        if spec.attn_softcap:
            s = spec.attn_softcap * torch.tanh(s / spec.attn_softcap)
        c = torch.tensor([ctx[i] for i in at], device="cuda")[:, None, None, None]
        j = torch.arange(rows.shape[3], device="cuda")
        hide = (j >= c) | (j < c - w) if w else j >= c
        p = torch.softmax(s.masked_fill(hide, -math.inf), -1)
        out[at] = torch.einsum("bhgn,bhnd->bhgd", p, rows[1].masked_fill((j >= c[:, :, 0, :])[..., None], 0.0)).reshape(len(at), -1)
    return out


def _rms(x, w, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _mm(a, w):
    """a [M, K] . w [N, K]^T in 64 bits, a slab of w at a time"""
    return torch.cat([a @ part.double().t() for part in w.split(16384)], 1)


def _rotation(spec, pos):
    inv = 1.0 / spec.rope_theta ** (torch.arange(0, spec.head_dim, 2, device="cuda", dtype=torch.float64) / spec.head_dim)
    r = spec.rope_scaling
    if r:
        wave, orig = 2 * math.pi / inv, r["original_max_position_embeddings"]
        smooth = ((orig / wave - r["low_freq_factor"]) / (r["high_freq_factor"] - r["low_freq_factor"])).clamp(0.0, 1.0)
        inv = (1 - smooth) * inv / r["factor"] + smooth * inv
    a = pos.double()[:, None] * inv[None]
    return a.cos()[:, None], a.sin()[:, None]


def _turn(x, cos, sin):
    a, b = x.chunk(2, -1)
    return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)


def _exact_step(case, seed):
    spec, w, meta, kv, ctx, _ = _step_inputs(case, seed)
    B, P, n, D = case["seqs"], case["prompts"], case["prompt"], spec.head_dim
    x = w["embed"][meta["tok"].long()].double()
    cos, sin = _rotation(spec, meta["pos"])
    T, nq, nk = x.shape[0], spec.n_q_heads, spec.n_kv_heads
    slot, t = meta["slot"].long(), (meta["slot"].long() % PAGE)[:, None]
    d = torch.arange(D, device="cuda")[None]
    place = ((d // 8) ^ (t & 7)) * 8 + d % 8
    for i in range(spec.n_layers):
        p = f"layers.{i}."
        qkv = _mm(_rms(x, w[p + "input_norm"].double(), spec.rms_eps), w[p + "qkv"]).view(T, -1, D)
        q, k, v = _turn(qkv[:, :nq], cos, sin), _turn(qkv[:, nq:nq + nk], cos, sin), qkv[:, nq + nk:]
        layer = kv[i].double()
        for which, rows in ((0, k), (1, v)):
            for h in range(nk):
                layer[slot[:, None] // PAGE, which, h, t, place] = rows[:, h]
        o = torch.empty(T, nq * D, dtype=torch.float64, device="cuda")
        o[:B] = _attend_one(q[:B], layer, meta["bt"][:B], ctx, spec)
        for s in range(P):
            rows = slice(B + s * n, B + (s + 1) * n)
            o[rows] = _attend(q[rows], k[rows], v[rows], torch.arange(n, device="cuda"), spec.attn_scale, 0.0, 0)
        x = x + _mm(o, w[p + "o"])
        y = _rms(x, w[p + "post_norm"].double(), spec.rms_eps)
        x = x + _mm(torch.nn.functional.silu(_mm(y, w[p + "gate"])) * _mm(y, w[p + "up"]), w[p + "down"])
    x = _rms(x, w["final_norm"].double(), spec.rms_eps)[meta["rows"].long()]
    return {"logits": _mm(x, w["embed"] if spec.tie_embeddings else w["lm_head"])}


def exact(case, seed):
    k = case["kind"]
    if k == "step":
        return _exact_step(case, seed)
    st = prepare(case, seed)
    if k == "linear":
        return _mm(st["a"].double(), st["w"])
    if k == "mlp":
        a, I = st["a"].double(), st["act"].shape[1]
        gu = st["gate_up"].view(I // 128, 2, 128, -1)
        gate, up = _mm(a, gu[:, 0].reshape(I, -1)), _mm(a, gu[:, 1].reshape(I, -1))
        act = torch.nn.functional.gelu(gate, approximate="tanh") if st["gated"] is L.gemm_geglu_bf16 else torch.nn.functional.silu(gate)
        act = act * up
        return {"act": act, "out": _mm(act, st["down"])}
    if k in ("decode", "portion"):
        s = BUILTIN_SPECS[case["model"]]
        q = st["qkv"][:, : s.n_q_heads * s.head_dim].double().view(-1, s.n_q_heads, s.head_dim)
        if k == "decode":
            return _attend_one(q, st["kv"], st["bt"], st["lens"], s)
        out, row, past = [], 0, case["past"]
        for i, n in enumerate(st["lens"]):
            keys, values = _keys_values(st["kv"], st["bt"][i], past + n)
            out.append(_attend(q[row:row + n], keys, values, torch.arange(past, past + n, device="cuda"), s.attn_scale, s.attn_softcap,
                               _window(s)))
            row += n
        return torch.cat(out)
    if k == "head":
        logits = _mm(_rms(st["x"].double(), st["norm"].double(), st["eps"]), st["w"])
        return {"logits": st["cap"] * torch.tanh(logits / st["cap"]) if st["cap"] else logits, "ids": None}
    T, F, E, top = case["rows"], case["ff"], case["experts"], case["top"]
    s = torch.sigmoid(st["scores"].double())
    choice = s + st["corr"].double()
    best = choice.view(T, case["groups"], -1).topk(2, -1).values.sum(-1).topk(case["keep"], -1).indices
    kept = torch.zeros(T, case["groups"], dtype=torch.bool, device="cuda").scatter_(1, best, True)
    idx = choice.masked_fill(~kept.repeat_interleave(E // case["groups"], 1), -math.inf).topk(top, -1).indices
    x, h = st["x0"].double(), st["h"].double()
    for e in range(E):
        t = (idx == e).any(1).nonzero()[:, 0]
        if len(t):
            gu = h[t] @ st["up"].view(E, 2 * F, -1)[e].double().t()
            y = (torch.nn.functional.silu(gu[:, :F]) * gu[:, F:]) @ st["down"].view(E, -1, F)[e].double().t()
            x[t] += s[t, e][:, None] * y
    return x
