"""The work that is timed when the speed of this framework is looked at, as a user's program gives it to the framework.

A case is one unit of such work through the public entry points (``Context``, ``TextModel``, ``StackModel``, ``VisionModel``).
Five kinds, each over the whole range of sizes it is used with:

  products    hgemm / hgemm_trans, alone or with the glue that follows them, on resident weights: the rows of a decode step,
              a short prompt, images, and the large square product; both weight layouts
  attention   the three scaled-dot-product entry points on resident tensors: all tokens of an image, a prompt under its mask,
              one new token against its cache
  phi         the Moondream text decoder (24 layers, float16): prompts of token ids or of an image's embedding rows, then greedy
              decoding, one request or up to eight together
  vision      the image encoder and projection (27 layers, float16) on host images, the result staying on the device
  stack       layer-stack decoders (Korupel and Nuvezen designs, bfloat16): prompts, then greedy decoding, one or up to eight

Weights are random.  What a trained model's weights have and the outputs depend on is kept: attention that looks at few
tokens, experts that are chosen by a clear margin, a next token that stands out (the row of the head that belongs to the
token SHIFT places on points at a token's embedding), so that greedy tokens do not hang on rounding.

``exact`` restates every kind in plain torch in 64 bits.
"""
import importlib
import math

import torch

import __graft_entry__

VOCAB = 51200
DECODER = dict(layers=24, width=2048, hidden=8192, heads=32, vocab=VOCAB)
ENCODER = dict(layers=27, width=1152, hidden=4304, heads=16, tokens=729, image=378, patch=14, proj=8192, out=2048)
KORUPEL = dict(layers=12, width=2048, heads=32, kv_heads=8, dim=64, vdim=64, window=1024, keep=4, experts=16, top=2, ff=4768, expert_ff=2368,
               taps=4, vocab=VOCAB)
NUVEZEN = dict(layers=12, width=2048, heads=16, dim=128, rot=64, vdim=128, q_rank=1024, kv_rank=512, window=1024, experts=16, top=2, ff=6144,
               expert_ff=2048, vocab=VOCAB)
SHIFT = 17             # a token's successor: the id this many places on
EPS16 = float(torch.tensor(1e-5).half())
EPS = 1e-5


def listed():
    return [
        # the five products of one decode step, one row: the smallest calls, bound by the weights' bytes and by latency
        {"name": "products_step_1", "kind": "step", "rows": 1, "width": 2048},
        # a prompt of 64 tokens through the first product of an MLP, four layers' weights in turn
        {"name": "products_64", "kind": "product", "rows": 64, "out": 8192, "in": 2048, "layout": "nn", "weights": 4, "glue": False},
        # the large square product
        {"name": "products_8192", "kind": "product", "rows": 8192, "out": 8192, "in": 8192, "layout": "nt", "weights": 1, "glue": False},
        # attention of an image crop, of an image-and-question prompt, and of a token late in an answer
        {"name": "attention_761", "kind": "attention", "tokens": 729, "prompt": 761, "before": 0, "cached": 961},
        # one question about an image: 761 embedding rows, then an answer of 32 tokens
        {"name": "phi_image_1", "kind": "phi", "prompt": 761, "less": 0, "batch": 1, "steps": 32, "image": True},
        # eight text requests of different lengths served together
        {"name": "phi_batch_8", "kind": "phi", "prompt": 761, "less": 61, "batch": 8, "steps": 32, "image": False},
        # one image of one crop, and a large image cut into thirteen
        {"name": "vision_1", "kind": "vision", "crops": 1},
        {"name": "vision_13", "kind": "vision", "crops": 13},
        # a long prompt whose next tokens are asked for
        {"name": "korupel_prompt_2048", "kind": "stack", "design": "korupel", "prompt": 2048, "less": 0, "batch": 1, "steps": 2},
        # eight chats with prompts of a few hundred tokens
        {"name": "korupel_batch_8", "kind": "stack", "design": "korupel", "prompt": 300, "less": 23, "batch": 8, "steps": 32},
        # a long prompt of odd length
        {"name": "nuvezen_prompt_1999", "kind": "stack", "design": "nuvezen", "prompt": 1999, "less": 0, "batch": 1, "steps": 2},
        # a short question, one request, a longer answer
        {"name": "nuvezen_chat_1", "kind": "stack", "design": "nuvezen", "prompt": 61, "less": 0, "batch": 1, "steps": 48},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _less(rng, prompt, batch):
    """By how many tokens each request's prompt is shorter than the one before it."""
    return rng.randint(0, prompt // 12) if batch > 1 else 0


def draw(rng):
    kind = rng.choice(["step", "product", "product", "attention", "phi", "phi", "vision", "stack", "stack", "stack"])
    if kind == "step":
        return {"kind": kind, "rows": rng.randint(1, 8), "width": 64 * rng.randint(8, 40)}
    if kind == "product":
        # the widths of models are multiples of 8; small products come in any size
        layout, glue = rng.choice(["nn", "nt"]), rng.random() < 0.5
        if rng.random() < 0.15:
            return {"kind": kind, "rows": _log(rng, 1, 600), "out": _log(rng, 3, 600), "in": _log(rng, 3, 600), "layout": layout, "weights": 1, "glue": glue}
        rows = _log(rng, 1, 8000)
        return {"kind": kind, "rows": rows, "out": 8 * _log(rng, 16, 1000), "in": 8 * _log(rng, 16, 1000), "layout": layout,
                "weights": rng.choice([1, 2, 4]) if rows <= 512 else 1, "glue": glue}
    if kind == "attention":
        return {"kind": kind, "tokens": _log(rng, 30, 1458), "prompt": _log(rng, 2, 1000), "before": rng.choice([0, rng.randint(1, 1000)]),
                "cached": _log(rng, 1, 2048)}
    if kind == "vision":
        return {"kind": kind, "crops": rng.randint(2, 12)}
    batch = rng.choice([1, 1, rng.randint(2, 8)])
    steps = _log(rng, 2, 32)
    if kind == "phi":
        image = rng.random() < 0.3
        prompt = 729 + _log(rng, 2, 200) if image else _log(rng, 4, 900 if batch == 1 else 4200 // batch)
        batch = 1 if image else batch
        return {"kind": kind, "prompt": prompt, "less": _less(rng, prompt, batch), "batch": batch, "steps": steps, "image": image}
    prompt = _log(rng, 4, 2048 if batch == 1 else 2400 // batch)
    return {"kind": kind, "design": rng.choice(["korupel", "nuvezen"]), "prompt": prompt, "less": _less(rng, prompt, batch), "batch": batch, "steps": steps}


# ---------------------------------------------------------------- weights and inputs

class Random:
    """Seeded values on the GPU."""

    def __init__(self, seed, dtype):
        self.g, self.dtype = torch.Generator(device="cuda").manual_seed(seed), dtype

    def normal(self, *shape, std=0.02):
        return (torch.randn(*shape, device="cuda", generator=self.g) * std).to(self.dtype)

    def linear(self, *shape, gain=1.0):
        return self.normal(*shape, std=gain / math.sqrt(shape[-1]))

    def vector(self, n, mean=1.0, std=0.1):
        """A vector of float32 that the model's type holds."""
        return (torch.randn(n, device="cuda", generator=self.g) * std + mean).to(self.dtype).float()

    def ids(self, n, vocab):
        return torch.randint(0, vocab, (n,), device="cuda", generator=self.g).cpu().numpy()


def _head(r, embed):
    """A head under which a token's successor stands out."""
    noise = r.normal(*embed.shape)
    return (noise.float() + 0.04 * torch.roll(embed, SHIFT, 0).float()).to(r.dtype)


def _phi_weights(r):
    L, D, F, V = (DECODER[k] for k in ("layers", "width", "hidden", "vocab"))
    w = {k: [] for k in ("ln_w", "ln_b", "wqkv", "bqkv", "wout", "bout", "wfc1", "bfc1", "wfc2", "bfc2")}
    deep = 0.02 / math.sqrt(2 * L)
    for _ in range(L):
        w["ln_w"].append(r.normal(D, std=0.1) + 1), w["ln_b"].append(r.normal(D))
        w["wqkv"].append(torch.cat([r.normal(2 * D, D, std=0.04), r.normal(D, D)])), w["bqkv"].append(r.normal(3 * D))
        w["wout"].append(r.normal(D, D, std=deep)), w["bout"].append(r.normal(D))
        w["wfc1"].append(r.normal(F, D)), w["bfc1"].append(r.normal(F))
        w["wfc2"].append(r.normal(D, F, std=deep)), w["bfc2"].append(r.normal(D))
    w["wte"] = r.normal(V, D, std=1.0)
    w["ln_out_w"], w["ln_out_b"], w["lm_w"], w["lm_b"] = r.normal(D, std=0.1) + 1, r.normal(D), _head(r, w["wte"]), r.normal(V)
    return w


def _vision_weights(r):
    z = ENCODER
    D, F, T = z["width"], z["hidden"], z["tokens"]
    names = ("ln1_w", "ln1_b", "wqkv", "bqkv", "wout", "bout", "ln2_w", "ln2_b", "wfc1", "bfc1", "wfc2", "bfc2")
    w = {k: [] for k in names}
    for _ in range(z["layers"]):
        for n in ("ln1", "ln2"):
            w[n + "_w"].append(r.normal(D, std=0.1) + 1), w[n + "_b"].append(r.normal(D))
        w["wqkv"].append(torch.cat([r.normal(D, 2 * D, std=0.05), r.normal(D, D)], 1).contiguous()), w["bqkv"].append(r.normal(3 * D))
        w["wout"].append(r.normal(D, D)), w["bout"].append(r.normal(D))
        w["wfc1"].append(r.normal(D, F)), w["bfc1"].append(r.normal(F))
        w["wfc2"].append(r.normal(F, D)), w["bfc2"].append(r.normal(D))
    w.update(patch_w=r.normal(3 * z["patch"] ** 2, D), patch_b=r.normal(D), pos_emb=r.normal(T, D, std=0.2), norm_w=r.normal(D, std=0.1) + 1, norm_b=r.normal(D),
             proj_fc1_w=r.normal(2 * D, z["proj"]), proj_fc1_b=r.normal(z["proj"]), proj_fc2_w=r.normal(z["proj"], z["out"]), proj_fc2_b=r.normal(z["out"]))
    return w


def _token_table(r, z):
    """Embeddings; the first channels rank the experts per token, in clear steps, and no sublayer writes to them."""
    embed = torch.randn(z["vocab"], z["width"], device="cuda", generator=r.g)
    E = z["experts"]
    rank = torch.argsort(torch.randn(z["vocab"], E, device="cuda", generator=r.g), 1)
    embed[:, :E] = 1.5 - 3.0 * rank / (E - 1)
    return embed.to(r.dtype)


def _apart(v, n):
    v[..., :n] = 0
    return v


def _router(r, E, W):
    w = r.linear(E, W, gain=0.015)
    w[:, :E] = 2.0 * torch.eye(E, device="cuda")
    return w


def _korupel_layers(r, models):
    z = KORUPEL
    W, H, G, d, e, E = z["width"], z["heads"], z["kv_heads"], z["dim"], z["vdim"], z["experts"]
    out = []
    for i in range(z["layers"]):
        s = {"norm1": r.vector(W), "norm2": r.vector(W), "norm1b": _apart(r.vector(W), E), "norm2b": _apart(r.vector(W), E), "heads": H, "dim": d, "vdim": e,
             "w_out": r.linear(W, H * e)}
        for n in ("conv1", "conv2"):
            s[n] = (torch.randn(W, z["taps"], device="cuda", generator=r.g) * 0.3).to(r.dtype).float()
            s[n][:E] = 0
        s["norm2"][:E] = 1
        if i % 3 == 2:
            rows = (H + G) * d + H
            s.update(mixer=models.MIXER_WINDOW_ATTENTION, kv_heads=G, scale=d ** -0.5, window=z["window"], keep_first=z["keep"],
                     r1=r.vector(H, 0.4), r2=r.vector(H, 0.4), b_in=torch.cat([r.vector((H + G) * d, 0.0, 0.3), torch.zeros(H, device="cuda")]),
                     w_in=r.linear(rows, W, gain=1.5))
        else:
            s.update(mixer=models.MIXER_LIGHTNING, decay=torch.linspace(0.6, 0.999, H, device="cuda"), mix_norm=r.vector(H * e),
                     w_in=r.linear(2 * H * (d + e), W))
        if i % 2 == 0:
            F = z["ff"]
            s.update(ff=models.FF_DENSE, act=models.ACT_GELU_TANH, ff_dim=F, w_gate_up=r.linear(2 * F, W), w_down=r.linear(W, F))
        else:
            F = z["expert_ff"]
            s.update(ff=models.FF_MOE, act=models.ACT_SILU, ff_dim=F, experts=E, top=z["top"], router=_router(r, E, W), w_gate_up=r.linear(E, 2 * F, W),
                     w_down=r.linear(E, W, F))
        out.append(s)
    return out


def _nuvezen_layers(r, models):
    z = NUVEZEN
    W, H, d, rot, e, Q, R, E = (z[k] for k in ("width", "heads", "dim", "rot", "vdim", "q_rank", "kv_rank", "experts"))
    out = []
    for i in range(z["layers"]):
        uk, uv = r.linear(H, d, R, gain=1.5), r.linear(H * e, R, gain=1.5)
        s = {"form": models.LAYER_PARALLEL, "mixer": models.MIXER_LATENT_ATTENTION, "norm1": r.vector(W), "norm2": r.vector(W),
             "ls1": _apart(r.vector(W, 0.5), E), "ls2": _apart(r.vector(W, 0.5), E), "heads": H, "dim": d, "vdim": e, "rot_dim": rot, "q_rank": Q,
             "kv_rank": R, "scale": (d + rot) ** -0.5, "window": z["window"], "rope_base": 10000.0, "w_in": r.linear(Q + R + rot, W),
             "w_out": r.linear(W, H * e), "w_uq": r.linear(H * (d + rot), Q, gain=1.5), "w_ukv": torch.cat([uk.reshape(H * d, R), uv]),
             "w_ukt": uk.transpose(1, 2).contiguous(), "q_norm": r.vector(Q), "kv_norm": r.vector(R), "sink": r.vector(H, 0.5, 1.0)}
        s["norm2"][:E] = 1
        if i % 2 == 0:
            F = z["ff"]
            s.update(ff=models.FF_DENSE, act=models.ACT_SILU, ff_dim=F, w_gate_up=r.linear(2 * F, W), w_down=r.linear(W, F))
        else:
            F = z["expert_ff"]
            s.update(ff=models.FF_MOE, act=models.ACT_CLAMPED, act_limit=2.0, act_alpha=1.702, ff_dim=F, experts=E, top=z["top"],
                     router_kind=models.ROUTER_SOFTMAX, router=torch.cat([_router(r, E, W), r.linear(1, W)]), w_gate_up=r.linear(E, 2 * F, W),
                     w_down=r.linear(E, W, F), shared_ff=F, shared_limit=1.0, shared_gate_up=r.linear(2 * F, W), shared_down=r.linear(W, F))
        out.append(s)
    return out


def _stack_weights(case, r, models):
    z = KORUPEL if case["design"] == "korupel" else NUVEZEN
    layers = _korupel_layers(r, models) if case["design"] == "korupel" else _nuvezen_layers(r, models)
    embed = _token_table(r, z)
    return {"layers": layers, "embed": embed, "head": _head(r, embed), "final_norm": r.vector(z["width"])}


def _lengths(case):
    return [case["prompt"] - i * case["less"] for i in range(case["batch"])]


def _prompts(case, r, vocab):
    return [r.ids(n, vocab) for n in _lengths(case)]


def _image_rows(case, r, wte):
    """An image's rows between the first and the other tokens of a question."""
    ids = torch.randint(0, wte.shape[0], (case["prompt"] - 729,), device="cuda", generator=r.g)
    return torch.cat([wte[ids[:1]], r.normal(729, wte.shape[1], std=1.0), wte[ids[1:]]]).contiguous()


def _step_shapes(case):
    """K, N of a decode step's products."""
    w = case["width"]
    return [(w, 3 * w), (w, w), (w, 4 * w), (4 * w, w), (w, VOCAB)]


def _step_inputs(case, r):
    shapes = _step_shapes(case)
    return [r.normal(case["rows"], k, std=1.0) for k, _ in shapes], [r.normal(n, k) for k, n in shapes]


def _product_inputs(case, r):
    M, N, K = case["rows"], case["out"], case["in"]
    x = r.normal(M, K, std=1.0)
    w = [r.normal(*((N, K) if case["layout"] == "nt" else (K, N))) for _ in range(case["weights"])]
    glue = {"bias": r.normal(N), "residual": r.normal(M, N, std=1.0)} if case["glue"] else {}
    return x, w, glue


def _attention_inputs(case, r):
    T, S, L, n = case["tokens"], case["prompt"], case["before"] + case["prompt"], case["cached"]
    def qkv(heads, q, kv, d):   # scores of a few units: some tokens matter more than others
        return r.normal(heads, q, d, std=1.6), r.normal(heads, kv, d, std=1.6), r.normal(heads, kv, d, std=1.0)
    return qkv(16, T, T, 72), qkv(32, S, L, 64), qkv(32, 1, n, 64)


# ---------------------------------------------------------------- the framework's side

_context = None


def _library():
    """The package, its models module and the process's one context."""
    global _context
    pkg = __graft_entry__.load_package()
    if _context is None:
        _context = pkg.Context(0)
    return pkg, importlib.import_module(__graft_entry__.PKG_NAME + ".models"), _context


class Served:
    """A model with its requests; both go with the last reference."""

    def __init__(self, model, batch):
        self.model, self.requests = model, [model.request() for _ in range(batch)]

    def __del__(self):
        for q in self.requests:
            q.close()
        self.model.close()


class Encoder:
    def __init__(self, model):
        self.model = model

    def __del__(self):
        self.model.close()


def prepare(case, seed):
    _, models, ctx = _library()
    kind = case["kind"]
    r = Random(seed, torch.bfloat16 if kind == "stack" else torch.float16)
    state = {"case": case, "ctx": ctx}
    if kind == "step":
        state["x"], state["w"] = _step_inputs(case, r)
        state["y"] = [torch.empty(case["rows"], n, device="cuda", dtype=torch.float16) for _, n in _step_shapes(case)]
    elif kind == "product":
        state["x"], state["w"], state["glue"] = _product_inputs(case, r)
        state["y"] = [torch.empty(case["rows"], case["out"], device="cuda", dtype=torch.float16) for _ in state["w"]]
    elif kind == "attention":
        state["qkv"] = _attention_inputs(case, r)
        S, L, n = case["prompt"], case["before"] + case["prompt"], case["cached"]
        state["mask"], state["all"] = torch.empty(S, L, device="cuda", dtype=torch.uint8), torch.ones(n, device="cuda", dtype=torch.uint8)
        state["y"] = [torch.empty_like(q) for q, _, _ in state["qkv"]]
    elif kind == "vision":
        w = _vision_weights(r)
        g = torch.Generator().manual_seed(seed)
        state["images"] = torch.randint(0, 256, (case["crops"], ENCODER["image"], ENCODER["image"], 3), dtype=torch.uint8, generator=g).numpy()
        state["out"] = torch.empty(ENCODER["tokens"], ENCODER["out"], device="cuda", dtype=torch.float16)
        torch.cuda.synchronize()
        state["encoder"] = Encoder(models.VisionModel(ctx, w, n_heads=ENCODER["heads"], max_crops=case["crops"]))
    elif kind == "phi":
        w = _phi_weights(r)
        if case["image"]:
            state["embeds"] = _image_rows(case, r, w["wte"])
        else:
            state["prompts"] = _prompts(case, r, DECODER["vocab"])
        torch.cuda.synchronize()
        state["served"] = Served(models.TextModel(ctx, w, n_heads=DECODER["heads"], max_seq=1024), case["batch"])
    else:
        z = KORUPEL if case["design"] == "korupel" else NUVEZEN
        w = _stack_weights(case, r, models)
        state["prompts"] = _prompts(case, r, z["vocab"])
        torch.cuda.synchronize()
        model = models.StackModel(ctx, w["layers"], embed=w["embed"], head=w["head"], final_norm=w["final_norm"], eps=EPS,
                                  residual_mult=0.5 if case["design"] == "korupel" else 1.0, taps=z.get("taps", 1), max_seq=2560)
        state["served"] = Served(model, case["batch"])
    torch.cuda.synchronize()     # the context works on a stream of its own
    return state


def run(state):
    case, ctx = state["case"], state["ctx"]
    kind = case["kind"]
    if kind == "step":
        for (k, n), x, w, y in zip(_step_shapes(case), state["x"], state["w"], state["y"]):
            ctx.hgemm_nt(x.data_ptr(), w.data_ptr(), case["rows"], n, k, out=y.data_ptr())
        return state["y"]
    if kind == "product":
        M, N, K, x, glue = case["rows"], case["out"], case["in"], state["x"].data_ptr(), state["glue"]
        for w, y in zip(state["w"], state["y"]):
            if glue:
                ctx.hgemm_fused(x, w.data_ptr(), y.data_ptr(), M, N, K, int(case["layout"] == "nt"), bias=glue["bias"].data_ptr(), gelu=True,
                                residual=glue["residual"].data_ptr())
            else:
                (ctx.hgemm_nt if case["layout"] == "nt" else ctx.hgemm_nn)(x, w.data_ptr(), M, N, K, out=y.data_ptr())
        return state["y"]
    if kind == "attention":
        (a, b, c), y, L = state["qkv"], state["y"], case["before"] + case["prompt"]
        ctx.sdpa_maskless(*(t.data_ptr() for t in a), 16, case["tokens"], case["tokens"], 72, out=y[0].data_ptr())
        ctx.create_attention_mask(case["before"], case["prompt"], out=state["mask"].data_ptr())
        ctx.sdpa_masked(*(t.data_ptr() for t in b), state["mask"].data_ptr(), 32, case["prompt"], L, 64, out=y[1].data_ptr())
        ctx.sdpa_single(*(t.data_ptr() for t in c), state["all"].data_ptr(), case["cached"], out=y[2].data_ptr())
        return y
    if kind == "vision":
        state["encoder"].model.encode(state["images"], out_ptr=state["out"].data_ptr())
        return state["out"]
    model, reqs = state["served"].model, state["served"].requests
    logits, firsts = [], []
    for i, q in enumerate(reqs):
        q.reset()
        if "embeds" in state:
            e = state["embeds"]
            _, row, token = model.forward(q, e.data_ptr(), want_hidden=False, rows=e.shape[0])
        else:
            p = state["prompts"][i]
            row, token = model.step(q, p, want=[len(p) - 1], want_token=True)
        logits.append(row.reshape(-1))
        firsts.append(token)
    if len(reqs) == 1:
        tokens, rows = model.generate(reqs[0], firsts[0], case["steps"], want_logits=True)
        return {"prompt": logits, "answer": rows, "tokens": tokens}
    return {"prompt": logits, "tokens": model.generate_batch(reqs, firsts, case["steps"])}


# ---------------------------------------------------------------- what a pass cannot do without

def _attention_pairs(n, window):
    """Visible pairs of a prompt of n tokens."""
    w = min(n, window)
    return w * (w + 1) // 2 + (n - w) * w


def work(case):
    kind = case["kind"]
    if kind == "step":
        M = case["rows"]
        return {"bytes": sum(2 * (M * k + k * n + M * n) for k, n in _step_shapes(case)), "flops": sum(2 * M * k * n for k, n in _step_shapes(case))}
    if kind == "product":
        M, N, K, c = case["rows"], case["out"], case["in"], case["weights"]
        return {"bytes": 2 * (M * K + c * K * N + c * M * N + (N + M * N if case["glue"] else 0)), "flops": 2 * c * M * N * K}
    if kind == "attention":
        T, S, L, n = case["tokens"], case["prompt"], case["before"] + case["prompt"], case["cached"]
        pairs = S * case["before"] + S * (S + 1) // 2
        return {"bytes": 2 * (16 * 72 * 4 * T + 32 * 64 * (2 * S + 2 * L) + 32 * 64 * (2 + 2 * n)) + 2 * S * L, "flops": 4 * (16 * 72 * T * T + 32 * 64 * (pairs + n))}
    if kind == "vision":
        z, c = ENCODER, case["crops"]
        D, F, T, P = z["width"], z["hidden"], z["tokens"], 3 * z["patch"] ** 2
        layer, ends = 4 * D * D + 2 * D * F, 2 * D * z["proj"] + z["proj"] * z["out"]
        return {"bytes": 2 * (z["layers"] * layer + P * D + ends + T * D + T * z["out"]) + c * 3 * z["image"] ** 2,
                "flops": 2 * (c * T * (z["layers"] * layer + P * D) + T * ends) + 4 * c * z["layers"] * T * T * D}
    lens, steps, B = _lengths(case), case["steps"], case["batch"]
    if kind == "phi":
        z = DECODER
        D, L = z["width"], z["layers"]
        weights, head = L * (4 * D * D + 2 * D * z["hidden"]), z["vocab"] * D
        cached = sum(sum(n + i + 1 for i in range(steps)) for n in lens)
        flops = 2 * (sum(lens) + B * steps) * weights + 2 * B * (1 + steps) * head + 4 * D * L * (sum(n * (n + 1) // 2 for n in lens) + cached)
        return {"bytes": 2 * (1 + steps) * (weights + head) + 4 * D * L * (2 * sum(lens) + cached), "flops": flops}
    korupel = case["design"] == "korupel"
    z = KORUPEL if korupel else NUVEZEN
    W, E, L = z["width"], z["experts"], z["layers"]
    if korupel:
        attn, light = W * ((z["heads"] + z["kv_heads"]) * z["dim"] + z["heads"] + z["heads"] * z["dim"]), W * 5 * z["heads"] * z["dim"]
        n_attn = L // 3
        mixers, entry, pair = n_attn * attn + (L - n_attn) * light, z["kv_heads"] * z["dim"], 4 * z["heads"] * z["dim"]
        shared = 0
    else:
        H, d, rot, e, Q, R = (z[k] for k in ("heads", "dim", "rot", "vdim", "q_rank", "kv_rank"))
        n_attn = L
        mixers, entry, pair = L * (W * (Q + R + rot) + Q * H * (d + rot) + R * H * (d + e) + W * H * e), R + rot, 2 * H * (d + rot + e)
        shared = z["expert_ff"]
    expert, half = 3 * W * z["expert_ff"], L // 2
    fixed = mixers + half * 3 * W * z["ff"] + half * 3 * W * shared
    used = lambda tokens: E * (1 - (1 - z["top"] / E) ** tokens)  # noqa: E731  experts that some token takes
    head = z["vocab"] * W
    cached = sum(sum(min(n + i + 1, z["window"]) for i in range(steps)) for n in lens)
    size = 2 * (fixed + half * used(sum(lens)) * expert + head) + 2 * steps * (fixed + half * used(B) * expert + head) + 2 * n_attn * entry * (sum(lens) + cached)
    state = 0 if not korupel else 8 * (L - n_attn) * z["heads"] * z["dim"] * z["vdim"] * B * steps
    active = fixed + half * z["top"] * expert
    pairs = sum(_attention_pairs(n, z["window"]) for n in lens)
    return {"bytes": size + state, "flops": 2 * active * (sum(lens) + B * steps) + 2 * head * B * (1 + steps) + n_attn * pair * (pairs + cached)}


def tolerance(case):
    # float16 results of one product or one attention (2e-4 from 64 bits): a last place here and there; with the glue, one of
    # each rounding
    if case["kind"] in ("step", "product", "attention"):
        return {"rel": 1e-3, "max": 1e-2}
    # many layers of 16-bit activations, whose roundings differ as soon as one sum does: 1.3e-3 (phi), 2.5e-3 (vision) and up to
    # 1.2e-2 (bfloat16) from 64 bits
    if case["kind"] == "phi":
        return {"rel": 6e-3, "max": 0.1}
    if case["kind"] == "vision":
        return {"rel": 1e-2, "max": 0.2}
    return {"rel": 3e-2, "max": 0.5}


# ---------------------------------------------------------------- 64-bit restatement

def _f(t):
    return t.double()


def _gelu(x):
    h = lambda v: float(torch.tensor(v).half())  # noqa: E731  the two constants are float16 values by definition
    return 0.5 * x * (1 + torch.tanh(h(math.sqrt(h(2 / h(math.pi)))) * (x + h(0.044715) * x ** 3)))


def _norm(x, w, b):
    x = x - x.mean(-1, keepdim=True)
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS16) * _f(w) + _f(b)


def _rms(x, w, eps=EPS):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * _f(w)


def _heads(q, k, v, scale, bias=None, sink=None):
    """Attention of [H, n, d] tensors, head by head; bias [n, m] or a function of the head."""
    out = []
    for h in range(q.shape[0]):
        s = _f(q[h]) @ _f(k[h]).T * scale
        if bias is not None:
            s = s + (bias(h) if callable(bias) else bias)
        if sink is not None:
            s = torch.cat([s, _f(sink[h]).expand(s.shape[0], 1)], 1)
        p = torch.softmax(s, -1)
        out.append(p[:, :k.shape[1]] @ _f(v[h]))
    return torch.stack(out)


def _causal(n, m, window=0, keep=0):
    """0 where token i (the last n of m) sees token j, else -inf; and the distances."""
    dist = torch.arange(m - n, m, device="cuda")[:, None] - torch.arange(m, device="cuda")[None, :]
    seen = dist >= 0
    if window:
        seen &= (dist < window) | (torch.arange(m, device="cuda")[None, :] < keep)
    return torch.where(seen, 0.0, -math.inf).double(), dist.clamp(min=0).double()


def _split(x, heads):
    return x.reshape(x.shape[0], heads, -1).transpose(0, 1)


def _join(x):
    return x.transpose(0, 1).reshape(x.shape[1], -1)


def _phi_exact(w, x, rows):
    """Logits of the wanted rows of a sequence of embedding rows."""
    H, D, n = DECODER["heads"], DECODER["width"], x.shape[0]
    d, rot = D // H, D // H // 2
    angle = torch.arange(n, device="cuda").double()[:, None] * 10000.0 ** (-torch.arange(0, rot, 2, device="cuda").double() / rot)
    c, s = torch.cos(angle), torch.sin(angle)
    mask, _ = _causal(n, n)

    def turn(t):
        a, b = t[..., :rot // 2], t[..., rot // 2:rot]
        return torch.cat([a * c - b * s, a * s + b * c, t[..., rot:]], -1)
    for i in range(DECODER["layers"]):
        h = _norm(x, w["ln_w"][i], w["ln_b"][i])
        q, k, v = (h @ _f(w["wqkv"][i]).T + _f(w["bqkv"][i])).split(D, 1)
        o = _join(_heads(turn(_split(q, H)), turn(_split(k, H)), _split(v, H), d ** -0.5, mask))
        m = _gelu(h @ _f(w["wfc1"][i]).T + _f(w["bfc1"][i]))
        x = x + o @ _f(w["wout"][i]).T + _f(w["bout"][i]) + m @ _f(w["wfc2"][i]).T + _f(w["bfc2"][i])
    return _norm(x[rows], w["ln_out_w"], w["ln_out_b"]) @ _f(w["lm_w"]).T + _f(w["lm_b"])


def _vision_exact(w, images):
    z = ENCODER
    D, H, T, p = z["width"], z["heads"], z["tokens"], z["patch"]
    n, side = images.shape[0], z["image"] // p
    x = torch.from_numpy(images).cuda().double().reshape(n, side, p, side, p, 3).permute(0, 1, 3, 5, 2, 4).reshape(n * T, -1)
    x = ((x / 255 - 0.5) / 0.5) @ _f(w["patch_w"]) + _f(w["patch_b"]) + _f(w["pos_emb"]).repeat(n, 1)
    for i in range(z["layers"]):
        qkv = (_norm(x, w["ln1_w"][i], w["ln1_b"][i]) @ _f(w["wqkv"][i]) + _f(w["bqkv"][i])).reshape(n, T, 3 * D)
        o = torch.cat([_join(_heads(*(_split(t, H) for t in crop.split(D, 1)), (D // H) ** -0.5)) for crop in qkv])
        x = x + o @ _f(w["wout"][i]) + _f(w["bout"][i])
        h = _gelu(_norm(x, w["ln2_w"][i], w["ln2_b"][i]) @ _f(w["wfc1"][i]) + _f(w["bfc1"][i]))
        x = x + h @ _f(w["wfc2"][i]) + _f(w["bfc2"][i])
    x = _norm(x, w["norm_w"], w["norm_b"]).reshape(n, T, D)
    h = _gelu(torch.cat([x[0], x[min(1, n - 1)]], 1) @ _f(w["proj_fc1_w"]) + _f(w["proj_fc1_b"]))
    return h @ _f(w["proj_fc2_w"]) + _f(w["proj_fc2_b"])


def _conv(u, w):
    taps, y = w.shape[1], torch.zeros_like(u)
    for j in range(taps):
        back = taps - 1 - j
        if back < u.shape[0]:
            y[back:] += _f(w[:, j]) * u[:u.shape[0] - back]
    return u + y


def _gated(h, gate_up, down, act):
    a = (h @ _f(gate_up).T).reshape(h.shape[0], -1, 2, 32)
    return act(a[:, :, 0].reshape(h.shape[0], -1), a[:, :, 1].reshape(h.shape[0], -1)) @ _f(down).T


def _clamped(limit):
    def act(g, u):
        g, u = g.clamp(max=limit), u.clamp(-limit, limit)
        return g * torch.sigmoid(1.702 * g) * (u + 1)
    return act


def _feed_forward(s, h, korupel, models):
    silu, tanh = (lambda g, u: g * torch.sigmoid(g) * u), (lambda g, u: torch.nn.functional.gelu(g, approximate="tanh") * u)
    if s["ff"] == models.FF_DENSE:
        return _gated(h, s["w_gate_up"], s["w_down"], tanh if korupel else silu)
    z = h @ _f(s["router"]).T
    best, sel = z[:, :s["experts"]].topk(s["top"], -1)
    share = torch.sigmoid(best) if korupel else torch.softmax(best, -1)
    y = torch.zeros_like(h)
    for e in range(s["experts"]):
        at, slot = torch.nonzero(sel == e, as_tuple=True)
        if at.numel():
            y[at] += share[at, slot][:, None] * _gated(h[at], s["w_gate_up"][e], s["w_down"][e], silu if korupel else _clamped(s["act_limit"]))
    if s.get("shared_ff"):
        y += torch.sigmoid(z[:, s["experts"]:]) * _gated(h, s["shared_gate_up"], s["shared_down"], _clamped(s["shared_limit"]))
    return y


def _korupel_mixer(s, h, models):
    H, n = s["heads"], h.shape[0]
    y = h @ _f(s["w_in"]).T
    if s["mixer"] == models.MIXER_WINDOW_ATTENTION:
        y = y + _f(s["b_in"])
        q, k, g = y.split([H * s["dim"], s["kv_heads"] * s["dim"], H], 1)
        k = _split(k, s["kv_heads"]).repeat_interleave(H // s["kv_heads"], 0)
        mask, dist = _causal(n, n, s["window"], s["keep_first"])
        o = _heads(_split(q, H), k, k, s["scale"], lambda i: mask - _f(s["r1"][i]) * torch.log1p(_f(s["r2"][i]) * dist))
        o = o * torch.sigmoid(g).T[:, :, None]
        return _join(o) @ _f(s["w_out"]).T
    q, k, v, g = y.split([H * s["dim"], H * s["dim"], H * s["vdim"], H * s["vdim"]], 1)
    q, k, v = (_split(t * torch.sigmoid(t), H) for t in (q, k, v))
    mask, dist = _causal(n, n)
    o = torch.stack([(q[i] @ k[i].T * torch.exp(dist * torch.log(_f(s["decay"][i])) + mask)) @ v[i] for i in range(H)])
    return (_rms(_join(o), s["mix_norm"]) * torch.sigmoid(g)) @ _f(s["w_out"]).T


def _nuvezen_mixer(s, h):
    H, d, rot, R, Q, n = s["heads"], s["dim"], s["rot_dim"], s["kv_rank"], s["q_rank"], h.shape[0]
    angle = torch.arange(n, device="cuda").double()[:, None] * s["rope_base"] ** (-torch.arange(0, rot, 2, device="cuda").double() / rot)

    def turn(t):
        a, b, c, sn = t[..., 0::2], t[..., 1::2], torch.cos(angle), torch.sin(angle)
        return torch.stack([a * c - b * sn, b * c + a * sn], -1).flatten(-2)
    cq, c, kr = (h @ _f(s["w_in"]).T).split([Q, R, rot], 1)
    cq, c = _rms(cq, s["q_norm"]), _rms(c, s["kv_norm"])
    q = _split(cq @ _f(s["w_uq"]).T, H)
    kv = c @ _f(s["w_ukv"]).T
    k, v = _split(kv[:, :H * d], H), _split(kv[:, H * d:], H)
    q = torch.cat([q[..., :d], turn(q[..., d:])], -1)
    k = torch.cat([k, turn(kr).expand(H, n, rot)], -1)
    return _join(_heads(q, k, v, s["scale"], _causal(n, n, s["window"])[0], s["sink"])) @ _f(s["w_out"]).T


def _stack_exact(w, case, tokens, rows, models):
    korupel = case["design"] == "korupel"
    x = _f(w["embed"][tokens])
    for s in w["layers"]:
        if korupel:
            x = x + 0.5 * _rms(_korupel_mixer(s, _conv(_rms(x, s["norm1"]), s["conv1"]), models), s["norm1b"])
            x = x + 0.5 * _rms(_feed_forward(s, _conv(_rms(x, s["norm2"]), s["conv2"]), True, models), s["norm2b"])
        else:
            x = x + _f(s["ls1"]) * _nuvezen_mixer(s, _rms(x, s["norm1"])) + _f(s["ls2"]) * _feed_forward(s, _rms(x, s["norm2"]), False, models)
    return _rms(x[rows], w["final_norm"]) @ _f(w["head"]).T


def _answer(case, prompts, logits_of):
    """Logits after each prompt and, for a single request, of its greedy answer: the successors, as the logits have to confirm."""
    out = []
    for prompt in prompts:
        n = prompt.shape[0]
        alone = case["batch"] == 1
        got = logits_of(prompt, case["steps"] if alone else 0, list(range(n - 1, n + (case["steps"] if alone else 0))))
        out.append(got)
    if case["batch"] > 1:
        return {"prompt": [g[0] for g in out], "tokens": None}
    g = out[0]
    best = g.argmax(-1)
    follows = bool(((best[1:] - best[:-1]) % g.shape[1] == SHIFT).all())
    return {"prompt": [g[0]], "answer": g[1:] if follows else None, "tokens": None}


def exact(case, seed):
    _, models, _ = _library()
    kind = case["kind"]
    r = Random(seed, torch.bfloat16 if kind == "stack" else torch.float16)
    if kind == "step":
        return [_f(a) @ _f(w).T for a, w in zip(*_step_inputs(case, r))]
    if kind == "product":
        x, ws, glue = _product_inputs(case, r)
        out = []
        for w in ws:
            y = _f(x) @ (_f(w).T if case["layout"] == "nt" else _f(w))
            out.append(_gelu(y + _f(glue["bias"])) + _f(glue["residual"]) if glue else y)
        return out
    if kind == "attention":
        a, b, c = _attention_inputs(case, r)
        mask, _ = _causal(case["prompt"], case["before"] + case["prompt"])
        return [_heads(*a, 72 ** -0.5), _heads(*b, 0.125, mask), _heads(*c, 0.125)]
    if kind == "vision":
        w = _vision_weights(r)
        g = torch.Generator().manual_seed(seed)
        return _vision_exact(w, torch.randint(0, 256, (case["crops"], ENCODER["image"], ENCODER["image"], 3), dtype=torch.uint8, generator=g).numpy())
    if kind == "phi":
        w = _phi_weights(r)
        if case["image"]:
            prompts = [_image_rows(case, r, w["wte"])]
        else:
            prompts = [w["wte"][torch.from_numpy(p).cuda()] for p in _prompts(case, r, DECODER["vocab"])]

        def logits(rows, steps, want):
            # the answer's first token from the prompt alone, the others are its successors
            x = _f(rows)
            if steps:
                first = int(_phi_exact(w, x, [x.shape[0] - 1]).argmax())
                x = torch.cat([x, _f(w["wte"][(first + SHIFT * torch.arange(steps, device="cuda")) % DECODER["vocab"]])])
            return _phi_exact(w, x, want)
        return _answer(case, prompts, logits)
    w = _stack_weights(case, r, models)
    vocab = w["embed"].shape[0]
    prompts = [torch.from_numpy(p).cuda() for p in _prompts(case, r, vocab)]

    def logits(ids, steps, want):
        if steps:
            first = int(ids[-1] + SHIFT)
            ids = torch.cat([ids, (first + SHIFT * torch.arange(steps, device="cuda")) % vocab])
        return _stack_exact(w, case, ids, want, models)
    return _answer(case, prompts, logits)
