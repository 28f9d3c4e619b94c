"""Timed cases of the decode backend: what a program that uses it has it do, through its public entry points.

Two levels are used in earnest.  A host that keeps its own model loop calls the op interface (`Eng`) op by op; everybody
else loads a `GemmaCudaModel` and either asks it for text (`generate_timed`), scores or continues given ids (`prefill`,
`forward`, `decode_token`), or puts the slot `Scheduler` on top.  Shapes are those of the repository's own
configurations (`e2b_config`, `e4b_config`, `tiny_config`) and of its kernel benchmarks; weights are random blocks in
the GGUF layouts.

A case is a dict of plain values; `kind` says what one pass does:

  matvec     one packed matrix times 1..256 rows (`matvec_wd` / `matvec_batch`)
  head       the end of a decode step: tied Q6_K lm_head and the greedy softcap arg-max
  attention  decode attention of several slots over their Q4_0 caches (`sdpa_decode`)
  layer      one decoder layer of a single token, op by op
  generate   rewind a slot, run a prompt, generate greedily (`generate_timed`)
  score      rewind a slot, run a prompt, feed a given continuation step by step, logits of every step
  first      rewind a slot, run a prompt, the first greedy token (`prefill` + `decode_token`)
  serve      requests with ragged prompts through the slot scheduler until all are done
"""
import numpy as np
import torch

from ksearch_b200 import model as ksm
from ksearch_b200.eng import Buffer, CudaContext, Eng, F16, F32, Q4K, Q6K, Q40
from ksearch_b200.scheduler import InferenceRequest, Scheduler, SchedulerConfig

HEAD_DIM = 256
SHAPES = {"e2b": ksm.e2b_config, "e4b": ksm.e4b_config, "tiny": ksm.tiny_config}
SIGMA = 1e-4                # fp16 super-block scale of one matrix or layer: weights of about 0.02 around zero
MIN_OVER_D = 7.5            # dmin over d there, the middle of the nibble range
# Whole models take the benchmark's random-init distribution (d and dmin alike, scale from the configuration): through
# dozens of layers with 4-bit caches it stays comparable, where weights around zero turn a last-bit difference into
# a percent of the logits.  f16 activations need it scaled down, or the FFN leaves the f16 range.
SIGMA_MODEL_F16 = 2e-6
WINDOW_EVERY = 6            # five sliding-window layers, then a full-attention one


def listed():
    return [
        # a hidden-sized batch of ragged length: what a short prompt or a scored sentence makes of one projection
        dict(name="gemm_q4k_55_rows", kind="matvec", dtype="q4k", rows=4096, cols=1536, n_tok=55),
        # a full prompt chunk through the stacked gate|up matrix of the larger model
        dict(name="gemm_q4k_256_rows", kind="matvec", dtype="q4k", rows=20480, cols=2560, n_tok=256),
        # every decoded token ends here
        dict(name="lm_head_q6k_argmax", kind="head", rows=262144, cols=1536),
        # four slots deep into their contexts, unequal lengths
        dict(name="attention_4_slots", kind="attention", act="f32", n_q=8, n_kv=2, lens="1024,4096,16384,16384"),
        # a host that keeps its own loop, f16 activations: one layer of one token
        dict(name="layer_ops_f16", kind="layer", act="f16", hidden=1536, ffn=6144, n_q=8, n_kv=1, tlen=700),
        # a short chat turn on the small model
        dict(name="generate_e2b", kind="generate", shape="e2b", act="f32", window=0, prompt=64, new=64),
        # the same far into a long context on the larger model
        dict(name="generate_e4b_long", kind="generate", shape="e4b", act="f32", window=0, prompt=4001, new=32),
        # a model whose layers are mostly sliding-window ones, prompt longer than the window
        dict(name="generate_e2b_window", kind="generate", shape="e2b", act="f32", window=512, prompt=777, new=24),
        # f16 activations: a prompt and a given continuation, as scoring or constrained decoding does it
        dict(name="score_e2b_f16", kind="score", shape="e2b", act="f16", window=0, prompt=121, new=16),
        # a long prompt until its first token
        dict(name="first_token_e2b_2048", kind="first", shape="e2b", act="f32", window=0, prompt=2048),
        # all slots of a server busy, greedy, ragged prompts
        dict(name="serve_e4b_8_slots", kind="serve", shape="e4b", slots=8, requests=8, prompt_lo=60, prompt_hi=300, new=20,
             temperature=0.0),
        # a few sampled chats
        dict(name="serve_e2b_4_sampled", kind="serve", shape="e2b", slots=4, requests=4, prompt_lo=15, prompt_hi=90, new=16,
             temperature=0.8),
    ]


def _log(rng, lo, hi):
    """A whole number between lo and hi, even over its logarithm."""
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    kind = rng.choice(["matvec", "matvec", "head", "attention", "layer", "generate", "generate", "score", "first", "serve", "serve"])
    if kind == "matvec":
        return dict(kind=kind, dtype=rng.choice(["q4k", "q4k", "q6k"]), rows=_log(rng, 256, 20480),
                    cols=256 * rng.choice([2, 4, 6, 8, 10, 16, 24, 40]), n_tok=rng.choice([1, _log(rng, 2, 256), _log(rng, 9, 256)]))
    if kind == "head":
        return dict(kind=kind, rows=_log(rng, 32768, 262144) // 4 * 4, cols=rng.choice([1536, 2560]))
    if kind == "attention":
        n = rng.choice([1, 2, 4, 8])
        lens = [_log(rng, 20, 16384 if n <= 4 else 8192) for _ in range(n)]
        return dict(kind=kind, act=rng.choice(["f32", "f32", "f16"]), n_q=8, n_kv=rng.choice([1, 2, 4]), lens=",".join(map(str, lens)))
    if kind == "layer":
        hidden, ffn, n_kv = rng.choice([(1536, 6144, 1), (2560, 10240, 2)])
        return dict(kind=kind, act=rng.choice(["f32", "f16"]), hidden=hidden, ffn=ffn, n_q=8, n_kv=n_kv, tlen=_log(rng, 10, 4096))
    if kind == "serve":
        lo = _log(rng, 5, 100)
        slots = rng.choice([2, 3, 4, 6, 8])
        return dict(kind=kind, shape=rng.choice(["tiny", "e2b", "e2b", "e4b"]), slots=slots, requests=slots + rng.choice([0, 0, 1, 2]),
                    prompt_lo=lo, prompt_hi=lo + _log(rng, 3, 200), new=rng.randint(4, 20), temperature=rng.choice([0.0, 0.0, 0.7, 1.0]))
    shape = rng.choice(["tiny", "e2b", "e2b", "e4b"])
    window = rng.choice([0, 0, 512]) if shape == "e2b" else 0
    if kind == "first":
        return dict(kind=kind, shape=shape, act="f32", window=window, prompt=_log(rng, 8, 2048))
    if kind == "score":
        return dict(kind=kind, shape="e2b" if shape == "e4b" else shape, act=rng.choice(["f32", "f16"]), window=0,
                    prompt=_log(rng, 8, 160), new=rng.randint(4, 16))
    return dict(kind=kind, shape=shape, act="f32", window=window, prompt=_log(rng, 8, 2048), new=rng.randint(8, 48))


# ---- what a program has in hand -------------------------------------------------------------------

_ctx = None


def _context():
    """One context per GPU and process, as the library wants it."""
    global _ctx
    if _ctx is None:
        torch.cuda.init()
        _ctx = CudaContext(0, flags=1)
    return _ctx


class _Device:
    """Device memory of the library for torch to look at; keeps the model that owns it alive."""

    def __init__(self, owner, ptr, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": typestr, "data": (ptr, False), "version": 2}


def _wrap(ctx, t):
    """A torch tensor as the library's buffer handle."""
    nbytes = t.numel() * t.element_size()
    return Buffer(ctx, ctx.lib.ks_buf_wrap(ctx.h, t.data_ptr(), nbytes), nbytes)


class _State:
    def __init__(self, **kw):
        self.__dict__.update(kw)


class _Model(ksm.GemmaCudaModel):
    """Closed with its last reference."""

    def __del__(self):
        if getattr(self, "h", None):
            self.close()


_FIELDS = {Q4K: (144, [0, 2]), Q6K: (210, [208]), Q40: (18, [0])}


def _blocks_gpu(gen, dtype, n_blocks, sigma):
    """n_blocks packed blocks on the GPU: payload bytes uniform, fp16 scales d = |N(0, sigma)|, Q6_K sub-scales in +-64."""
    size, halves = _FIELDS[dtype]
    b = torch.randint(0, 256, (n_blocks, size), dtype=torch.uint8, device="cuda", generator=gen)
    if dtype == Q6K:
        b[:, 192:208] = ((b[:, 192:208] & 0x7F).to(torch.int16) - 64).to(torch.int8).view(torch.uint8)
    d = torch.randn(n_blocks, device="cuda", generator=gen).abs() * sigma
    for i, at in enumerate(halves):
        b[:, at:at + 2] = (d * MIN_OVER_D if i else d).to(torch.float16).view(torch.uint8).reshape(n_blocks, 2)
    return b.reshape(-1)


def _normals(gen, n, act=F32, sigma=1.0):
    return (torch.randn(n, device="cuda", generator=gen) * sigma).to(torch.float16 if act == F16 else torch.float32)


def _norm_weight(gen, n, act):
    return (1.0 + 0.1 * torch.randn(n, device="cuda", generator=gen)).to(torch.float16).to(torch.float16 if act == F16 else torch.float32)


def _blocks_host(rng, dtype, n_blocks, sigma):
    size, halves = _FIELDS[dtype]
    b = np.frombuffer(rng.bytes(n_blocks * size), np.uint8).reshape(n_blocks, size).copy()
    if dtype == Q6K:
        b[:, 192:208] = ((b[:, 192:208] & 0x7F).astype(np.int16) - 64).astype(np.int8).view(np.uint8)
    for at in halves:
        d = np.abs(rng.standard_normal(n_blocks, np.float32) * sigma).astype(np.float16)
        b[:, at:at + 2] = d.view(np.uint8).reshape(n_blocks, 2)
    return b


def _model_config(case, slots, max_seq):
    cfg = SHAPES[case["shape"]](max_seq=max_seq, n_slots=slots)
    if case.get("act") == "f16":
        cfg.act, cfg.sigma_w = F16, SIGMA_MODEL_F16
    if case.get("window"):
        cfg.sliding_window = case["window"]
        cfg.swa_layers = sum(1 << l for l in range(cfg.n_layers) if (l + 1) % WINDOW_EVERY)
    return cfg


def _build_model(ctx, cfg, seed):
    """A random-init model.  Every tensor is a run of blocks, at a place of its own, out of one random pool per format:
    as many bytes for the device to stream as distinct weights, quick to make."""
    rng = np.random.Generator(np.random.SFC64(seed))
    m = _Model(ctx, cfg)
    most = max(cfg.ffn * cfg.hidden, cfg.n_q * cfg.hd * cfg.hidden) // 256
    q4 = _blocks_host(rng, Q4K, most + 65536, cfg.sigma_w)
    for name, kind, rows, cols in ksm.tensor_specs(cfg):
        if kind == "norm":
            w = (1.0 + 0.1 * rng.standard_normal(cols, np.float32)).astype(np.float16).astype(np.float32)
            m.upload_tensor(name, w)
        elif kind == "q4k":
            n = rows * cols // 256
            at = int(rng.integers(0, len(q4) - n + 1))
            m.upload_tensor(name, q4[at:at + n])
        else:  # the tied table: distinct rows, or ids would share embeddings and logits
            m.upload_tensor(name, _blocks_host(rng, cfg.embd_dtype, rows * cols // 256, cfg.sigma_embd))
    return m, rng


def _logits(m, slot, slots=1):
    """The logits the last step of `slots` neighbouring slots left on the device."""
    ptr = m.lib.ks_model_debug_ptr(m.h, 1, slot)
    return torch.as_tensor(_Device(m, ptr, (slots * m.cfg.vocab,), "<f2" if m.cfg.act == F16 else "<f4"), device="cuda")


def _max_seq(n):
    """Slots are sized in steps of 256 positions."""
    return -(-n // 256) * 256


def prepare(case, seed):
    ctx = _context()
    kind = case["kind"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    act = F16 if case.get("act") == "f16" else F32
    eng = Eng(act)
    if kind in ("matvec", "head"):
        n = case.get("n_tok", 1)
        dt = Q6K if kind == "head" or case["dtype"] == "q6k" else Q4K
        W = _blocks_gpu(gen, dt, case["rows"] * case["cols"] // 256, SIGMA)
        x = _normals(gen, n * case["cols"])
        y = torch.zeros((n, case["rows"]), dtype=torch.float32, device="cuda")
        tok = torch.zeros(1, dtype=torch.float32, device="cuda")
        s = _State(kind=kind, case=case, ctx=ctx, eng=eng, dt=dt, keep=(W, x), y=y, tok=tok, bW=_wrap(ctx, W), bx=_wrap(ctx, x),
                   by=_wrap(ctx, y), btok=_wrap(ctx, tok))
    elif kind == "attention":
        lens = [int(v) for v in case["lens"].split(",")]
        n, n_q, n_kv, max_t = len(lens), case["n_q"], case["n_kv"], _max_seq(max(lens))
        stride = max_t * n_kv * HEAD_DIM // 32 * 18
        K, V = (_blocks_gpu(gen, Q40, n * stride // 18, 0.1) for _ in range(2))
        q = _normals(gen, n * n_q * HEAD_DIM, act)
        meta = torch.tensor([[t, 0, 0, 0] for t in lens], dtype=torch.float32, device="cuda")
        out = torch.zeros((n, n_q * HEAD_DIM), dtype=q.dtype, device="cuda")
        splits = ctx.lib.ks_sdpa_pick_splits(ctx.h, n, n_kv, max_t)
        tmp = torch.zeros(max(4, eng.sdpa_tmp_floats(n_q, HEAD_DIM, splits, n)), dtype=torch.float32, device="cuda")
        s = _State(kind=kind, case=case, ctx=ctx, eng=eng, n=n, max_t=max_t, stride=stride, keep=(K, V, q, meta, tmp), out=out,
                   bK=_wrap(ctx, K), bV=_wrap(ctx, V), bq=_wrap(ctx, q), bmeta=_wrap(ctx, meta), btmp=_wrap(ctx, tmp), bout=_wrap(ctx, out))
    elif kind == "layer":
        H, F, n_q, n_kv, t = (case[k] for k in ("hidden", "ffn", "n_q", "n_kv", "tlen"))
        qn, kvn, max_t = n_q * HEAD_DIM, n_kv * HEAD_DIM, _max_seq(case["tlen"])
        T = {k: _blocks_gpu(gen, Q4K, r * c // 256, SIGMA) for k, r, c in
             (("wq", qn, H), ("wk", kvn, H), ("wv", kvn, H), ("wo", H, qn), ("wg", F, H), ("wu", F, H), ("wd", H, F))}
        T.update({k: _norm_weight(gen, w, act) for k, w in
                  (("n_attn", H), ("n_q", HEAD_DIM), ("n_k", HEAD_DIM), ("n_post", H), ("n_ffn", H), ("n_ffw", H), ("n_next", H))})
        T["x"] = _normals(gen, H, act)
        dt = T["x"].dtype
        T.update({k: torch.zeros(w, dtype=dt, device="cuda") for k, w in
                  (("x2", H), ("q", qn), ("k", kvn), ("v", kvn), ("o", qn), ("ff", F), ("xa", H), ("xb", H), ("yb", H))})
        nb = max_t * n_kv * HEAD_DIM // 32
        T["K"], T["V"] = (_blocks_gpu(gen, Q40, nb, 0.1) for _ in range(2))
        T["meta"] = torch.tensor([t, 0, 0, 0], dtype=torch.float32, device="cuda")
        half = HEAD_DIM // 2
        ang = torch.arange(max_t, device="cuda").float()[:, None] * 1e6 ** (-torch.arange(half, device="cuda").float() * 2 / HEAD_DIM)
        T["rope"] = torch.cat([ang.cos(), ang.sin()], 1).contiguous()
        T["tmp"] = torch.zeros(eng.sdpa_tmp_floats(n_q, HEAD_DIM, _lib_max_splits(ctx, n_kv, max_t)), dtype=torch.float32, device="cuda")
        s = _State(kind=kind, case=case, ctx=ctx, eng=eng, T=T, B={k: _wrap(ctx, v) for k, v in T.items()}, max_t=max_t)
    elif kind == "serve":
        cfg = _model_config(case, case["slots"], _max_seq(case["prompt_hi"] + case["new"] + 1))
        m, rng = _build_model(ctx, cfg, seed)
        lens = rng.integers(case["prompt_lo"], case["prompt_hi"] + 1, case["requests"])
        s = _State(kind=kind, case=case, ctx=ctx, model=m, prompts=[rng.integers(0, cfg.vocab, n).tolist() for n in lens],
                   logits=_logits(m, 0, case["slots"]))
    else:
        cfg = _model_config(case, 1, _max_seq(case["prompt"] + case.get("new", 1) + 1))
        m, rng = _build_model(ctx, cfg, seed)
        slot = m.slot_alloc()
        s = _State(kind=kind, case=case, ctx=ctx, model=m, slot=slot, prompt=rng.integers(0, cfg.vocab, case["prompt"]).tolist(),
                   given=rng.integers(0, cfg.vocab, case.get("new", 1)).tolist(), logits=_logits(m, slot))
    torch.cuda.synchronize()
    return s


def _lib_max_splits(ctx, n_kv, max_t):
    return max(Eng.SDPA_MWG_NWG, ctx.lib.ks_sdpa_pick_splits(ctx.h, 1, n_kv, max_t))


# ---- one pass ---------------------------------------------------------------------------------------

def run(s):
    return _RUN[s.kind](s)


def _run_matvec(s):
    c = s.case
    if c["n_tok"] == 1:
        s.eng.matvec_wd(s.ctx, c["rows"], c["cols"], s.dt, s.bW, s.bx, s.by)
    else:
        s.eng.matvec_batch(s.ctx, c["rows"], c["cols"], c["n_tok"], s.dt, s.bW, s.bx, s.by)
    return s.y


def _run_head(s):
    s.eng.matvec_wd(s.ctx, s.case["rows"], s.case["cols"], s.dt, s.bW, s.bx, s.by)
    s.eng.softcap_argmax(s.ctx, s.case["rows"], 30.0, s.by, s.btok)
    return {"logits": s.y, "token": s.tok}


def _run_attention(s):
    s.eng.sdpa_decode(s.ctx, s.n, s.case["n_q"], s.case["n_kv"], HEAD_DIM, s.max_t, s.bq, s.bK, s.bV, s.bmeta, s.btmp, s.bout,
                      scale=HEAD_DIM ** -0.5, slot_stride_bytes=s.stride)
    return s.out


def _run_layer(s):
    c, e, x, B = s.case, s.eng, s.ctx, s.B
    H, F, n_q, n_kv, t = (c[k] for k in ("hidden", "ffn", "n_q", "n_kv", "tlen"))
    row = (t - 1) * n_kv * HEAD_DIM // 32 * 18
    e.rmsnorm(x, H, 1e-6, B["x"], B["n_attn"], B["x2"])
    e.matvec_qkv_wd(x, n_q * HEAD_DIM, n_kv * HEAD_DIM, H, Q4K, B["wq"], B["wk"], B["wv"], B["x2"], B["q"], B["k"], B["v"])
    e.rmsnorm_per_head_qkv_q40_off(x, n_q, n_kv, HEAD_DIM, 1e-6, B["q"], B["n_q"], B["rope"], (t - 1) * HEAD_DIM, B["k"], B["n_k"],
                                   B["v"], B["q"], B["K"], B["V"], row)
    e.sdpa_hybrid_kv(x, n_q, n_kv, HEAD_DIM, s.max_t, t, Q40, B["q"], B["K"], B["V"], B["meta"], B["tmp"], B["o"], HEAD_DIM ** -0.5)
    e.matvec_wd(x, H, n_q * HEAD_DIM, Q4K, B["wo"], B["o"], B["yb"])
    e.rmsnorm_add_then_rmsnorm(x, H, 1e-6, B["yb"], B["n_post"], B["x"], B["n_ffn"], B["xa"], B["x2"])
    e.matvec_gate_up_gelu_wd(x, F, H, Q4K, B["wg"], B["wu"], B["x2"], B["ff"])
    e.matvec_wd(x, H, F, Q4K, B["wd"], B["ff"], B["yb"])
    e.rmsnorm_add_then_rmsnorm(x, H, 1e-6, B["yb"], B["n_ffw"], B["xa"], B["n_next"], B["xb"], B["x2"])
    return {"x": s.T["xb"], "x2": s.T["x2"]}


def _run_generate(s):
    toks, _ = s.model.generate_timed(s.prompt, s.case["new"], s.slot)
    return {"tokens": np.array(toks), "logits": s.logits}


def _run_score(s):
    m = s.model
    m.slot_reset(s.slot)
    m.prefill(s.slot, s.prompt)
    for t in s.given:
        m.forward(s.slot, 1, [t], True)
    return s.logits


def _run_first(s):
    m = s.model
    m.slot_reset(s.slot)
    m.prefill(s.slot, s.prompt[:-1])
    return {"token": m.decode_token([s.prompt[-1]], s.slot)[0], "logits": s.logits}


def _run_serve(s):
    c = s.case
    reqs = [InferenceRequest(p, max_tokens=c["new"], temperature=c["temperature"], min_p=0.05, seed=7 + i) for i, p in enumerate(s.prompts)]
    sched = Scheduler(s.model, SchedulerConfig(slots=c["slots"]))
    for r in reqs:
        sched.submit(r)
    sched.run()
    bad = [e for r in reqs for e in r.events if e[0] == "error"]
    if bad:
        raise RuntimeError(bad[0][1])
    tokens = np.full((len(reqs), c["new"]), -1)   # a request may stop early
    for row, r in zip(tokens, reqs):
        got = [e[1] for e in r.events if e[0] == "token"]
        row[:len(got)] = got
    return {"tokens": tokens, "logits": s.logits}


_RUN = {"matvec": _run_matvec, "head": _run_head, "attention": _run_attention, "layer": _run_layer, "generate": _run_generate,
        "score": _run_score, "first": _run_first, "serve": _run_serve}


# ---- what a pass cannot do without, and how far a correct one may be off -------------------------------

def _layer_weights(cfg):
    """Weights of one layer (all Q4_K)."""
    qn, kvn = cfg.n_q * cfg.hd, cfg.n_kv * cfg.hd
    return cfg.hidden * (2 * qn + 2 * kvn + 3 * cfg.ffn)


def _model_work(cfg, prompt_tokens, prompt_passes, steps, rows_per_step, context):
    """prompt_passes: how often the layers' weights must be read for prompts; steps decode steps of rows_per_step rows each
    at about `context` positions."""
    lw, head = _layer_weights(cfg) * cfg.n_layers, cfg.vocab * cfg.hidden
    kv = cfg.n_layers * cfg.n_kv * cfg.hd // 32 * 18 * 2
    byt = lw * 144 / 256 * (prompt_passes + steps) + head * 210 / 256 * steps + kv * (prompt_tokens + steps * rows_per_step * context)
    flo = 2.0 * lw * (prompt_tokens + steps * rows_per_step) + 2.0 * head * steps * rows_per_step
    flo += 4.0 * cfg.n_layers * cfg.n_q * cfg.hd * (prompt_tokens * context / 2 + steps * rows_per_step * context)
    return {"bytes": byt, "flops": flo}


def work(case):
    kind = case["kind"]
    if kind in ("matvec", "head"):
        n, r, c = case.get("n_tok", 1), case["rows"], case["cols"]
        per = 210 if kind == "head" or case["dtype"] == "q6k" else 144
        return {"bytes": r * c / 256 * per + 4 * n * (r + c), "flops": 2.0 * n * r * c}
    if kind == "attention":
        lens = [int(v) for v in case["lens"].split(",")]
        a = 2 if case["act"] == "f16" else 4
        return {"bytes": sum(lens) * case["n_kv"] * HEAD_DIM // 32 * 18 * 2 + 2 * a * len(lens) * case["n_q"] * HEAD_DIM,
                "flops": 4.0 * sum(lens) * case["n_q"] * HEAD_DIM}
    if kind == "layer":
        H, F, n_q, n_kv, t = (case[k] for k in ("hidden", "ffn", "n_q", "n_kv", "tlen"))
        w = H * HEAD_DIM * (2 * n_q + 2 * n_kv) + 3 * H * F
        return {"bytes": w * 144 / 256 + t * n_kv * HEAD_DIM // 32 * 18 * 2 + 4 * H * 8, "flops": 2.0 * w + 4.0 * t * n_q * HEAD_DIM}
    if kind == "serve":
        cfg = _model_config(case, case["slots"], 256)
        mean = (case["prompt_lo"] + case["prompt_hi"]) / 2
        rounds = -(-case["requests"] // case["slots"]) * case["new"]
        return _model_work(cfg, case["requests"] * (mean - 1), 1, rounds, case["requests"] * case["new"] / rounds, mean)
    cfg = _model_config(case, 1, 256)
    steps = case.get("new", 1)
    return _model_work(cfg, case["prompt"], 1, steps, 1, min(case["prompt"], case.get("window") or case["prompt"]))


def tolerance(case):
    kind = case["kind"]
    if case.get("act") == "f16":
        # every op rounds to f16 (2^-11); a layer is ~10 roundings of the residual stream, a model dozens of layers
        return {"rel": 5e-3} if kind in ("score", "generate", "first") else {"rel": 3e-3}
    if kind in ("matvec", "attention"):
        return {"rel": 1e-5}            # f32 sums over hundreds to ten thousand terms
    if kind == "head":
        return {"rel": 1e-5}            # the arg-max comes back as a float: it has to be the same token
    if kind == "layer":
        return {"rel": 1e-4}            # a cache value on a rounding boundary may move by one of 15 steps
    # f32 throughout, but the caches are 4-bit: a last-bit difference can move a cached value by a step, and later layers
    # see that.  Greedy and sampled ids may differ where two candidates tie.
    return {"rel": 1e-4, "max": 1e-2, "differ": 0.01}
