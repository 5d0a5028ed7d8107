"""The work a user has this framework do, as measurable cases: training steps, token steps, prompts and whole requests.

Training recipes and model sizes are those of ``configs/``; layer-list models have the sizes of ``bench_layers.py``.  A case is
plain values:

* ``train``: one optimizer step of a recipe through :class:`CudaEngine` (``accum`` micro-batches of ``rows`` x ``seq`` tokens fused
  into one pass, as the trainer fuses them): host tokens in, loss and gradient norm out, weights updated.
* ``token``: one token for each of ``batch`` sequences that hold ``context`` tokens, through :class:`InferenceEngine`.
* ``prompt``: a prompt of ``tokens`` tokens per sequence into an empty cache, through the same engine.
* ``list_prompt`` / ``list_request``: a prompt, and a whole greedy generation, of a layer-list model through :class:`LayerEngine`.

Weights are drawn, not trained, but arranged so that decisions are as clear as a trained model's: a token's embedding carries
its experts' order of preference (so no router choice hangs on the last bit of a 16-bit number), and the output rows of layer-list
models follow their embeddings in another order (so that a greedy continuation is a walk through the vocabulary).
"""
import math
import os
from unittest import mock

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
LEVEL, SIGMA, FINAL = 2.0, 0.5, 0.02       # spacing of expert preferences, scale of embeddings, weight of the last norm
STEP, LR = 100, 1e-5                       # a step of the warm-up


# ------------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # a pre-training step of the mid-sized recipe: 32768 tokens of packed documents, AdamW
        {"name": "train_480m", "kind": "train", "recipe": "flash_480m_2xt4", "rows": 2, "seq": 1024, "accum": 16, "dtype": "fp16"},
        # the largest recipe with short accumulation (many GPUs share a global batch), Lion
        {"name": "train_1b_small_step", "kind": "train", "recipe": "pro_1b_2xt4", "rows": 1, "seq": 512, "accum": 16, "dtype": "fp16"},
        # the dense recipe in bf16
        {"name": "train_dense_bf16", "kind": "train", "recipe": "t4_en_120m_fast", "rows": 4, "seq": 1024, "accum": 4, "dtype": "bf16"},
        # the compact recipe on one odd-length batch: fine-tuning with few tokens per step, where launches count
        {"name": "train_109m_short", "kind": "train", "recipe": "flash_109m_compact_2xt4", "rows": 1, "seq": 1000, "accum": 1, "dtype": "fp16"},
        # chat with the largest model: one sequence, 16-bit weights
        {"name": "token_1b_f16", "kind": "token", "recipe": "pro_1b_2xt4", "fmt": "f16", "batch": 1, "context": 1024},
        # chat deep into a conversation with a 4-bit file
        {"name": "token_480m_q4_deep", "kind": "token", "recipe": "flash_480m_2xt4", "fmt": "q4_0", "batch": 1, "context": 3001},
        # serving a batch from an 8-bit file
        {"name": "token_480m_q8_batch32", "kind": "token", "recipe": "flash_480m_2xt4", "fmt": "q8_0", "batch": 32, "context": 500},
        # reading a question and its documents
        {"name": "prompt_480m", "kind": "prompt", "recipe": "flash_480m_2xt4", "fmt": "f16", "batch": 1, "tokens": 1501},
        # a long document through the state-space model, in portions
        {"name": "list_prompt_mamba", "kind": "list_prompt", "design": "Zikedra", "size": "m", "layers": 12, "batch": 1, "tokens": 8192},
        # two documents of an odd length through the latent-attention model
        {"name": "list_prompt_latent", "kind": "list_prompt", "design": "Dunavik", "size": "m", "layers": 12, "batch": 2, "tokens": 3001},
        # a short question and its answer, one user
        {"name": "list_request_mamba", "kind": "list_request", "design": "Zikedra", "size": "s", "layers": 12, "batch": 1, "tokens": 100, "new": 64},
        # a batch of requests
        {"name": "list_request_latent_batch32", "kind": "list_request", "design": "Dunavik", "size": "s", "layers": 12, "batch": 32, "tokens": 128, "new": 64},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("train", "token", "token", "prompt", "list_prompt", "list_request"))
    small = ("flash_109m_compact_2xt4", "flash_109m_compact_2xt4", "flash_480m_2xt4")
    if kind == "train":
        recipe = rng.choice(small + ("t4_en_120m_fast",))
        seq, most = _log(rng, 128, 2048), 8192 if recipe == "flash_480m_2xt4" else 16384
        rows = rng.randint(1, max(1, min(4, most // seq)))
        # balance statistics stay per micro-batch where these are whole routing blocks of 256 tokens
        accum = rng.choice((1, 2, 4, 8)) if rows * seq % 256 == 0 else 1
        while rows * seq * accum > most:
            accum //= 2
        return {"kind": kind, "recipe": recipe, "rows": rows, "seq": seq, "accum": accum, "dtype": rng.choice(("fp16", "fp16", "bf16"))}
    if kind == "token":
        batch = rng.choice((1, 1, 1, 2, 3, 4, 7, 8, 16, 24, 32))
        return {"kind": kind, "recipe": rng.choice(small), "fmt": rng.choice(("f16", "q8_0", "q4_0")), "batch": batch,
                "context": _log(rng, 20, min(4000, 16384 // batch))}
    if kind == "prompt":
        return {"kind": kind, "recipe": rng.choice(small), "fmt": "f16", "batch": rng.choice((1, 1, 2, 4)), "tokens": _log(rng, 66, 4000)}
    design, size = rng.choice(("Zikedra", "Dunavik")), rng.choice(("s", "m"))
    if kind == "list_prompt":
        batch = rng.choice((1, 1, 2, 4))
        return {"kind": kind, "design": design, "size": size, "layers": rng.choice((4, 8, 12)), "batch": batch, "tokens": _log(rng, 100, 8192 // batch)}
    return {"kind": kind, "design": design, "size": size, "layers": rng.choice((4, 8, 12)), "batch": rng.choice((1, 1, 2, 4, 8, 16, 32)),
            "tokens": _log(rng, 20, 500), "new": rng.choice((16, 32, 64))}


# ------------------------------------------------------------------------------------------------ configurations
def _model_config(case):
    from ghassan_b200.models.config import ModelConfig
    from ghassan_b200.utils.config import Config
    return ModelConfig.from_config(Config.from_file(os.path.join(ROOT, "configs", case["recipe"] + ".yaml")))


def _trainer_config(case):
    from ghassan_b200.training.config import TrainerConfig
    from ghassan_b200.utils.config import Config
    t = TrainerConfig.from_config(Config.from_file(os.path.join(ROOT, "configs", case["recipe"] + ".yaml")))
    t.compute_dtype = case["dtype"]
    t.seq_len, t.batch_size, t.grad_accum = case["seq"], case["rows"] * case["accum"], 1
    t.micro_tokens = case["rows"] * case["seq"] if case["accum"] > 1 else 0
    return t


SIZES = {"s": dict(width=1024, ff=2816, H=16, G=4, hd=64, mh=32), "m": dict(width=2560, ff=6912, H=20, G=5, hd=128, mh=80)}
LATENT = {"s": dict(dim=64, rot_dim=32, vdim=64, kv_rank=256, q_rank=512), "m": dict(dim=64, rot_dim=64, vdim=128, kv_rank=512, q_rank=768)}
VOCAB = 32000


def _list_json(case):
    z, side = SIZES[case["size"]], case["design"] == "Dunavik"
    mlp = {"kind": "dense", "ff": z["ff"]}
    attn = {"heads": z["H"], "kv_heads": z["G"], "dim": z["hd"], "vdim": z["hd"], "scale": z["hd"] ** -0.5}
    if side:
        la = LATENT[case["size"]]
        most = {"type": "attention", "mlp": mlp, "mixer": dict(attn, softcap=30.0, mask={"size": 1024}, q_temp={"coef": 0.1, "every": 4096})}
        each4 = {"type": "latent_attention", "mlp": mlp,
                 "mixer": dict(la, heads=z["H"], scale=(la["dim"] + la["rot_dim"]) ** -0.5, rot={"base": 500000.0, "dims": la["rot_dim"]})}
    else:
        most = {"type": "mamba2", "mlp": mlp, "mixer": {"heads": z["mh"], "vdim": 64, "state": 128, "groups": 1, "conv": 4, "norm_groups": 1}}
        each4 = {"type": "attention", "mlp": mlp,
                 "mixer": dict(attn, mask={"size": 1024, "keep_first": 8}, rot={"base": 500000.0, "dims": z["hd"], "scaling": None})}
    d = {"architecture": case["design"], "layers": [each4 if i % 4 == 3 else most for i in range(case["layers"])], "width": z["width"],
         "vocab": VOCAB, "norm": {"eps": 1e-5}}
    d.update({"residual_mult": 0.5} if side else {"logit_softcap": 30.0})
    return d


# ------------------------------------------------------------------------------------------------ weights
def _snap(w, fmt):
    """``w`` rounded to what format ``fmt`` stores (so that what is stored is what is drawn)."""
    if fmt == "f16":
        return w.half().float()
    b = w.reshape(-1, 32)
    if fmt == "q8_0":
        d = (b.abs().amax(1, keepdim=True) / 127.0).half().float()
        return (torch.round(b / d).clamp_(-127, 127) * d).reshape(w.shape)
    top = b.gather(1, b.abs().argmax(1, keepdim=True))
    d = (top / -8.0).half().float()
    return ((torch.floor(b / d + 8.5).clamp_(0, 15) - 8.0) * d).reshape(w.shape)


def _weights(cfg, seed, fmt):
    """fp32 tensors on the GPU by parameter name."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    n = lambda *s: torch.randn(s, device="cuda", generator=g)
    d, ne = cfg.hidden_size, cfg.num_experts
    u = torch.linalg.qr(n(d, ne))[0] if cfg.use_moe else None
    out = {}
    for s in cfg.param_specs():
        leaf = s.name.split(".")[-1]
        if leaf == "tok_embeddings":
            t = n(*s.shape)
            if cfg.use_moe:
                wish = torch.rand(s.shape[0], ne, device="cuda", generator=g).argsort(1).float() - (ne - 1) / 2
                t += (LEVEL * wish - t @ u) @ u.t()
            t = (t * SIGMA).half().float()
        elif leaf == "final_norm":
            t = FINAL * (1.0 + 0.1 * n(*s.shape))
        elif s.init == "ones":
            t = 1.0 + 0.1 * n(*s.shape)
        elif s.init == "router":
            t = 0.5 * u.t()[torch.randperm(ne, device="cuda", generator=g)] + 0.01 * n(*s.shape)
        else:
            t = _snap(n(*s.shape) * (cfg.init_std if s.init == "normal" else cfg.init_std / math.sqrt(2.0 * cfg.num_layers)), fmt)
        out[s.name] = t
    return out


def _list_weights(case, seed):
    from ghassan_b200.models.layer_list import LayerListConfig, random_parameters
    cfg = LayerListConfig.from_json(_list_json(case))
    w = random_parameters(cfg, seed, device="cuda")
    g = torch.Generator(device="cuda").manual_seed(seed + 1)
    order = torch.randperm(VOCAB, device="cuda", generator=g)
    w["embed"] = (3.0 * w["embed"].float()).to(w["embed"].dtype)
    w["head"] = (w["embed"].float()[order] / 3.0 * cfg.hidden_size ** -0.5).to(w["embed"].dtype)
    return cfg, w


# ------------------------------------------------------------------------------------------------ inputs
def _train_batch(case, cfg, seed):
    """Packed documents: token ids, next-token targets (the first tokens of some documents unsupervised), document ids."""
    r = np.random.RandomState(seed % (1 << 32))
    B, T = case["rows"] * case["accum"], case["seq"]
    ids = r.randint(0, cfg.vocab_size, (B, T + 1))
    seg, mask = np.zeros((B, T), dtype=np.int64), np.zeros((B, T), dtype=bool)
    for b in range(B):
        at, k = 0, 0
        while at < T:
            n = int(np.exp(r.uniform(math.log(16), math.log(2048))))
            seg[b, at:at + n] = k
            mask[b, max(0, at + n - 1):at + n] = True                 # the next document's first token is no target
            if r.rand() < 0.3:
                mask[b, at:at + n // 4] = True
            at, k = at + n, k + 1
    tg = np.where(mask, -100, ids[:, 1:])
    i32 = lambda a: torch.from_numpy(np.ascontiguousarray(a.reshape(-1), dtype=np.int32))
    return i32(ids[:, :-1]), i32(tg), i32(seg)


def _prompts(batch, n, vocab, seed):
    r = np.random.RandomState((seed + 77) % (1 << 32))
    return torch.from_numpy(r.randint(3, vocab, (batch, n)).astype(np.int32))


# ------------------------------------------------------------------------------------------------ prepare, run
def prepare(case, seed):
    from ghassan_b200.utils import log
    log.set_log_level(log.WARN)
    kind = case["kind"]
    if kind == "train":
        return _prepare_train(case, seed)
    if kind in ("token", "prompt"):
        return _prepare_decoder(case, seed)
    from ghassan_b200.inference.generator import Generator
    from ghassan_b200.inference.layer_engine import LayerEngine
    from ghassan_b200.inference.token_loop import SamplingParams
    cfg, w = _list_weights(case, seed)
    eng = LayerEngine(cfg, w, batch=case["batch"], max_len=case["tokens"] + case.get("new", 0) + 64)
    prompts = _prompts(case["batch"], case["tokens"], VOCAB, seed)
    st = {"kind": kind, "eng": eng, "prompts": prompts}
    if kind == "list_request":
        st.update(gen=Generator(eng), new=case["new"], sp=SamplingParams(greedy=True, repetition_penalty=1.0, seed=1))
        st["gen"].generate(prompts.tolist(), max_new_tokens=4, sampling=st["sp"], stop_tokens=())      # a server's first request: captures the step
    return st


def _prepare_train(case, seed):
    from ghassan_b200.models.cuda_model import CudaModel
    from ghassan_b200.training.cuda_engine import CudaEngine
    cfg, tcfg = _model_config(case), _trainer_config(case)
    named = _weights(cfg, seed, "f16")
    # weights come from a checkpoint; drawing the recipe's initial ones on the host would take longer than all the rest
    with mock.patch.object(CudaModel, "init_weights", lambda self, s: self.load_named(named)):
        eng = CudaEngine(cfg, tcfg)
    pin = lambda t: t.pin_memory()
    ids, tg, sg = (pin(t) for t in _train_batch(case, cfg, seed))
    st = {"kind": "train", "eng": eng, "batch": (ids, tg, sg if tcfg.pack_sequences else None, tcfg.batch_size, tcfg.seq_len),
          "scale": 8192.0 if case["dtype"] == "fp16" else 1.0, "lr": 0.0}
    for _ in range(3):                       # the pass is captured in the third step of a run; a zero rate leaves the weights alone
        run(st)
    opt = eng.optimizer
    for m in (opt.m_flat, opt.v_flat):
        if m is not None:
            m.zero_()
    eng.set_opt_step(0)
    st["lr"] = LR
    return st


def _prepare_decoder(case, seed):
    from ghassan_b200.inference.engine import InferenceEngine, SamplingParams
    cfg, B = _model_config(case), case["batch"]
    n = case.get("context") or case["tokens"]
    named = {k: v.cpu().numpy() for k, v in _weights(cfg, seed, case["fmt"]).items()}
    eng = InferenceEngine(cfg, named, fmt=case["fmt"], batch=B, max_len=n + 64, prefill_chunk=n)
    st = {"kind": case["kind"], "eng": eng, "prompts": _prompts(B, n, cfg.vocab_size, seed)}
    eng.reset(1)
    if case["kind"] == "prompt":
        eng.prefill(_prompts(B, min(n, 80), cfg.vocab_size, seed + 1))       # a server has answered before: the prompt pass has its weights
        return st
    eng.prefill(st["prompts"])
    st["sp"] = SamplingParams(seed=1)
    st["saved"] = [t.clone() for t in (eng.state, eng.pos, eng.hist_len)]
    st["next"] = torch.from_numpy(np.random.RandomState((seed + 5) % (1 << 32)).randint(3, cfg.vocab_size, B).astype(np.int32)).cuda()
    eng.decode_steps(1, st["sp"])            # the first step is captured
    return st


def run(state):
    kind, eng = state["kind"], state["eng"]
    if kind == "train":
        eng.begin_step(STEP, state["scale"])
        eng.micro_step(*state["batch"])
        res = eng.end_step(state["lr"])
        return {"loss": float(res.loss), "norm": float(res.gnorm), "grads": eng.model.Gr[eng.model.layout.decay_start:],
                "grads_vocab": eng.model.Gr[:eng.model.layout.decay_start], "weights": eng.model.P}
    if kind == "token":                      # continue from the kept context
        eng.reset(1)
        for t, s in zip((eng.state, eng.pos, eng.hist_len), state["saved"]):
            t.copy_(s)
        eng.cur_tok.copy_(state["next"])
        eng.decode_steps(1, state["sp"])
        return {"logits": eng.logits}
    if kind == "prompt":
        eng.reset(1)
        eng.prefill(state["prompts"])
        return {"logits": eng.logits, "k": [L.cK for L in eng.layers], "v": [L.cV for L in eng.layers]}
    if kind == "list_prompt":
        eng.reset(1)
        eng.prefill(state["prompts"])
        return {"logits": eng.logits, "memory": [{k: getattr(c, k) for k in ("k", "v", "rows", "conv", "ssm") if hasattr(c, k)} for c in eng.mem.layers]}
    res = state["gen"].generate(state["prompts"].tolist(), max_new_tokens=state["new"], sampling=state["sp"], stop_tokens=())
    return {"tokens": np.asarray([[int(t) for t in row] for row in res.tokens], dtype=np.int64), "logits": eng.logits}


# ------------------------------------------------------------------------------------------------ what a pass cannot do without
def work(case):
    kind = case["kind"]
    if kind.startswith("list"):
        return _list_work(case)
    c = _model_config(case)
    d, L, E = c.hidden_size, c.num_layers, c.moe_expert_dim if c.use_moe else c.intermediate_size
    attn, head = d * (2 * c.q_dim + 2 * c.kv_dim), c.vocab_size * d
    sh = int(c.moe_shared) if c.use_moe else 1
    per, router = 3 * d * E, (c.num_experts * d if c.use_moe else 0)
    top = c.moe_top_k if c.use_moe else 0
    active = L * (attn + (top + sh) * per + router) + head
    total = c.count_parameters()
    if kind == "train":
        n = case["rows"] * case["seq"] * case["accum"]
        keys = min(case["seq"], 300) / 2.0                       # documents are log-uniform up to 2048 tokens
        state = 16 if _trainer_config(case).optimizer == "adamw" else 8      # moments, read and written
        return {"bytes": total * (12.0 + state) + n * 12, "flops": 6.0 * n * active + 12.0 * n * L * keys * c.q_dim}
    B = case["batch"]
    if kind == "token":
        per_param = {"f16": 2.0, "q8_0": 34 / 32, "q4_0": 18 / 32}[case["fmt"]]
        seen = (c.num_experts * (1 - (1 - top / c.num_experts) ** B) if c.use_moe else 0) + sh
        kv = B * case["context"] * 2 * c.kv_dim * 2.0 * L
        return {"bytes": L * (attn + seen * per) * per_param + L * router * 4 + head * 2.0 + kv + B * c.vocab_size * 4,
                "flops": 2.0 * B * active + 4.0 * B * case["context"] * c.q_dim * L}
    n = case["tokens"]
    flops = 2.0 * B * n * (active - head) + 2.0 * B * head + 4.0 * B * n * n / 2 * c.q_dim * L
    return {"bytes": (total - head) * 2.0 + B * n * (2 * c.kv_dim * 2.0 * L + d * 4) + head * 2, "flops": flops}


def _list_work(case):
    z, side, L, B = SIZES[case["size"]], case["design"] == "Dunavik", case["layers"], case["batch"]
    d, H, hd, G = z["width"], z["H"], z["hd"], z["G"]
    n4 = L // 4
    mlp = (2 if side else 3) * d * z["ff"]
    attn = d * hd * (2 * H + 2 * G) + (0 if side else d * H * hd)
    if side:
        la = LATENT[case["size"]]
        qk = la["dim"] + la["rot_dim"]
        lat = d * (la["q_rank"] + la["kv_rank"] + la["rot_dim"] + 2 * H * la["vdim"]) + H * (la["q_rank"] * qk + la["kv_rank"] * (la["dim"] + la["vdim"]))
        params = (L - n4) * attn + n4 * lat + L * mlp
    else:
        inner = z["mh"] * 64
        mamba = d * (3 * inner + 2 * 128 + z["mh"]) + 4 * (inner + 256)
        params = (L - n4) * mamba + n4 * attn + L * mlp

    def tokens(n):
        w = min(n, 1024)
        keys = w * n - w * w / 2.0
        f = 2.0 * n * params + (L - n4 if side else n4) * 4.0 * keys * H * hd
        if side:
            f += n4 * 2.0 * (n * n / 2.0) * H * (qk + la["vdim"])
        else:
            f += (L - n4) * 6.0 * n * inner * 128
        return f
    memory = (L - n4) * (2 * G * hd * 2.0 if side else 0) + n4 * ((la["kv_rank"] + la["rot_dim"]) * 2.0 if side else 2 * G * hd * 2.0)   # bytes a token
    fixed = 0 if side else (L - n4) * z["mh"] * 64 * 128 * 4.0
    n = case["tokens"]
    flops = B * (tokens(n) + 2.0 * VOCAB * d)
    nbytes = params * 2.0 + VOCAB * d * 2.0 + B * (n * (memory + d * 2.0) + fixed + VOCAB * 4)
    if case["kind"] == "list_request":
        new = case["new"] - 1
        flops += B * new * (2.0 * (params + VOCAB * d))
        nbytes += new * (params * 2.0 + VOCAB * d * 2.0 + B * (n * memory + 2 * fixed + VOCAB * 4))
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """About four times what another order of the sums shows."""
    kind = case["kind"]
    if kind == "train":
        return {"rel": 0.005 if case["dtype"] == "fp16" else 0.02, "max": 0.4}
    if kind in ("token", "prompt"):
        return {"rel": 0.02, "max": 0.4}
    return {"rel": 0.03, "max": 0.5, "differ": 0.002}


# ------------------------------------------------------------------------------------------------ 64-bit values
def exact(case, seed):
    kind = case["kind"]
    if kind == "train":
        return _exact_train(case, seed)
    with torch.no_grad():
        if kind in ("token", "prompt"):
            return _exact_decoder(case, seed)
        return _exact_list(case, seed)


def _rms(x, eps):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps)


def _turn(x, freq, pos):
    """[tokens, heads, dim]: neighbouring dimensions below 2 * len(freq) turn by position * frequency."""
    a = pos.double()[:, None] * freq[None, :]
    c, s = torch.cos(a)[:, None], torch.sin(a)[:, None]
    m = 2 * freq.numel()
    u, v = x[..., 0:m:2], x[..., 1:m:2]
    return torch.cat([torch.stack([u * c - v * s, u * s + v * c], -1).flatten(-2), x[..., m:]], -1)


def _attend(q, k, v, scale, see):
    """[T, H, hd] queries, [S, G, hd] keys; ``see`` [T, S]."""
    H, G = q.shape[1], k.shape[1]
    out = []
    for h in range(H):
        s = (q[:, h] @ k[:, h * G // H].t() * scale).masked_fill(~see, float("-inf"))
        out.append(torch.softmax(s, -1) @ v[:, h * G // H])
    return torch.cat(out, -1)


def _jitter(n, ne, seed):
    """The uniform number of (token, expert) under the step's seed: a 64-bit mix, high bits."""
    with np.errstate(over="ignore"):
        t, e = np.meshgrid(np.arange(n, dtype=np.uint64), np.arange(ne, dtype=np.uint64), indexing="ij")
        h = t * np.uint64(0x9E3779B97F4A7C15) ^ e * np.uint64(0xC2B2AE3D27D4EB4F) ^ np.uint64((seed + 0x9E3779B97F4A7C15) % (1 << 64))
        for m in (0xFF51AFD7ED558CCD, 0xC4CEB9FE1A85EC53):
            h = (h ^ (h >> np.uint64(33))) * np.uint64(m)
        h ^= h >> np.uint64(33)
    return torch.from_numpy((h >> np.uint64(40)).astype(np.float64) / (1 << 24) - 0.5).cuda()


def _decoder(c, w, ids, B, T, segments=None, jitter=None, keep=None):
    """Hidden states [B * T, d] of the decoder and the layers' balance terms; ``w(i, name)`` gives layer tensors, experts stacked."""
    d, H, G, hd = c.hidden_size, c.num_heads, c.num_kv_heads, c.head_dim
    pos = torch.arange(T, device="cuda")
    freq = c.rope_theta ** (-2.0 * torch.arange(hd // 2, device="cuda", dtype=torch.float64) / hd)
    x = w(-1, "tok_embeddings")[ids.reshape(-1)]
    aux = []
    causal = pos[None, :] <= pos[:, None]
    ffn = lambda h, wg, wu, wd: (torch.nn.functional.silu(h @ wg.t()) * (h @ wu.t())) @ wd.t()
    for l in range(c.num_layers):
        h = _rms(x, c.rms_eps) * w(l, "attn_norm")
        q, k, v = (t.view(B, T, -1, hd) for t in (h @ w(l, "wqkv").t()).split((c.q_dim, c.kv_dim, c.kv_dim), 1))
        if c.use_qk_norm:
            q, k = _rms(q, c.rms_eps) * w(l, "qk_qnorm"), _rms(k, c.rms_eps) * w(l, "qk_knorm")
        att, keys = [], []
        for b in range(B):
            see = causal if segments is None else causal & (segments[b][:, None] == segments[b][None, :])
            keys.append(_turn(k[b], freq, pos))
            att.append(_attend(_turn(q[b], freq, pos), keys[-1], v[b], hd ** -0.5, see))
        if keep is not None:
            keep.append((torch.stack(keys).reshape(B, T, -1), v.reshape(B, T, -1)))
        x = x + torch.cat(att) @ w(l, "wo").t()
        h = _rms(x, c.rms_eps) * w(l, "ffn_norm")
        gate, up, down = w(l, "gate"), w(l, "up"), w(l, "down")
        if not c.use_moe:
            x = x + ffn(h, gate[0], up[0], down[0])
            continue
        ne, K = c.num_experts, c.moe_top_k
        logits = h @ w(l, "router").t()
        if jitter is not None:
            logits = logits * (1.0 + 2.0 * c.moe_jitter * jitter)
        p = torch.softmax(logits, -1)
        idx = p.detach().topk(K, -1).indices
        wt = p.gather(1, idx)
        wt = wt / wt.sum(-1, keepdim=True)
        out = ffn(h, gate[ne], up[ne], down[ne]) if c.moe_shared else torch.zeros_like(x)
        for e in range(ne):
            at, slot = (idx == e).nonzero(as_tuple=True)
            out = out.index_add(0, at, ffn(h[at], gate[e], up[e], down[e]) * wt[at, slot][:, None])
        share = torch.bincount(idx.reshape(-1), minlength=ne).double() / idx.numel()
        aux.append(ne * (p.mean(0) * share).sum())
        x = x + out
    return _rms(x, c.rms_eps) * w(-1, "final_norm"), aux


def _segments(c):
    """Names and shapes of the flat parameter buffer, in its order: what takes no weight decay, routers, matrices."""
    d, hd, n1 = c.hidden_size, c.head_dim, c.num_experts + int(c.moe_shared) if c.use_moe else 1
    E = c.moe_expert_dim if c.use_moe else c.intermediate_size
    no = [((-1, "tok_embeddings"), (c.vocab_size, d)), ((-1, "final_norm"), (d,))]
    rt, mt = [], []
    for l in range(c.num_layers):
        no += [((l, "attn_norm"), (d,)), ((l, "ffn_norm"), (d,))]
        no += [((l, "qk_qnorm"), (hd,)), ((l, "qk_knorm"), (hd,))] if c.use_qk_norm else []
        rt += [((l, "router"), (c.num_experts, d))] if c.use_moe else []
        mt += [((l, "wqkv"), (c.q_dim + 2 * c.kv_dim, d)), ((l, "wo"), (d, c.q_dim)), ((l, "gu"), (n1, E // 64, 2, 64, d)), ((l, "down"), (n1, d, E))]
    return no, rt + mt


def _named_to(c, named, key):
    """One segment of the flat buffer from the named tensors."""
    l, n = key
    r = "layers.%d." % l
    cat = lambda *p: torch.cat([named[r + x] for x in p], 0)
    sh = c.use_moe and c.moe_shared
    if l < 0:
        return named[n]
    if n == "wqkv":
        return cat("wq", "wk", "wv")
    if n == "router":
        return named[r + "moe_router"]
    if n in ("gate", "up", "down"):
        t = named[r + "w_" + n] if not c.use_moe else cat(*(["moe_" + n] + (["moe_sh_" + n] if sh else [])))
        n1 = c.num_experts + int(sh) if c.use_moe else 1
        return t.reshape(n1, -1, t.shape[1])
    return named[r + n]


def _exact_train(case, seed):
    c, t = _model_config(case), _trainer_config(case)
    named = _weights(c, seed, "f16")
    no, rest = _segments(c)
    up = lambda n: (n + 63) // 64 * 64
    start = sum(up(math.prod(s)) for _, s in no)
    total = start + sum(up(math.prod(s)) for _, s in rest)
    P, G = (torch.zeros(total, dtype=torch.float64, device="cuda") for _ in range(2))
    leaf, off = {}, 0
    for key, shape in no + rest:
        n = math.prod(shape)
        v = P[off:off + n].view(shape)
        if key[1] == "gu":
            g, u = (_named_to(c, named, (key[0], x)) for x in ("gate", "up"))
            v.copy_(torch.stack([x.view(shape[0], shape[1], 64, shape[4]) for x in (g, u)], 2))
        else:
            v.copy_(_named_to(c, named, key).view(shape))
        leaf[key] = v.detach().requires_grad_()
        leaf[key].grad = G[off:off + n].view(shape)
        off += up(n)
    del named

    def w(l, n):
        if n in ("gate", "up"):
            x = leaf[l, "gu"][:, :, 0 if n == "gate" else 1]
            return x.reshape(x.shape[0], -1, x.shape[-1]).unbind(0)
        return leaf[l, n].unbind(0) if n == "down" else leaf[l, n]
    ids, tg, sg = (x.view(case["accum"], case["rows"], case["seq"]).long().cuda() for x in _train_batch(case, c, seed))
    scale = 8192.0 if case["dtype"] == "fp16" else 1.0
    js = (t.seed ^ ((STEP * 0x9E3779B97F4A7C15) % (1 << 64))) % (1 << 64)
    n = case["rows"] * case["seq"]
    jit = _jitter(n, c.num_experts, js) if c.use_moe and c.moe_jitter > 0 else None
    loss, ntok = 0.0, int((tg >= 0).sum())
    for a in range(case["accum"]):
        h, aux = _decoder(c, w, ids[a], case["rows"], case["seq"], sg[a] if t.pack_sequences else None, jit)
        y = tg[a].reshape(-1)
        on = y >= 0
        logits = h[on] @ leaf[-1, "tok_embeddings"].t()
        z = torch.logsumexp(logits, -1)
        obj = (z - logits.gather(1, y[on][:, None])[:, 0] + c.z_loss_scale * z * z).sum()
        if aux and c.moe_aux_scale > 0:
            obj = obj + int(on.sum()) * c.moe_aux_scale / c.num_layers * torch.stack(aux).sum()
        (obj * scale).backward()
        loss += float(obj.detach())
        del h, aux, logits, z, obj
    gs = 1.0 / (ntok * scale)
    norm = float(G.norm()) * gs
    gi = G * (gs * (min(1.0, t.grad_clip / (norm + 1e-6)) if t.grad_clip > 0 and norm > t.grad_clip else 1.0))
    step = gi / (gi.abs() + t.eps) if t.optimizer == "adamw" else torch.sign(gi)       # first step: zero moments
    step[start:] += t.weight_decay * P[start:]
    return {"loss": loss / ntok, "norm": norm, "grads": G[start:], "grads_vocab": G[:start], "weights": P - LR * step}


def _exact_decoder(case, seed):
    c, B = _model_config(case), case["batch"]
    n = case.get("context") or case["tokens"]
    named = {k: v.double() for k, v in _weights(c, seed, case["fmt"]).items()}
    ids = _prompts(B, n, c.vocab_size, seed).long().cuda()
    if case["kind"] == "token":
        nxt = np.random.RandomState((seed + 5) % (1 << 32)).randint(3, c.vocab_size, B)
        ids = torch.cat([ids, torch.from_numpy(nxt).long().cuda()[:, None]], 1)
    T, keep = ids.shape[1], []
    w = lambda l, x: _named_to(c, named, (l, x))
    h, _ = _decoder(c, w, ids, B, T, keep=keep if case["kind"] == "prompt" else None)
    logits = h.view(B, T, -1)[:, -1] @ named["tok_embeddings"].t()
    if case["kind"] == "token":
        return {"logits": logits}
    pad = lambda t: torch.nn.functional.pad(t, (0, 0, 0, 64))
    return {"logits": logits, "k": [pad(k) for k, _ in keep], "v": [pad(v) for _, v in keep]}


def _ring(x, keep, cap):
    """Rows of a cache that holds the last positions of x [T, ...] behind its first ``keep``."""
    out = torch.zeros((cap,) + tuple(x.shape[1:]), dtype=x.dtype, device=x.device)
    T = x.shape[0]
    p = torch.arange(T, device=x.device)
    ring = cap - keep
    p = p[(p < keep) | (p >= T - ring)]
    out[torch.where(p < keep, p, keep + (p - keep) % ring)] = x[p]
    return out


def _exact_list(case, seed):
    j = _list_json(case)
    _, raw = _list_weights(case, seed)
    w = {k: v.double() for k, v in raw.items()}
    del raw
    B, n = case["batch"], case["tokens"]
    ids = _prompts(B, n, VOCAB, seed).long().cuda()
    if case["kind"] == "list_request":
        # the continuation that follows the output rows' order, checked below by the logits themselves
        follow = torch.empty(VOCAB, dtype=torch.long, device="cuda")
        g = torch.Generator(device="cuda").manual_seed(seed + 1)
        order = torch.randperm(VOCAB, device="cuda", generator=g)
        follow[order] = torch.arange(VOCAB, device="cuda")
        for _ in range(case["new"] - 1):
            ids = torch.cat([ids, follow[ids[:, -1:]]], 1)
    logits, tokens, memory = [], [], None
    cap = n + 64
    for b in range(B):
        lg, mem = _list_forward(j, w, ids[b], n - 1, cap)
        logits.append(lg[-1])
        tokens.append(lg.argmax(-1))
        if case["kind"] == "list_prompt":
            memory = memory or [{k: [] for k in m} for m in mem]
            for a, m in zip(memory, mem):
                for k in m:
                    a[k].append(m[k])
    out = {"logits": torch.stack(logits)}
    if case["kind"] == "list_request":
        return dict(out, tokens=torch.stack(tokens).cpu().numpy())
    return dict(out, memory=[{k: (torch.stack(v) if v[0] is not None else None) for k, v in m.items()} for m in memory])


def _list_forward(j, w, ids, first, cap):
    """Logits of positions ``first`` on, and every layer's memory, for one sequence of a layer-list model in 64 bits."""
    eps, side, T = j["norm"]["eps"], j["architecture"] == "Dunavik", ids.numel()
    pos = torch.arange(T, device="cuda")
    up = lambda a: (a + 127) // 128 * 128

    def ln(x, name):
        x = x - x.mean(-1, keepdim=True)
        return _rms(x, eps) * w[name] + w[name + ".b"]
    turn = lambda x, r: _turn(x, float(r["base"]) ** (-2.0 * torch.arange(r["dims"] // 2, device="cuda", dtype=torch.float64) / r["dims"]), pos)
    x, memory = w["embed"][ids], []
    if side:
        x = ln(x, "embed.norm")
    for i, layer in enumerate(j["layers"]):
        m, t = layer["mixer"], {k[len("l%d.mix." % i):]: v for k, v in w.items() if k.startswith("l%d.mix." % i)}
        h = ln(x, "l%d.norm1" % i) if side else x
        heads = lambda a, H: a.view(T, H, -1)
        if layer["type"] == "mamba2":
            y, mem = _mamba(h, m, t, eps)
        elif layer["type"] == "latent_attention":
            H, R, dn = m["heads"], m["kv_rank"], m["dim"]
            q = heads((_rms(h @ t["dq"].t(), eps) * t["dq.norm"]) @ t["uq"].t(), H)
            down = h @ t["dkv"].t()
            c = _rms(down[:, :R], eps) * t["dkv.norm"]
            kr = turn(down[:, None, R:], m["rot"])
            k = torch.cat([heads(c @ t["uk"].t(), H), kr.expand(-1, H, -1)], -1)
            q = torch.cat([q[..., :dn], turn(q[..., dn:], m["rot"])], -1)
            y = _attend(q, k, heads(c @ t["uv"].t(), H), m["scale"], pos[None, :] <= pos[:, None])
            y = (y * torch.sigmoid(h @ t["g"].t())) @ t["o"].t()
            rows = torch.cat([c, kr[:, 0]], -1)
            mem = {"rows": torch.nn.functional.pad(rows, (0, 0, 0, up(cap) - T))}
        else:
            H, G, win, kf = m["heads"], m["kv_heads"], m["mask"]["size"], m["mask"].get("keep_first", 0)
            q, k, v = heads(h @ t["q"].t(), H), heads(h @ t["k"].t(), G), heads(h @ t["v"].t(), G)
            back = pos[:, None] - pos[None, :]
            see = (back >= 0) & ((back < win) | (pos[None, :] < kf))
            out = []
            if side:
                q = q * (1.0 + m["q_temp"]["coef"] * torch.log1p(((pos + 1) // m["q_temp"]["every"]).double()))[:, None, None]
            else:
                q, k = _rms(turn(q, m["rot"]), eps), _rms(turn(k, m["rot"]), eps)
            for a in range(H):
                s = q[:, a] @ k[:, a * G // H].t() * m["scale"]
                if side:
                    s = m["softcap"] * torch.tanh(s / m["softcap"]) - 2.0 ** (-8.0 * (a + 1) / H) * back
                    p = torch.softmax(s.masked_fill(~see, float("-inf")), -1)
                else:
                    s = torch.cat([s.masked_fill(~see, float("-inf")), t["sink"][a].expand(T, 1)], -1)
                    p = torch.softmax(s, -1)[:, :-1]
                out.append(p @ v[:, a * G // H])
            y = torch.cat(out, -1)
            y = (y if side else y * torch.sigmoid(h @ t["g"].t())) @ t["o"].t()
            chunk = min(2048, cap)
            rows = kf + up(min(cap - kf, win - 1 + chunk))
            mem = {"k": _ring(k, kf, rows), "v": _ring(v, kf, rows)}
        memory.append(mem)
        mlp = lambda n: w["l%d.mlp.%s" % (i, n)]
        if side:
            x = x + j["residual_mult"] * (y + torch.relu(h @ mlp("up").t()).square() @ mlp("down").t())
        else:
            x = x + _rms(y, eps) * w["l%d.norm1" % i]
            y = (torch.nn.functional.silu(x @ mlp("gate").t()) * (x @ mlp("up").t())) @ mlp("down").t()
            x = x + _rms(y, eps) * w["l%d.norm2" % i]
    x = x[first:]
    h = ln(x, "final.norm") if side else _rms(x, eps) * w["final.norm"]
    logits = h @ w["head"].t()
    cap = j.get("logit_softcap")
    return (cap * torch.tanh(logits / cap) if cap else logits), memory


def _mamba(h, m, t, eps):
    """The state recurrence in pieces of 128 tokens: inside a piece by its decay-weighted scores, between pieces by the state."""
    T, H, P, N, taps = h.shape[0], m["heads"], m["vdim"], m["state"], m["conv"]
    n = H * P
    p = h @ t["in"].t()
    z, xbc, dt = p[:, :n], p[:, n:2 * n + 2 * N], p[:, 2 * n + 2 * N:]
    xx = torch.nn.functional.pad(xbc, (0, 0, taps - 1, 0))
    xbc = torch.nn.functional.silu(t["conv.b"] + sum(xx[k:k + T] * t["conv"][:, k] for k in range(taps)))
    x, B, C = xbc[:, :n].reshape(T, H, P), xbc[:, n:n + N], xbc[:, n + N:]
    dt = torch.nn.functional.softplus(dt + t["dt_bias"])
    fall = -torch.exp(t["A_log"]) * dt                                      # log of each token's decay
    S, y = torch.zeros(H, P, N, dtype=h.dtype, device=h.device), torch.empty_like(x)
    for a in range(0, T, 128):
        s = slice(a, min(T, a + 128))
        f = fall[s].cumsum(0)                                               # [L, H]
        L = f.shape[0]
        tri = torch.ones(L, L, dtype=torch.bool, device=h.device).tril()
        wgt = torch.exp((f[:, None] - f[None, :]).masked_fill(~tri[..., None], float("-inf"))) * (C[s] @ B[s].t())[..., None] * dt[s][None]
        y[s] = torch.einsum("ijh,jhp->ihp", wgt, x[s]) + torch.exp(f)[..., None] * torch.einsum("in,hpn->ihp", C[s], S)
        S = torch.exp(f[-1])[:, None, None] * S + torch.einsum("jh,jhp,jn->hpn", torch.exp(f[-1] - f) * dt[s], x[s], B[s])
    y = (y + t["D"][:, None] * x).reshape(T, n) * torch.nn.functional.silu(z)
    y = _rms(y, eps) * t["norm"]
    return y @ t["o"].t(), {"conv": None, "ssm": S}
