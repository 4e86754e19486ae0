"""Performance cases: the work that users of this framework have it do, through its public entry points.

    gpt2_train       one optimizer step of GPT-2 small through ``trainer.train_step``, the path of ``bench.py`` and
                     ``scripts/train.py``; bf16 compute, fp32 master weights, tokens from pinned host memory
    qwen_prefill     a prompt of the Qwen3.5-style hybrid (the ``ns`` widths, one group of three Gated-DeltaNet layers and a
                     gated-attention layer) into a fresh cache, experts on the fused expert kernel
    qwen_decode      one token of every sequence on that model's CUDA-graph decode engine
    qwen_train       one optimizer step of the hybrid on ``TreeTrainEngine``
    deepseek_prefill prompts of the DeepSeek-V3 shape (full widths, one dense and one expert layer holding the 32 experts of
                     an eighth of the model) into the paged latent cache
    deepseek_decode  one token of every sequence over that cache on the CUDA-graph decode engine
    fp8_linear       forward and backward of a block-scaled FP8 projection at DeepSeek-V3 widths
    fovudra_prefill  a packed batch of prompts of mixed lengths on the step engine (mLSTM, lightning and windowed attention)
    fovudra_decode   one token of every sequence on the step engine
"""
from __future__ import annotations

import functools
import math

import torch
import torch.nn.functional as F

BF = torch.bfloat16
F64 = torch.float64


def listed():
    return [
        # the headline benchmark and the trainer's default micro-batch
        dict(name="gpt2_train_16x1024", path="gpt2_train", batch=16, tokens=1024),
        # short sequences, few of them: where launches and small grids count
        dict(name="gpt2_train_3x333", path="gpt2_train", batch=3, tokens=333),
        # a long prompt for one user, and a few short ragged ones
        dict(name="qwen_prefill_1x4096", path="qwen_prefill", batch=1, tokens=4096),
        dict(name="qwen_prefill_3x171", path="qwen_prefill", batch=3, tokens=171),
        # one user's next token, and a busy server's
        dict(name="qwen_decode_1_at_1000", path="qwen_decode", batch=1, tokens=1000),
        dict(name="qwen_decode_32_at_2048", path="qwen_decode", batch=32, tokens=2048),
        # a training step of the hybrid
        dict(name="qwen_train_1x2048", path="qwen_train", batch=1, tokens=2048),
        # latent attention: two prompts, and 64 sequences a step
        dict(name="deepseek_prefill_2x1024", path="deepseek_prefill", batch=2, tokens=1024),
        dict(name="deepseek_decode_64_at_2048", path="deepseek_decode", batch=64, tokens=2048),
        # the FP8 recipe on a shared expert's gate projection
        dict(name="fp8_linear_4096x7168x2048", path="fp8_linear", tokens=4096, wide=7168, out=2048),
        # a packed batch of ragged prompts, and eight users' next tokens
        dict(name="fovudra_prefill_4_to_1500", path="fovudra_prefill", batch=4, tokens=1500),
        dict(name="fovudra_decode_8_at_700", path="fovudra_decode", batch=8, tokens=700),
    ]


#: (in, out) of projections of the DeepSeek-V3 shape
FP8_SHAPES = [(7168, 1536), (1536, 24576), (512, 32768), (16384, 7168), (7168, 2048), (2048, 7168), (7168, 18432)]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.5)))))
    path = rng.choice(["gpt2_train", "qwen_prefill", "qwen_decode", "qwen_train", "deepseek_prefill", "deepseek_decode",
                       "fp8_linear", "fovudra_prefill", "fovudra_decode"])
    if path == "gpt2_train":
        return dict(path=path, batch=log(1, 15), tokens=log(64, 1024))
    if path == "qwen_prefill":
        b = log(1, 8)
        return dict(path=path, batch=b, tokens=log(16, 4000 // b))
    if path == "qwen_decode":
        return dict(path=path, batch=log(1, 32), tokens=log(64, 2000))
    if path == "qwen_train":
        b = log(1, 2)
        return dict(path=path, batch=b, tokens=log(400 // b, 2000 // b))
    if path == "deepseek_prefill":
        b = log(1, 4)
        return dict(path=path, batch=b, tokens=log(16, 2000 // b))
    if path == "deepseek_decode":
        return dict(path=path, batch=log(1, 63), tokens=log(64, 2000))
    if path == "fp8_linear":
        wide, out = rng.choice(FP8_SHAPES)
        return dict(path=path, tokens=128 * log(1, 16), wide=wide, out=out)
    if path == "fovudra_prefill":
        return dict(path=path, batch=log(1, 8), tokens=log(16, 1400))
    return dict(path=path, batch=log(1, 16), tokens=log(32, 1000))


# ---- what a program holds ------------------------------------------------------------------------------------------
#: tokens that a decode engine's cache has room for beyond the prompt; a sequence that used them up starts anew
ROOM = 4096


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _ids(seed, vocab, *shape):
    return torch.randint(0, vocab, shape, generator=_gen(seed + 7), device="cuda")


@functools.lru_cache(None)
def _communicator():
    import torch.distributed as dist
    from jax_gpt_b200.comm.symm import Communicator
    if not dist.is_initialized():
        dist.init_process_group("nccl", rank=0, world_size=1, store=dist.HashStore(), device_id=torch.device("cuda", 0))
    return Communicator(device=torch.device("cuda", 0))


@functools.lru_cache(None)
def _experts(d_model, inter, n, top):
    """A server's expert runtime: one for all its batches."""
    from jax_gpt_b200.parallel.expert_parallel import EPMoEInferenceRuntime
    return EPMoEInferenceRuntime(_communicator(), d_model, inter, n, top)


@functools.lru_cache(4)
def _experts_training(tokens, d_model, inter, n, top):
    from jax_gpt_b200.parallel.expert_parallel import EPMoERuntime, FusedEPMoE
    return EPMoERuntime(FusedEPMoE(_communicator(), tokens, d_model, inter, n, top, training=True))


def _tree(t, f, path=()):
    return {k: _tree(v, f, path + (k,)) for k, v in t.items()} if isinstance(t, dict) else f(path, t)


def _alike(bank, axis, own):
    """Experts as training leaves them: near-tied ones do nearly the same (one base and a part ``own``), so that a token whose
    rounding picks the other one comes out nearly the same. Experts without anything in common would turn rounding into noise."""
    base = bank.select(axis, 0).unsqueeze(axis).clone()
    bank.mul_(own).add_(base, alpha=(1 - own * own) ** 0.5)


# ---- GPT-2 ---------------------------------------------------------------------------------------------------------
def _gpt2_inputs(case, seed):
    from jax_gpt_b200.models.gpt2 import GPT, GPTConfig
    cfg = GPTConfig.from_model_type("gpt2")
    tok = torch.randint(0, cfg.vocab_size, (case["batch"], case["tokens"] + 1), generator=torch.Generator().manual_seed(seed),
                        dtype=torch.int32)
    return cfg, GPT(cfg, seed=seed), tok[:, :-1].contiguous().pin_memory(), tok[:, 1:].contiguous().pin_memory()


class Gpt2Train:
    @staticmethod
    def prepare(case, seed):
        from jax_gpt_b200.trainer.config import TrainConfig
        from jax_gpt_b200.trainer.optimizer import create_optimizer
        from jax_gpt_b200.trainer.train_state import create_train_state
        cfg, model, x, y = _gpt2_inputs(case, seed)
        tc = TrainConfig(micro_batch_size=case["batch"], seq_len=case["tokens"])
        return {"state": create_train_state(model, create_optimizer(model, tc), train_config=tc, device="cuda"), "batch": (x, y)}

    @staticmethod
    def run(s):
        from jax_gpt_b200.trainer.train_step import train_step
        st, metrics = train_step(s["state"], s["batch"])
        return {"loss": metrics["loss"], "grad_norm": metrics["grad_norm"], "params": st.model.params, "mu": st.opt_state.mu}

    @staticmethod
    def work(case):
        n, d, V, L = case["batch"] * case["tokens"], 768, 50257, 12
        mat = L * 12 * d * d
        flops = 6.0 * n * (mat + V * d) + 3.0 * 2 * L * case["batch"] * case["tokens"] ** 2 * d
        # the optimizer: gradient in; master weights, two moments and the bf16 copy in and out (the untied head matrix too)
        p = mat + 2 * V * d + 1024 * d
        return {"bytes": p * (4 + 8 + 16 + 2.0) + 2 * 2.0 * (mat + V * d) + 8.0 * n, "flops": flops}

    @staticmethod
    def exact(case, seed):
        cfg, model, x, y = _gpt2_inputs(case, seed)
        init = {k: v.cuda() for k, v in model.params.items()}
        p = {k: v.to(BF).to(F64).requires_grad_(True) for k, v in init.items()}
        B, T, L, H = case["batch"], case["tokens"], cfg.n_layers, cfg.n_head
        x, y = x.cuda().long(), y.cuda().long()
        ln = lambda h, n, l=None: F.layer_norm(h, h.shape[-1:], *[p[f"{n}.layer_norm.{w}"] if l is None else p[f"{n}.layer_norm.{w}"][l]
                                                                  for w in ("scale", "bias")])
        lin = lambda h, n, l: h @ p[n + ".kernel"][l] + p[n + ".bias"][l]
        total, per = 0.0, max(1, 2048 // T)
        for b in range(0, B, per):
            h = p["wte.embedding"][x[b:b + per]] + p["wpe.embedding"][:T]
            n = h.shape[0]
            for l in range(L):
                q, k, v = [t.reshape(n, T, H, -1).transpose(1, 2) for t in lin(ln(h, "h.ln_1", l), "h.attn.c_attn", l).chunk(3, -1)]
                a = (q @ k.transpose(-1, -2) * q.shape[-1] ** -0.5).masked_fill(_after(T), -math.inf).softmax(-1) @ v
                h = h + lin(a.transpose(1, 2).reshape(n, T, -1), "h.attn.c_proj", l)
                h = h + lin(F.gelu(lin(ln(h, "h.ln_2", l), "h.mlp.c_fc", l), approximate="tanh"), "h.mlp.c_proj", l)
            logits = ln(h, "ln_f") @ p["wte.embedding"].t()
            loss = F.cross_entropy(logits.reshape(n * T, -1), y[b:b + per].reshape(-1), reduction="sum") / (B * T)
            loss.backward()
            total += float(loss)
            del logits, loss, h, a, q, k, v
        grads = {k: v.grad if v.grad is not None else torch.zeros_like(v) for k, v in p.items()}
        norm = sum(g.square().sum() for g in grads.values()).sqrt()
        clip = 0.1 * min(1.0, 1.0 / (float(norm) + 1e-6))
        # the schedule's first rate is zero: the first step leaves the weights where they are
        return {"loss": torch.tensor([total], dtype=F64), "grad_norm": norm.reshape(1), "params": {k: v.to(F64) for k, v in init.items()},
                "mu": {k: g * clip for k, g in grads.items()}}


@functools.lru_cache(8)
def _after(T):
    return torch.ones(T, T, device="cuda", dtype=torch.bool).triu(1)


# ---- Qwen3.5-style hybrid ------------------------------------------------------------------------------------------
def _qwen_config(train=False):
    from jax_gpt_b200.models.qwen35.config import Qwen35Config
    c = Qwen35Config.ns().replace(n_layers=4)
    return c.replace(n_routed_experts=64, vocab_size=8192) if train else c


def _qwen_params(case, seed):
    from jax_gpt_b200.models.qwen35 import init_params
    c = _qwen_config(case["path"] == "qwen_train")
    params = init_params(c, seed, dtype=BF, device="cuda", on_device=True)
    train = case["path"] == "qwen_train"
    for layers in params["groups"].values():
        layers["moe"]["gate_weight"].mul_(4.0 if train else 3.0)      # a trained router's choices are clear ones
        for n in ("gate_proj", "up_proj", "down_proj"):
            _alike(layers["moe"][n], -3, 0.3 if train else 0.1)
    return c, params


def _qwen_weights(c):
    """Parameters outside the experts of one group, parameters of an expert."""
    D, qk, v = c.d_model, c.delta_key_dim, c.delta_value_dim
    q, kv = c.gqa_n_q_heads * c.gqa_head_dim, c.gqa_n_kv_heads * c.gqa_head_dim
    moe = D * c.n_routed_experts + 3 * D * c.shared_expert_intermediate_size
    return 3 * D * (2 * qk + 2 * v + 2 * c.delta_n_v_heads + v) + D * (3 * q + 2 * kv) + 4 * moe, 3 * D * c.moe_intermediate_size


def _touched(n, top, tokens):
    """Experts that ``tokens`` tokens reach when each picks ``top`` of ``n`` at random."""
    return n * (1 - (1 - top / n) ** tokens)


def _qwen_work(c, batch, tokens, context, last_only):
    n = batch * tokens
    dense, expert = _qwen_weights(c)
    state = 3 * batch * c.delta_n_v_heads * 128 * 128
    kv = 2 * batch * c.gqa_n_kv_heads * c.gqa_head_dim
    flops = 2.0 * n * (dense + 4 * c.n_experts_per_token * expert + c.d_model * c.vocab_size)
    flops += 3 * n * c.delta_n_v_heads * 6.0 * 128 * 128
    flops += 4.0 * n * c.gqa_n_q_heads * c.gqa_head_dim * (context + (tokens + 1) / 2)
    data = 2.0 * (dense + 4 * _touched(c.n_routed_experts, c.n_experts_per_token, n) * expert + c.d_model * c.vocab_size)
    data += 2.0 * n * c.vocab_size + 2.0 * kv * (context + tokens) + (8.0 if last_only else 2.0) * state
    return {"bytes": data, "flops": flops}


class QwenPrefill:
    @staticmethod
    def prepare(case, seed):
        c, params = _qwen_params(case, seed)
        return {"c": c, "params": params, "tokens": _ids(seed, c.vocab_size, case["batch"], case["tokens"]),
                "ep": _experts(c.d_model, c.moe_intermediate_size, c.n_routed_experts, c.n_experts_per_token)}

    @staticmethod
    @torch.no_grad()
    def run(s):
        from jax_gpt_b200.models.qwen35 import forward, init_cache
        B, T = s["tokens"].shape
        cache = init_cache(s["c"], B, T + 64, dtype=BF, device="cuda")
        logits, cache = forward(s["params"], s["tokens"], s["c"], cache=cache, ep_group=s["ep"])
        return {"logits": logits, "state": cache.delta_M, "conv": cache.delta_conv, "k": cache.gqa_k, "v": cache.gqa_v}

    @staticmethod
    def work(case):
        return _qwen_work(_qwen_config(), case["batch"], case["tokens"], 0, False)

    @staticmethod
    @torch.no_grad()
    def exact(case, seed):
        c, params = _qwen_params(case, seed)
        logits, out = _qwen64(params, c, _ids(seed, c.vocab_size, case["batch"], case["tokens"]))
        return {"logits": logits, "state": out["M"], "conv": out["conv"], "k": F.pad(out["k"], (0, 0, 0, 64)), "v": F.pad(out["v"], (0, 0, 0, 64))}


class QwenDecode:
    @staticmethod
    def inputs(case, seed):
        """A cache as a prompt leaves it: unit-scale keys, and values, states and windows of the size that the projections give."""
        from jax_gpt_b200.models.qwen35 import init_cache
        c, params = _qwen_params(case, seed)
        cache = init_cache(c, case["batch"], case["tokens"] + ROOM, dtype=BF, device="cuda")
        g = _gen(seed + 3)
        cache.delta_M.normal_(0.0, 0.1, generator=g)
        cache.delta_conv.normal_(0.0, 0.9, generator=g)
        for t, std in ((cache.gqa_k, 1.0), (cache.gqa_v, 0.9)):
            t[:, :, :, :case["tokens"]].normal_(0.0, std, generator=g)
        cache.pos = case["tokens"]
        return c, params, cache, _ids(seed, c.vocab_size, 64, case["batch"])

    @staticmethod
    def engine(s):
        from jax_gpt_b200.models.qwen35.decode_engine import Qwen35DecodeEngine
        ep = _experts(s["c"].d_model, s["c"].moe_intermediate_size, s["c"].n_routed_experts, s["c"].n_experts_per_token)
        s["engine"], s["done"] = Qwen35DecodeEngine(s["params"], s["c"], s["cache"], ep=ep), 0

    @staticmethod
    def prepare(case, seed):
        c, params, cache, tokens = QwenDecode.inputs(case, seed)
        s = {"c": c, "params": params, "cache": cache, "tokens": tokens}
        QwenDecode.engine(s)
        return s

    @staticmethod
    def run(s):
        if s["done"] == ROOM:
            QwenDecode.engine(s)
        e = s["engine"]
        e.step(s["tokens"][s["done"] % 64])
        s["done"] += 1
        return {"logits": e.logits, "state": e.M, "conv": e.conv}

    @staticmethod
    def work(case):
        return _qwen_work(_qwen_config(), case["batch"], 1, case["tokens"], True)

    @staticmethod
    @torch.no_grad()
    def exact(case, seed):
        c, params, cache, tokens = QwenDecode.inputs(case, seed)
        logits, out = _qwen64(params, c, tokens[0][:, None], cache)
        return {"logits": logits[:, 0], "state": out["M"], "conv": out["conv"]}


class QwenTrain:
    @staticmethod
    def prepare(case, seed):
        from jax_gpt_b200.parallel.expert_parallel import is_expert_leaf
        from jax_gpt_b200.trainer.lm_loss import qwen35_loss_fn, qwen35_unstack
        from jax_gpt_b200.trainer.tree_engine import TreeTrainEngine
        c, params = _qwen_params(case, seed)
        ep = _experts_training(case["batch"] * case["tokens"], c.d_model, c.moe_intermediate_size, c.n_routed_experts, c.n_experts_per_token)
        engine = TreeTrainEngine(params, qwen35_loss_fn(c, ep), device="cuda", local=is_expert_leaf, unstack=qwen35_unstack,
                                 lr=6e-4, min_lr=6e-5, warmup_steps=2000, lr_decay_steps=600000, consume_params=True)
        tok = _ids(seed, c.vocab_size, case["batch"], case["tokens"] + 1)
        return {"engine": engine, "x": tok[:, :-1].contiguous(), "y": tok[:, 1:].contiguous(), "mu": engine.dense_state()[1],
                "experts": engine.local_state()[1]}

    @staticmethod
    def run(s):
        out = s["engine"].train_step(s["x"], s["y"])
        return {"loss": out["loss"], "norm_sq": out["grad_norm_sq"], "mu": s["mu"], "experts": s["experts"]}

    @staticmethod
    def work(case):
        c = _qwen_config(True)
        w = _qwen_work(c, case["batch"], case["tokens"], 0, False)
        dense, expert = _qwen_weights(c)
        p = dense + 4 * c.n_routed_experts * expert + 2 * c.d_model * c.vocab_size
        return {"bytes": 30.0 * p + 4.0 * p, "flops": 3.0 * w["flops"]}

    @staticmethod
    def exact(case, seed):
        c, params = _qwen_params(case, seed)
        params = _tree(params, lambda path, t: t.to(F64).requires_grad_(True))
        tok = _ids(seed, c.vocab_size, case["batch"], case["tokens"] + 1)
        logits, _ = _qwen64(params, c, tok[:, :-1])
        loss = F.cross_entropy(logits.reshape(-1, c.vocab_size), tok[:, 1:].reshape(-1))
        del logits
        loss.backward()
        grads = _tree(params, lambda path, t: t.grad)
        sq = []
        _tree(grads, lambda path, t: sq.append(t.square().sum()))
        sq = sum(sq)
        clip = 0.1 * min(1.0, 1.0 / (float(sq.sqrt()) + 1e-6))
        routed = lambda path: "moe" in path and path[-1] in ("gate_proj", "up_proj", "down_proj")
        pick = lambda t, want, path=(): {k: pick(v, want, path + (k,)) if isinstance(v, dict) else v * clip for k, v in t.items()
                                         if isinstance(v, dict) or routed(path + (k,)) == want}
        return {"loss": loss.detach(), "norm_sq": sq.reshape(1), "mu": pick(grads, False), "experts": pick(grads, True)}


def _rms(x, w, eps=1e-6):
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * w


def _turn(x, first, dims, theta):
    """x (B, T, H, d): the first ``dims`` features, i with i + dims / 2, turn by the angles of positions ``first`` on."""
    inv = theta ** (-torch.arange(0, dims, 2, device=x.device, dtype=F64) / dims)
    ang = (first + torch.arange(x.shape[1], device=x.device, dtype=F64))[:, None, None] * inv
    u, v = x[..., :dims // 2], x[..., dims // 2:dims]
    return torch.cat([u * ang.cos() - v * ang.sin(), v * ang.cos() + u * ang.sin(), x[..., dims:]], -1)


def _by_expert(x, w, idx, expert):
    """sum_j w[:, j] expert(idx[:, j], x), the rows of an expert together."""
    flat, k = idx.reshape(-1), idx.shape[1]
    order = flat.argsort(stable=True)
    out, at = torch.zeros_like(x), 0
    for e, n in enumerate(flat.bincount().tolist()):
        if n:
            rows = order[at:at + n]
            out = out.index_add(0, rows // k, expert(e, x[rows // k]) * w.reshape(-1)[rows][:, None])
        at += n
    return out


def _swiglu(x, gate, up, down):
    return (F.silu(x @ gate.to(F64)) * (x @ up.to(F64))) @ down.to(F64)


def _qwen_moe64(x, p, at, c):
    w = lambda n: p[n][at].to(F64)
    B, T, D = x.shape
    x = x.reshape(-1, D)
    prob, idx = (x @ w("gate_weight")).softmax(-1).topk(c.n_experts_per_token, -1)
    prob = prob / prob.sum(-1, keepdim=True)
    bank = [p[n][at] for n in ("gate_proj", "up_proj", "down_proj")]
    out = _by_expert(x, prob, idx, lambda e, rows: _swiglu(rows, *[t[e] for t in bank]))
    shared = _swiglu(x, w("shared_gate_proj"), w("shared_up_proj"), w("shared_down_proj"))
    return (out + shared * torch.sigmoid(x @ w("shared_expert_gate_weight"))).reshape(B, T, D)


def _delta64(x, p, at, c, M, conv):
    w = lambda n: p[n][at].to(F64)
    B, T, _ = x.shape
    Hk, Hv, d, C = c.delta_n_qk_heads, c.delta_n_v_heads, 128, 64
    raw = torch.cat([torch.zeros(B, 4, c.delta_conv_dim, device=x.device, dtype=F64) if conv is None else conv.to(F64).transpose(1, 2),
                     x @ w("in_proj_qkv")], 1)
    cw = w("conv_weight")
    y = F.silu(sum(raw[:, i + 1:i + 1 + T] * cw[:, i] for i in range(4)))
    unit = lambda t: t * torch.rsqrt(t.square().sum(-1, keepdim=True) + 1e-6)
    q, k, v = y.split([Hk * d, Hk * d, Hv * d], -1)
    q, k = [unit(t.reshape(B, T, Hk, d)).repeat_interleave(Hv // Hk, 2).transpose(1, 2) for t in (q, k)]
    q, v = q * d ** -0.5, v.reshape(B, T, Hv, d).transpose(1, 2)
    beta = torch.sigmoid(x @ w("in_proj_b")).transpose(1, 2)
    g = -(w("A_log").exp() * F.softplus(x @ w("in_proj_a") + w("dt_bias"))).transpose(1, 2)
    S = torch.zeros(B, Hv, d, d, device=x.device, dtype=F64) if M is None else M.to(F64)
    outs = []
    for t in range(0, T, C):
        qc, kc, vc, bc, G = q[:, :, t:t + C], k[:, :, t:t + C], v[:, :, t:t + C], beta[:, :, t:t + C, None], g[:, :, t:t + C].cumsum(-1)
        n = G.shape[-1]
        decay = (G[..., :, None] - G[..., None, :]).masked_fill(_after(n), -math.inf).exp()
        A = (bc * kc) @ kc.transpose(-1, -2) * decay * (1 - torch.eye(n, device=x.device, dtype=F64))
        E = G[..., None].exp()
        u = torch.linalg.solve_triangular(A + torch.eye(n, device=x.device, dtype=F64), bc * (vc - E * (kc @ S)), upper=False)
        outs.append(E * (qc @ S) + (qc @ kc.transpose(-1, -2) * decay) @ u)
        S = E[:, :, -1:] * S + (kc * (G[..., -1:] - G)[..., None].exp()).transpose(-1, -2) @ u
    o = torch.cat(outs, 2).transpose(1, 2)
    z = (x @ w("in_proj_z")).reshape(B, T, Hv, d)
    return (_rms(o, w("norm_weight")) * F.silu(z)).reshape(B, T, -1) @ w("out_proj"), S, raw[:, -4:].transpose(1, 2)


def _gated_attention64(x, p, at, c, past):
    w = lambda n: p[n][at].to(F64)
    B, T, _ = x.shape
    H, G, d = c.gqa_n_q_heads, c.gqa_n_kv_heads, c.gqa_head_dim
    q, gate = (x @ w("q_proj")).reshape(B, T, H, 2 * d).chunk(2, -1)
    k, v = [(x @ w(n)).reshape(B, T, G, d) for n in ("k_proj", "v_proj")]
    first = 0 if past is None else past.pos
    q = _turn(_rms(q, 1 + w("q_norm")), first, c.gqa_rope_dim, c.gqa_rope_theta).transpose(1, 2)
    k, v = _turn(_rms(k, 1 + w("k_norm")), first, c.gqa_rope_dim, c.gqa_rope_theta).transpose(1, 2), v.transpose(1, 2)
    if past is not None:
        k, v = [torch.cat([t[at][:, :, :first].to(F64), n], 2) for t, n in ((past.gqa_k, k), (past.gqa_v, v))]
    outs = []
    for h in range(H):
        s = q[:, h] @ k[:, h * G // H].transpose(-1, -2) * d ** -0.5
        outs.append((s.masked_fill(_after(T), -math.inf) if T > 1 else s).softmax(-1) @ v[:, h * G // H])
    o = torch.stack(outs, 2) * torch.sigmoid(gate)
    return o.reshape(B, T, -1) @ w("o_proj"), k, v


def _qwen64(params, c, tokens, past=None):
    """Logits and what the cache holds afterwards, in 64 bits."""
    eps = c.rms_norm_eps
    x = params["embed"][tokens].to(F64)
    out = {"M": [], "conv": [], "k": [], "v": []}
    for gi in range(c.n_groups):
        lp = params["groups"]["delta_layers"]
        Ms, convs = [], []
        for i in range(c.n_delta_per_group):
            at = (gi, i)
            a, M, conv = _delta64(_rms(x, 1 + lp["attn_norm"][at].to(F64), eps), lp["attn"], at, c, None if past is None else past.delta_M[at],
                                  None if past is None else past.delta_conv[at])
            x = x + a
            x = x + _qwen_moe64(_rms(x, 1 + lp["moe_norm"][at].to(F64), eps), lp["moe"], at, c)
            Ms.append(M)
            convs.append(conv)
        lp = params["groups"]["gqa_layer"]
        a, k, v = _gated_attention64(_rms(x, 1 + lp["attn_norm"][gi].to(F64), eps), lp["attn"], gi, c, past)
        x = x + a
        x = x + _qwen_moe64(_rms(x, 1 + lp["moe_norm"][gi].to(F64), eps), lp["moe"], gi, c)
        for n, t in (("M", torch.stack(Ms)), ("conv", torch.stack(convs)), ("k", k), ("v", v)):
            out[n].append(t)
    return _rms(x, 1 + params["final_norm"].to(F64), eps) @ params["lm_head"].to(F64), {n: torch.stack(t) for n, t in out.items()}


# ---- DeepSeek-V3 shape ---------------------------------------------------------------------------------------------
def _deepseek_config():
    from jax_gpt_b200.models.deepseek_v3 import DeepSeekV3Config
    return DeepSeekV3Config.eight_layer().replace(n_layers=2, n_routed_experts=32, max_position_embeddings=8192)


def _deepseek_params(seed):
    from jax_gpt_b200.models.deepseek_v3 import init_params
    c = _deepseek_config()
    params = init_params(c, seed, dtype=BF, device="cuda", on_device=True)
    for n in ("gate_proj", "up_proj", "down_proj"):
        _alike(params["moe_layers"]["moe"][n], -3, 0.1)
    return c, params


def _deepseek_cache(c, batch, room):
    from jax_gpt_b200.models.deepseek_v3 import make_cache
    per = (room + c.page_size - 1) // c.page_size
    return make_cache(c, batch * per, batch, per, BF, "cuda")


def _deepseek_work(c, batch, tokens, context):
    n, D, H = batch * tokens, c.d_model, c.n_heads
    attn = D * (c.q_lora_rank + c.latent_dim) + c.q_lora_rank * H * c.qk_head_dim + c.kv_lora_rank * H * 256 + H * 128 * D
    dense = 2 * attn + 3 * D * c.dense_intermediate_size + D * c.n_routed_experts + 3 * D * c.moe_intermediate_size + D * c.vocab_size
    expert = 3 * D * c.moe_intermediate_size
    flops = 2.0 * n * (dense + c.n_experts_per_token * expert)
    # a prompt attends with decompressed heads, a single token over the latents
    flops += 2 * 2.0 * n * H * ((c.qk_head_dim + 128) * (tokens + 1) / 2 if tokens > 1 else (c.latent_dim + 512) * context)
    data = 2.0 * (dense + _touched(c.n_routed_experts, c.n_experts_per_token, n) * expert) + 2.0 * n * c.vocab_size
    return {"bytes": data + 2 * 2.0 * batch * (context + tokens) * c.latent_dim, "flops": flops}


class DeepseekPrefill:
    @staticmethod
    def prepare(case, seed):
        c, params = _deepseek_params(seed)
        return {"c": c, "params": params, "cache": _deepseek_cache(c, case["batch"], case["tokens"] + 64),
                "tokens": _ids(seed, c.vocab_size, case["batch"], case["tokens"]),
                "ep": _experts(c.d_model, c.moe_intermediate_size, c.n_routed_experts, c.n_experts_per_token)}

    @staticmethod
    @torch.no_grad()
    def run(s):
        from jax_gpt_b200.models.deepseek_v3 import forward
        ids = list(range(s["tokens"].shape[0]))
        for i in ids:                                    # the sequences that held the pages before are done
            if s["cache"].length(i):
                s["cache"].release(i)
        logits = forward(s["params"], s["tokens"], s["c"], s["cache"], ids, ep=s["ep"])
        return {"logits": logits, "latents": s["cache"].pool}

    @staticmethod
    def work(case):
        return _deepseek_work(_deepseek_config(), case["batch"], case["tokens"], 0)

    @staticmethod
    @torch.no_grad()
    def exact(case, seed):
        c, params = _deepseek_params(seed)
        return {"logits": _deepseek64(params, c, _ids(seed, c.vocab_size, case["batch"], case["tokens"])), "latents": None}


class DeepseekDecode:
    @staticmethod
    def latents(case, seed, layer):
        """Cached rows as a prompt leaves them: a normalised latent and a rotated key of the size that the projection gives."""
        c = _deepseek_config()
        rows = torch.randn(case["batch"], case["tokens"], c.latent_dim, generator=_gen(seed + 11 + layer), device="cuda", dtype=BF)
        rows[..., c.kv_lora_rank:] *= 0.02 * c.d_model ** 0.5
        return rows

    @staticmethod
    def fill(s):
        cache, ids = s["cache"], list(range(s["case"]["batch"]))
        for i in ids:
            if cache.length(i):
                cache.release(i)
        for layer in range(s["c"].n_layers):
            cache.append(layer, ids, DeepseekDecode.latents(s["case"], s["seed"], layer))
        cache.commit(ids, s["case"]["tokens"])
        s["done"] = 0

    @staticmethod
    def prepare(case, seed):
        from jax_gpt_b200.models.deepseek_v3.decode_engine import DeepSeekV3DecodeEngine
        c, params = _deepseek_params(seed)
        s = {"case": case, "seed": seed, "c": c, "cache": _deepseek_cache(c, case["batch"], case["tokens"] + ROOM + 64),
             "tokens": _ids(seed, c.vocab_size, 64, case["batch"])}
        DeepseekDecode.fill(s)
        s["engine"] = DeepSeekV3DecodeEngine(params, c, s["cache"], list(range(case["batch"])), max_len=case["tokens"] + ROOM,
                                             ep=_experts(c.d_model, c.moe_intermediate_size, c.n_routed_experts, c.n_experts_per_token))
        return s

    @staticmethod
    def run(s):
        if s["done"] == ROOM:
            DeepseekDecode.fill(s)
        e = s["engine"]
        e.step(s["tokens"][s["done"] % 64])
        s["done"] += 1
        return {"logits": e.logits}

    @staticmethod
    def work(case):
        return _deepseek_work(_deepseek_config(), case["batch"], 1, case["tokens"])

    @staticmethod
    @torch.no_grad()
    def exact(case, seed):
        c, params = _deepseek_params(seed)
        past = [DeepseekDecode.latents(case, seed, l) for l in range(c.n_layers)]
        return {"logits": _deepseek64(params, c, _ids(seed, c.vocab_size, 64, case["batch"])[0][:, None], past)[:, 0]}


def _latent_attention64(x, p, at, c, past):
    w = lambda n: p[n][at].to(F64)
    B, T, _ = x.shape
    H, dn, dr, R, eps = c.n_heads, c.qk_nope_head_dim, c.qk_rope_head_dim, c.kv_lora_rank, c.rms_norm_eps
    first = 0 if past is None else past.shape[1]
    q = (_rms(x @ w("q_a_proj"), w("q_a_norm"), eps) @ w("q_b_proj")).reshape(B, T, H, dn + dr)
    kv = x @ w("kv_a_proj_with_mqa")
    lat = _rms(kv[..., :R], w("kv_a_norm"), eps)
    qr, kr = _turn(q[..., dn:], first, dr, c.rope_theta), _turn(kv[..., None, R:], first, dr, c.rope_theta)[:, :, 0]
    if past is not None:
        lat, kr = torch.cat([past[..., :R].to(F64), lat], 1), torch.cat([past[..., R:].to(F64), kr], 1)
    up = w("kv_b_proj").reshape(R, H, -1)
    outs = []
    for h in range(H):
        s = (q[:, :, h, :dn] @ up[:, h, :dn].t()) @ lat.transpose(1, 2) + qr[:, :, h] @ kr.transpose(1, 2)
        s = s * c.softmax_scale
        outs.append(((s.masked_fill(_after(T), -math.inf) if T > 1 else s).softmax(-1) @ lat) @ up[:, h, dn:])
    return torch.cat(outs, -1) @ w("o_proj")


def _deepseek_moe64(x, p, at, c):
    w = lambda n: p[n][at].to(F64)
    B, T, D = x.shape
    x = x.reshape(-1, D)
    score = torch.sigmoid(x @ w("gate_weight"))
    groups = (score + w("e_score_correction_bias")).reshape(x.shape[0], c.n_group, -1)
    keep = torch.zeros_like(groups[..., 0]).scatter(1, groups.topk(2, -1).values.sum(-1).topk(c.topk_group, -1).indices, 1.0)
    idx = groups.masked_fill(keep[..., None] == 0, 0.0).reshape(x.shape[0], -1).topk(c.n_experts_per_token, -1).indices
    prob = score.gather(1, idx)
    prob = prob / (prob.sum(-1, keepdim=True) + 1e-20) * c.routed_scaling_factor
    bank = [p[n][at] for n in ("gate_proj", "up_proj", "down_proj")]
    out = _by_expert(x, prob, idx, lambda e, rows: _swiglu(rows, *[t[e] for t in bank]))
    return (out + _swiglu(x, w("shared_gate_proj"), w("shared_up_proj"), w("shared_down_proj"))).reshape(B, T, D)


def _deepseek64(params, c, tokens, past=None):
    x, eps = params["embed"][tokens].to(F64), c.rms_norm_eps
    for layer, (kind, at) in enumerate((("dense_layers", 0), ("moe_layers", 0))):
        p = params[kind]
        x = x + _latent_attention64(_rms(x, p["attn_norm"][at].to(F64), eps), p["attn"], at, c, None if past is None else past[layer])
        h = _rms(x, p["ffn_norm"][at].to(F64), eps)
        x = x + (_deepseek_moe64(h, p["moe"], at, c) if "moe" in p else _swiglu(h, *[p["mlp"][n][at] for n in ("gate_proj", "up_proj", "down_proj")]))
    return _rms(x, params["final_norm"].to(F64), eps) @ params["lm_head"].to(F64)


# ---- block-scaled FP8 projection -----------------------------------------------------------------------------------
class Fp8Linear:
    @staticmethod
    def prepare(case, seed):
        g = _gen(seed)
        n = lambda std, *s: torch.randn(*s, generator=g, device="cuda", dtype=BF).mul_(std)
        # a normalised activation, initial weights, the gradient of a mean loss
        return {"x": n(1.0, case["tokens"], case["wide"]).requires_grad_(True), "w": n(0.02, case["wide"], case["out"]).requires_grad_(True),
                "dy": n(1e-3, case["tokens"], case["out"])}

    @staticmethod
    def run(s):
        from jax_gpt_b200.ops.fp8_linear import fp8_linear
        y = fp8_linear(s["x"], s["w"])
        dx, dw = torch.autograd.grad(y, (s["x"], s["w"]), s["dy"])
        return {"y": y, "dx": dx, "dw": dw}

    @staticmethod
    def work(case):
        m, k, n = case["tokens"], case["wide"], case["out"]
        return {"bytes": 2.0 * 2 * (m * k + k * n + m * n), "flops": 6.0 * m * k * n}

    @staticmethod
    @torch.no_grad()
    def exact(case, seed):
        s = {k: t.detach().to(F64) for k, t in Fp8Linear.prepare(case, seed).items()}
        return {"y": s["x"] @ s["w"], "dx": s["dy"] @ s["w"].t(), "dw": s["x"].t() @ s["dy"]}


# ---- a family on the step engine -----------------------------------------------------------------------------------
def _fovudra_inputs(case, seed):
    """Prompts of mixed lengths, the longest ``tokens``: b, b - 1 .. 1 parts of b, an odd token off."""
    from jax_gpt_b200.models.fovudra import FovudraConfig, init_params
    c, b = FovudraConfig.serving(), case["batch"]
    ids = _ids(seed, c.vocab_size, b, case["tokens"] + 64).tolist()
    params = init_params(c, seed, dtype=BF, device="cuda", on_device=True)
    for layer in params["layers"]:
        for n in ("gate_up", "down"):
            _alike(layer["mlp"][n], 0, 0.1)
    return c, params, [t[:n] for t, n in zip(ids, _lengths(case))], [t[-64:] for t in ids]


def _lengths(case):
    b = case["batch"]
    return [max(1, case["tokens"] * (b - i) // b - (i % 2)) for i in range(b)]


def _fovudra_engine(case, c, params, room):
    from jax_gpt_b200.models.fovudra import FovudraEngine, make_cache
    per = (case["tokens"] + room + c.page_size - 1) // c.page_size
    return FovudraEngine(params, c, make_cache(c, case["batch"] * per, case["batch"], per, BF, "cuda"))


def _fovudra_work(lengths, contexts):
    from jax_gpt_b200.models.fovudra import FovudraConfig
    c = FovudraConfig.serving()
    D, n, E, top, ff, sff = c.width, sum(lengths), 64, 6, 1024, 128
    dense = 2 * (D * 18 * 128 + D * D) + 6 * 5 * D * D + 3 * 2 * 16 * D + 8 * (D * E + 3 * D * sff)
    flops = 2.0 * n * (dense + 8 * top * 3 * D * ff) + 2.0 * len(lengths) * D * c.vocab_size + 6 * n * 16 * 4.0 * 128 * 128
    seen = sum(min(k + t / 2, 1024 + 64) * t for t, k in zip(lengths, contexts))
    flops += 2 * 4.0 * 16 * 128 * seen
    data = 2.0 * (dense + 8 * _touched(E, top, n) * 3 * D * ff + D * c.vocab_size)
    data += 4.0 * len(lengths) * c.vocab_size + 2 * 2.0 * 512 * sum(min(k, 1088) + t for t, k in zip(lengths, contexts))
    return {"bytes": data + 6 * 4.0 * 16 * 128 * 128 * sum(2 if k else 1 for k in contexts), "flops": flops}


class FovudraPrefill:
    @staticmethod
    def prepare(case, seed):
        c, params, prompts, _ = _fovudra_inputs(case, seed)
        return {"engine": _fovudra_engine(case, c, params, 64), "prompts": prompts}

    @staticmethod
    def run(s):
        e, ids = s["engine"], list(range(len(s["prompts"])))
        for i in ids:
            if i in e.cache:
                e.release(i)
        return {"logits": e.step(ids, s["prompts"]), "states": e.cache.states}

    @staticmethod
    def work(case):
        return _fovudra_work(_lengths(case), [0] * case["batch"])

    @staticmethod
    @torch.no_grad()
    def exact(case, seed):
        c, params, prompts, _ = _fovudra_inputs(case, seed)
        return {"logits": _fovudra64(params, c, prompts), "states": None}


class FovudraDecode:
    @staticmethod
    def fill(s):
        e, ids = s["engine"], s["ids"]
        for i in ids:
            if i in e.cache:
                e.release(i)
        e.step(ids, s["prompts"])
        s["done"] = 0

    @staticmethod
    def prepare(case, seed):
        c, params, prompts, following = _fovudra_inputs(case, seed)
        s = {"engine": _fovudra_engine(case, c, params, ROOM), "prompts": prompts, "ids": list(range(case["batch"])),
             "following": torch.tensor(following, dtype=torch.int32, device="cuda").t().contiguous()}
        FovudraDecode.fill(s)
        return s

    @staticmethod
    def run(s):
        if s["done"] == ROOM:
            FovudraDecode.fill(s)
        logits = s["engine"].decode(s["ids"], s["following"][s["done"] % 64])
        s["done"] += 1
        return {"logits": logits, "states": s["engine"].cache.states}

    @staticmethod
    def work(case):
        return _fovudra_work([1] * case["batch"], _lengths(case))

    @staticmethod
    @torch.no_grad()
    def exact(case, seed):
        c, params, prompts, following = _fovudra_inputs(case, seed)
        return {"logits": _fovudra64(params, c, [p + f[:1] for p, f in zip(prompts, following)]), "states": None}


def _fovudra64(params, c, prompts):
    """Logits after the last token of every prompt, in 64 bits: prompts padded at their end to one length."""
    n = torch.tensor([len(p) for p in prompts], device="cuda")
    T, B, eps = int(n.max()), len(prompts), c.norm_eps
    tok = torch.tensor([p + [0] * (T - len(p)) for p in prompts], device="cuda")
    w64 = lambda t: t.to(F64)
    lin = lambda x, w: x @ w64(w).t()
    x = _rms(w64(params["embed"])[tok], w64(params["embed_norm"]), eps)
    for layer, lp in zip(c.layers, params["layers"]):
        m, p, h = layer.mixer, lp["mix"], _rms(x, w64(lp["norm1"]), eps)
        kind = type(m).__name__
        if kind == "WindowAttention":
            qk = (lin(h, p["qk"]) + w64(p["qk_b"])).reshape(B, T, -1, m.dim)
            v = qk[:, :, m.heads:]
            qk = _rms(_banded_turn(qk, m.rot), 1.0, eps)
            at = torch.arange(T, device="cuda")
            hidden = (at[None] > at[:, None]) | ((at[:, None] - at[None] >= m.window) & (at[None] >= m.keep_first))
            outs = []
            for i in range(m.heads):
                g = i * m.kv_heads // m.heads
                s = qk[:, :, i] @ qk[:, :, m.heads + g].transpose(1, 2) * m.scale
                outs.append(s.masked_fill(hidden, -math.inf).softmax(-1) @ v[:, :, g])
            y = lin(torch.cat(outs, -1), p["o"])
        else:
            H, d, P = m.heads, m.dim, m.vdim
            z = lin(h, p["in"])
            q, k, v, g = z[..., :2 * H * (d + P)].split([H * d, H * d, H * P, H * P], -1)
            if kind == "MLstm":
                raw = z[..., -2 * H:] + w64(p["gate_b"])
                i, f = (m.gate_cap * torch.tanh(raw / m.gate_cap)).chunk(2, -1)
                f = F.logsigmoid(f)
                q = q * d ** -0.5
            else:
                q, k, v = F.silu(q), F.silu(k), F.silu(v)
            q, k, v = [t.reshape(B, T, H, -1) for t in (q, k, v)]
            S = torch.zeros(B, H, d, P, device="cuda", dtype=F64)
            nrm, top = torch.zeros(B, H, d, device="cuda", dtype=F64), torch.zeros(B, H, device="cuda", dtype=F64)
            o = torch.empty(B, T, H, P, device="cuda", dtype=F64)
            for t in range(T):
                if kind == "MLstm":
                    new = torch.maximum(f[:, t] + top, i[:, t])
                    keep, add = (f[:, t] + top - new).exp()[..., None], (i[:, t] - new).exp()[..., None]
                    S = keep[..., None] * S + (add * k[:, t])[..., None] * v[:, t, :, None]
                    nrm, top = keep * nrm + add * k[:, t], new
                    den = torch.maximum((nrm * q[:, t]).sum(-1).abs(), (-top).exp()) + 1e-6
                    o[:, t] = (q[:, t, :, None] @ S)[:, :, 0] / den[..., None]
                else:
                    S = w64(p["decay"])[:, None, None] * S + k[:, t][..., None] * v[:, t, :, None]
                    o[:, t] = (q[:, t, :, None] @ S)[:, :, 0]
            o = _rms(o, 1.0, eps).reshape(B, T, -1) if kind == "MLstm" else _rms(o.reshape(B, T, -1), 1.0, eps)
            y = lin(o * w64(p["norm"]) * torch.sigmoid(g), p["o"])
        x = x + _rms(y, w64(lp["norm1b"]), eps)
        if layer.mlp is not None:
            f, h = lp["mlp"], _rms(x, w64(lp["norm2"]), eps).reshape(B * T, -1)
            glu = lambda r, gu, down: lin(F.silu(lin(r, gu).chunk(2, -1)[0]) * lin(r, gu).chunk(2, -1)[1], down)
            score, idx = torch.sigmoid(lin(h, f["router"])).topk(layer.mlp.top, -1)
            y = glu(h, f["shared_gate_up"], f["shared_down"])
            for j in range(layer.mlp.top):                # the score scales the expert's input
                y = y + _by_expert(h * score[:, j:j + 1], torch.ones_like(score[:, :1]), idx[:, j:j + 1], lambda e, r: glu(r, f["gate_up"][e], f["down"][e]))
            x = x + _rms(y.reshape(B, T, -1), w64(lp["norm2b"]), eps)
    last = x[torch.arange(B, device="cuda"), n - 1]
    return lin(_rms(last, w64(params["final_norm"]), eps), params["head"])


def _banded_turn(x, rot):
    """Half-split rotation with long waves slowed by a factor and a middle band blended."""
    f = rot.base ** (-torch.arange(0, rot.dims, 2, device=x.device, dtype=F64) / rot.dims)
    if rot.scaling:
        sc = dict(rot.scaling)
        turns = sc["original"] * f / (2 * math.pi)
        blend = ((turns - sc["low"]) / (sc["high"] - sc["low"])).clamp(0, 1)
        f = (1 - blend) * f / sc["factor"] + blend * f
    ang = torch.arange(x.shape[1], device=x.device, dtype=F64)[:, None, None] * f
    u, v = x[..., :rot.dims // 2], x[..., rot.dims // 2:rot.dims]
    return torch.cat([u * ang.cos() - v * ang.sin(), v * ang.cos() + u * ang.sin(), x[..., rot.dims:]], -1)


# ---- the file's functions ------------------------------------------------------------------------------------------
PATHS = {"gpt2_train": Gpt2Train, "qwen_prefill": QwenPrefill, "qwen_decode": QwenDecode, "qwen_train": QwenTrain,
         "deepseek_prefill": DeepseekPrefill, "deepseek_decode": DeepseekDecode, "fp8_linear": Fp8Linear,
         "fovudra_prefill": FovudraPrefill, "fovudra_decode": FovudraDecode}


def prepare(case, seed):
    return PATHS[case["path"]].prepare(case, seed), case["path"]


def run(state):
    s, path = state
    return PATHS[path].run(s)


def work(case):
    return PATHS[case["path"]].work(case)


def exact(case, seed):
    return PATHS[case["path"]].exact(case, seed)


#: four times the difference that another order of sums or another exact form of the same bf16 path shows
TOLERANCE = {"gpt2_train": 2e-2, "qwen_prefill": 3e-2, "qwen_decode": 3e-2, "qwen_train": 3e-2, "deepseek_prefill": 3e-2,
             "deepseek_decode": 3e-2, "fp8_linear": 1e-2, "fovudra_prefill": 3e-2, "fovudra_decode": 3e-2}


def tolerance(case):
    return {"rel": TOLERANCE[case["path"]], "max": 0.9}
