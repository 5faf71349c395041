"""The work of one reinforcement-learning step on a dense decoder, phase by phase, as the workers drive it.

* ``rollout``: ``RolloutEngine.generate`` on given prompts (prefill, paged cache, CUDA-graph decode, sampler).  The
  weights are those of a policy that is sure of its next token (the head's rows are the embeddings' under a fixed
  permutation), as a trained one mostly is; decoding is greedy, as in validation.  The prefix cache is off: otherwise a
  second pass on the same prompts would skip their prefill, which new prompts pay for.
* ``prefill``: ``TraceReplay.step`` on long prompts: the engine's prefill alone, and the logits after the last token.
* ``score``: log-probs (and entropy) of the responses of a padded batch, without gradients: the passes over the old and
  the reference policy.
* ``update``: one policy update: zeroed gradients, forward, group advantages, clipped loss with KL and entropy terms,
  backward, AdamW.
* ``loss``: the token-level part alone (advantages, loss, its gradient), which small policies and the critic-free
  algorithms run on whole batches.

Models are the presets ``qwen2.5-0.5b`` (head width 64, tied head) and ``qwen2.5-7b`` (head width 128), whole or cut to
their first layers; batches have unequal prompt and response lengths.  Weights are random with a spread that keeps the
layers' outputs of the embeddings' size."""
import math

import torch
import torch.nn.functional as F
from torch.utils.checkpoint import checkpoint

from siirl_b200.engine.packing import pack_batch
from siirl_b200.engine.rollout.native_engine import RolloutEngine, SamplingParams
from siirl_b200.engine.rollout.trace_replay import TraceReplay
from siirl_b200.models.config import get_config
from siirl_b200.models.decoder import build_model
from siirl_b200.ops.rl import gae_scan, grpo_group_advantage, ppo_token_loss
from siirl_b200.parallel.flat_params import FlatParamStore

SMALL, LARGE = "qwen2.5-0.5b", "qwen2.5-7b"
LR, KL_COEF, ENTROPY_COEF, CLIP = 1e-6, 1e-3, 1e-3, 0.2


def _rollout(model, layers, prompts, samples, prompt, new):
    return {"kind": "rollout", "model": model, "layers": layers, "prompts": prompts, "samples": samples,
            "prompt": prompt, "new": new}


def _prefill(model, layers, prompts, prompt):
    return {"kind": "prefill", "model": model, "layers": layers, "prompts": prompts, "prompt": prompt}


def _scored(kind, model, layers, rows, prompt, response, entropy, checkpointing=False):
    case = {"kind": kind, "model": model, "layers": layers, "rows": rows, "prompt": prompt, "response": response,
            "entropy": entropy}
    return dict(case, checkpointing=checkpointing) if kind == "update" else case


def _loss(rows, response, adv, mode, agg, entropy):
    return {"kind": "loss", "rows": rows, "response": response, "adv": adv, "mode": mode, "agg": agg, "entropy": entropy}


def listed():
    return [
        # a micro-batch of short answers: nothing but latency
        dict(_loss(8, 130, "grpo", "vanilla", "token-mean", False), name="loss-8x130"),
        # the whole batch of the headline configuration: 32 prompts x 8 samples, up to 4096 tokens
        dict(_loss(256, 4096, "grpo", "vanilla", "token-mean", True), name="loss-256x4096"),
        # interactive use and validation of a small policy: the latency of a step
        dict(_rollout(SMALL, 24, 5, 1, 150, 33), name="rollout-0.5b-5"),
        # a batch of prompts on a small policy
        dict(_rollout(SMALL, 24, 96, 1, 500, 33), name="rollout-0.5b-96"),
        # the headline rollout, cut in its response length: 32 prompts of 256-1024 tokens, 8 samples each
        dict(_rollout(LARGE, 28, 32, 8, 1024, 33), name="rollout-7b-32x8"),
        # long prompts, prefill only
        dict(_prefill(LARGE, 6, 3, 8000), name="prefill-7b-3x8000"),
        # scoring of one micro-batch of short samples
        dict(_scored("score", SMALL, 24, 4, 100, 300, True), name="score-0.5b-4"),
        # the headline micro-batch: 8 rows of up to 1024 + 2048 tokens
        dict(_scored("score", LARGE, 4, 8, 1024, 2048, True), name="score-7b-8"),
        # a reference pass over long answers
        dict(_scored("score", SMALL, 24, 2, 700, 15000, False), name="score-0.5b-long"),
        # updates: a small policy with checkpointed layers; wide layers without; long answers
        dict(_scored("update", SMALL, 12, 8, 512, 1024, False, True), name="update-0.5b-8"),
        dict(_scored("update", LARGE, 2, 8, 1024, 2048, True, False), name="update-7b-8"),
        dict(_scored("update", SMALL, 12, 1, 700, 10000, False, True), name="update-0.5b-long"),
    ]


def _between(rng, lo, hi):
    """A whole number between ``lo`` and ``hi``, spread over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["rollout", "rollout", "prefill", "score", "update", "update", "loss"])
    if kind == "loss":
        return _loss(_between(rng, 4, 256), _between(rng, 64, 4096), rng.choice(["grpo", "gae"]),
                     rng.choice(["vanilla", "gspo"]), rng.choice(["token-mean", "seq-mean-token-mean"]),
                     rng.random() < 0.5)
    model = rng.choice([SMALL, LARGE])
    if kind == "prefill":
        return _prefill(model, rng.randint(4, 24) if model == SMALL else rng.randint(1, 6), rng.randint(1, 3),
                        _between(rng, 500, 8000))
    if kind == "rollout":
        layers = rng.randint(6, 24) if model == SMALL else rng.randint(2, 12)
        prompts, samples = _between(rng, 4, 32), rng.choice([1, 2, 4, 8])
        return _rollout(model, layers, prompts, samples, _between(rng, 40, 1024), rng.choice([17, 33]))
    deep = kind == "score"
    layers = rng.randint(4, 24 if deep else 12) if model == SMALL else rng.randint(1, 4 if deep else 2)
    prompt, rows = _between(rng, 30, 1024), _between(rng, 1, 8)
    response = _between(rng, 60, 2048 if model == LARGE or rows > 2 else 8000)
    return _scored(kind, model, layers, rows, prompt, response, rng.random() < 0.5, rng.random() < 0.5)


# ---- sizes --------------------------------------------------------------------------------------
def _config(case):
    over = {"num_layers": case["layers"]}
    if case["kind"] in ("rollout", "prefill"):
        over["tie_word_embeddings"] = False
    return get_config(case["model"], over)


def _lengths(n, lo, hi, shift):
    """``n`` unequal lengths in ``[lo, hi]``; part of the case, not of its random values."""
    return [lo + int((hi - lo + 1) * (((i + 1) * 0.6180339887 + shift) % 1.0)) for i in range(n)]


def _prompt_lengths(case):
    n = case["prompts"] if "prompts" in case else case["rows"]
    top = case["prompt"]
    return _lengths(n, top - top // 8 if top > 2000 else max(1, top // 4), top, 0.1)


def _response_lengths(case):
    top = case["response"]
    return _lengths(case["rows"], top - top // 8 if top > 4096 else max(1, top // 4), top, 0.7)


def _layer_weights(cfg):
    return cfg.hidden_size * (cfg.qkv_width + cfg.q_width + 3 * cfg.intermediate_size)


def work(case):
    if case["kind"] == "loss":
        n = case["rows"] * case["response"]
        # rewards, mask, log-probs of three policies in; advantages and gradients out
        moved = 4 * n * ((5 + 2) + (2 if case["entropy"] else 0) + (2 if case["adv"] == "gae" else 0))
        return {"bytes": moved, "flops": 20 * n}
    cfg = _config(case)
    layer, head, width = _layer_weights(cfg), cfg.vocab_size * cfg.hidden_size, cfg.q_width
    L = cfg.num_layers
    if case["kind"] in ("rollout", "prefill"):
        lens, n, new = _prompt_lengths(case), case.get("samples", 1), case.get("new", 1)
        rows, kv = len(lens) * n, 2 * cfg.num_kv_heads * cfg.head_dim * 2
        flops = 2 * L * layer * sum(lens) + 2 * L * width * sum(x * x for x in lens) + 2 * head * rows
        steps = new - 1
        flops += steps * rows * 2 * (L * layer + head) + 4 * L * width * n * sum(steps * x + steps * steps // 2 for x in lens)
        moved = 2 * new * (L * layer + head) + L * kv * (n * sum(steps * x + steps * steps // 2 for x in lens) + sum(lens))
        return {"bytes": moved, "flops": flops}
    p, r = _prompt_lengths(case), _response_lengths(case)
    flops = 2 * L * layer * (sum(p) + sum(r)) + 2 * L * width * sum((a + b) ** 2 for a, b in zip(p, r)) + 2 * head * sum(r)
    weights = L * layer + head * (1 if cfg.tie_word_embeddings else 2)
    if case["kind"] == "score":
        return {"bytes": 2 * weights, "flops": flops}
    # gradients written and read once, master weights and two moments read and written, weights read and written
    return {"bytes": weights * (4 + 4 + 24 + 2 + 2), "flops": 3 * flops}


def tolerance(case):
    return {"rollout": {"rel": 0.012, "max": 0.2, "differ": 0.01}, "prefill": {"rel": 0.02, "max": 0.2},
            "score": {"rel": 0.003, "max": 0.1}, "update": {"rel": 0.03, "max": 0.9},
            "loss": {"rel": 1e-5, "max": 1e-3}}[case["kind"]]


# ---- inputs -------------------------------------------------------------------------------------
def _fill(tensors, cfg, case, seed):
    """Fills the model's parameters, by name, with the weights of the case: a function of the seed alone."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    std = 0.6 / math.sqrt(cfg.hidden_size)
    served = case["kind"] in ("rollout", "prefill")
    for name in ["embed_tokens"] + [f"layers.{i}.{x}" for i in range(cfg.num_layers) for x in (
            "input_layernorm", "qkv_proj_weight", "qkv_proj_bias", "o_proj_weight", "post_attention_layernorm",
            "gate_up_proj_weight", "down_proj_weight")] + ["norm"] + ([] if cfg.tie_word_embeddings else ["lm_head"]):
        t = tensors[name]
        if name == "lm_head" and served:
            # the head's row of the next token is the embedding of this one: its logit is near 13, others near 0
            t[_successors(cfg)] = (tensors["embed_tokens"].float() * (17.0 / cfg.hidden_size)).to(t.dtype)
        elif name == "norm" or "layernorm" in name:
            t.normal_(1.0, 0.0 if served and name == "norm" else 0.1, generator=gen)
        elif name == "embed_tokens":
            t.normal_(0.0, 1.0 if served else std, generator=gen)
        else:
            t.normal_(0.0, 0.1 if name.endswith("bias") else std, generator=gen)


def _successors(cfg):
    """The token that follows each token: a fixed permutation of the vocabulary."""
    ids = torch.arange(cfg.vocab_size, device="cuda")
    return (ids + 7919) % cfg.vocab_size


def _prompts(case, cfg, seed):
    gen = torch.Generator().manual_seed(seed)
    return [torch.randint(3, cfg.vocab_size, (n,), generator=gen).tolist() for n in _prompt_lengths(case)]


def _token_values(rows, response, seed, lens):
    """Token-level inputs ``[rows, response]``: rewards at the last token, mask, log-probs, values, entropies."""
    gen = torch.Generator(device="cuda").manual_seed(seed + 1)
    shape = (rows, response)
    n = torch.tensor(lens, device="cuda")
    at = torch.arange(response, device="cuda")
    mask = (at[None] < n[:, None]).float()
    score = torch.bernoulli(torch.full((rows,), 0.4, device="cuda"), generator=gen)
    score += 0.01 * torch.randn(rows, generator=gen, device="cuda")
    rewards = torch.zeros(shape, device="cuda")
    rewards[torch.arange(rows, device="cuda"), n - 1] = score
    logp = -torch.empty(shape, device="cuda").exponential_(0.7, generator=gen)
    noise = [torch.randn(shape, generator=gen, device="cuda") for _ in range(3)]
    return {"rewards": rewards, "mask": mask, "logp": logp * mask, "old": (logp + 0.1 * noise[0]) * mask,
            "ref": (logp + 0.2 * noise[1]) * mask, "values": 0.5 * noise[2] * mask,
            "entropy": torch.empty(shape, device="cuda").exponential_(2.0, generator=gen) * mask,
            "group": torch.arange(rows, device="cuda", dtype=torch.int32) // min(8, max(2, rows // 4))}


def _padded(case, cfg, seed):
    """Prompts left-padded, responses right-padded, as the rollout hands them on."""
    gen = torch.Generator(device="cuda").manual_seed(seed + 2)
    P, R, rows = case["prompt"], case["response"], case["rows"]
    ids = torch.randint(3, cfg.vocab_size, (rows, P + R), generator=gen, device="cuda")
    p = torch.tensor(_prompt_lengths(case), device="cuda")[:, None]
    r = torch.tensor(_response_lengths(case), device="cuda")[:, None]
    at = torch.arange(P + R, device="cuda")[None]
    return ids, ((at >= P - p) & (at < P + r)).long()


def prepare(case, seed):
    kind = case["kind"]
    if kind == "loss":
        t = _token_values(case["rows"], case["response"], seed, _response_lengths(case))
        return {"case": case, "groups": int(t["group"].max()) + 1, **t}
    cfg = _config(case)
    model = build_model(cfg, dtype=torch.bfloat16, device="cuda", seed=0,
                        gradient_checkpointing=bool(case.get("checkpointing")))
    with torch.no_grad():
        _fill({k: v.data for k, v in model.named_parameters()}, cfg, case, seed)
    state = {"case": case, "model": model}
    if kind in ("rollout", "prefill"):
        lens, n, new = _prompt_lengths(case), case.get("samples", 1), case.get("new", 1)
        state["prompts"] = _prompts(case, cfg, seed)
        state["engine"] = RolloutEngine(model, max_num_seqs=max(8, -(-len(lens) * n // 8) * 8),
                                        max_model_len=max(lens) + new, enable_prefix_caching=False,
                                        num_blocks=n * sum(-(-(x + new) // 64) for x in lens) + 8)
        if kind == "prefill":
            state["replay"] = TraceReplay(state["engine"], max_slots=8)
        return state
    state["ids"], state["attention"] = _padded(case, cfg, seed)
    if kind == "update":
        state["store"] = FlatParamStore(model)
        t = _token_values(case["rows"], case["response"], seed, _response_lengths(case))
        # the reference policy's log-probs of random tokens under a spread-out distribution
        state.update(rewards=t["rewards"], mask=t["mask"], group=t["group"], groups=int(t["group"].max()) + 1,
                     ref=(0.3 * t["logp"] - math.log(cfg.vocab_size)) * t["mask"])
    else:
        model.requires_grad_(False)
    return state


# ---- one pass -----------------------------------------------------------------------------------
def _logprobs(state):
    case, model = state["case"], state["model"]
    pk = pack_batch(state["ids"], state["attention"], case["response"])
    hidden = model.forward_hidden(pk.input_ids, pk.positions, pk.info)
    logp, ent = model.token_logprobs(hidden.index_select(0, pk.sel), pk.labels, 1.0, case["entropy"])
    return pk.scatter(logp), pk.scatter(ent) if ent is not None else None


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "rollout":
        outs = state["engine"].generate(state["prompts"], SamplingParams(
            n=case["samples"], temperature=0.0, max_new_tokens=case["new"], ignore_eos=True))
        return {"tokens": torch.tensor([o.token_ids for o in outs]),
                "logprobs": torch.tensor([o.logprobs for o in outs])}
    if kind == "prefill":
        rows = [(str(i), x, [len(x) - 1]) for i, x in enumerate(state["prompts"])]
        logits = state["replay"].step(rows)
        state["replay"].end([x[0] for x in rows])
        return {"logits": logits}
    if kind == "score":
        with torch.no_grad():
            logp, ent = _logprobs(state)
        return {"logp": logp} if ent is None else {"logp": logp, "entropy": ent}
    if kind == "loss":
        logp = state["logp"].detach().requires_grad_()
        entropy = state["entropy"].detach().requires_grad_() if case["entropy"] else None
        if case["adv"] == "gae":
            adv, _ = gae_scan(state["rewards"], state["values"], state["mask"], 1.0, 0.95)
        else:
            adv = grpo_group_advantage(state["rewards"], state["mask"], state["group"], state["groups"])
        loss, _ = ppo_token_loss(logp, state["old"], adv, state["mask"], entropy=entropy, ref_logp=state["ref"],
                                 mode=case["mode"], loss_agg_mode=case["agg"], clip_lo=CLIP, clip_hi=CLIP,
                                 kl_coef=KL_COEF, entropy_coef=ENTROPY_COEF if case["entropy"] else 0.0)
        loss.backward()
        out = {"advantages": adv, "grad": logp.grad}
        return dict(out, grad_entropy=entropy.grad) if case["entropy"] else out
    store = state["store"]
    store.zero_grad()
    adv = grpo_group_advantage(state["rewards"], state["mask"], state["group"], state["groups"])
    logp, ent = _logprobs(state)
    # one mini-batch and one epoch: the old policy is the current one
    loss, _ = ppo_token_loss(logp, logp.detach(), adv, state["mask"], entropy=ent, ref_logp=state["ref"],
                             clip_lo=CLIP, clip_hi=CLIP, kl_coef=KL_COEF,
                             entropy_coef=ENTROPY_COEF if case["entropy"] else 0.0)
    loss.backward()
    store.step(LR)
    return {"logp": logp.detach(), "grad": store.flat_grad, "weights": store.master}


# ---- the same in 64 bits ------------------------------------------------------------------------
class _Plain:
    """The decoder in plain 64-bit torch, on packed sequences."""

    def __init__(self, case, seed, grad):
        self.cfg = cfg = _config(case)
        H, L = cfg.hidden_size, cfg.num_layers
        shapes = {"embed_tokens": (cfg.vocab_size, H), "norm": (H,)}    # in the order of the flat buffers
        if not cfg.tie_word_embeddings:
            shapes["lm_head"] = (cfg.vocab_size, H)
        for i in range(L):
            shapes.update({f"layers.{i}.input_layernorm": (H,), f"layers.{i}.qkv_proj_weight": (cfg.qkv_width, H),
                           f"layers.{i}.qkv_proj_bias": (cfg.qkv_width,), f"layers.{i}.o_proj_weight": (H, cfg.q_width),
                           f"layers.{i}.post_attention_layernorm": (H,),
                           f"layers.{i}.gate_up_proj_weight": (2 * cfg.intermediate_size, H),
                           f"layers.{i}.down_proj_weight": (H, cfg.intermediate_size)})
        self.w = {k: torch.empty(s, dtype=torch.bfloat16, device="cuda") for k, s in shapes.items()}
        _fill(self.w, cfg, case, seed)
        self.grad = grad
        if grad:
            for k in list(self.w):
                self.w[k] = self.w[k].double().requires_grad_()

    def get(self, name):
        return self.w[name] if self.grad else self.w[name].double()

    def norm(self, x, name):
        return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + self.cfg.rms_norm_eps) * self.get(name)

    def attend(self, qkv, n):
        cfg, D = self.cfg, self.cfg.head_dim
        q, k, v = (x.reshape(n, -1, D).transpose(0, 1) for x in qkv.split(
            [cfg.q_width, cfg.num_kv_heads * D, cfg.num_kv_heads * D], -1))
        inv = 1.0 / cfg.rope_theta ** (torch.arange(0, D, 2, dtype=torch.float64, device="cuda") / D)
        ang = torch.arange(n, dtype=torch.float64, device="cuda")[:, None] * inv
        cos, sin = torch.cat([ang.cos()] * 2, -1), torch.cat([ang.sin()] * 2, -1)
        turn = lambda x: x * cos + torch.cat([-x[..., D // 2:], x[..., :D // 2]], -1) * sin  # noqa: E731
        q, k, rep, out = turn(q), turn(k), cfg.num_heads // cfg.num_kv_heads, []
        hidden = torch.ones(n, n, dtype=torch.bool, device="cuda").triu_(1)
        for g in range(cfg.num_kv_heads):
            s = (q[g * rep:(g + 1) * rep] @ k[g].T / math.sqrt(D)).masked_fill(hidden, -math.inf)
            out.append(torch.softmax(s, -1) @ v[g])
        return torch.cat(out).transpose(0, 1).reshape(n, -1)

    def layer(self, h, lens, i):
        at = f"layers.{i}."
        qkv = F.linear(self.norm(h, at + "input_layernorm"), self.get(at + "qkv_proj_weight"), self.get(at + "qkv_proj_bias"))
        a = torch.cat([self.attend(x, n) for x, n in zip(qkv.split(lens), lens)])
        h = h + F.linear(a, self.get(at + "o_proj_weight"))
        gate, up = F.linear(self.norm(h, at + "post_attention_layernorm"), self.get(at + "gate_up_proj_weight")).chunk(2, -1)
        return h + F.linear(F.silu(gate) * up, self.get(at + "down_proj_weight"))

    def hidden(self, ids, lens):
        h = self.w["embed_tokens"][ids].double()
        for i in range(self.cfg.num_layers):
            h = checkpoint(self.layer, h, lens, i, use_reentrant=False) if self.grad else self.layer(h, lens, i)
        return self.norm(h, "norm")

    def scores(self, x, labels):
        """Log-prob of the label, entropy and most likely token of every row."""
        head = self.get("embed_tokens" if self.cfg.tie_word_embeddings else "lm_head")

        def part(xs, ys):
            logp = torch.log_softmax(xs @ head.T, -1)
            return logp.gather(1, ys[:, None])[:, 0], -(logp.exp() * logp).sum(-1), logp.argmax(-1)
        parts = [checkpoint(part, a, b, use_reentrant=False) if self.grad else part(a, b)
                 for a, b in zip(x.split(1024), labels.split(1024))]
        return tuple(torch.cat(t) for t in zip(*parts))


def _exact_advantages(t, groups):
    score = t["rewards"].double().sum(-1)
    adv = torch.zeros_like(score)
    for g in range(groups):
        mine = t["group"] == g
        if int(mine.sum()) > 1:
            adv[mine] = (score[mine] - score[mine].mean()) / (score[mine].std() + 1e-6)
        else:
            adv[mine] = score[mine] / (1.0 + 1e-6)
    return adv[:, None] * t["mask"].double()


def _exact_loss(case, t, logp, old, adv, entropy, ref):
    m = t["mask"].double()
    if case.get("mode") == "gspo":
        mean = (((logp - old) * m).sum(-1) / m.sum(-1).clamp(min=1)).detach()
        ratio = torch.exp(mean.clamp(max=10.0)[:, None] + logp - logp.detach())
    else:
        ratio = torch.exp((logp - old).clamp(-20, 20))
    pg = torch.maximum(-adv * ratio, -adv * ratio.clamp(1 - CLIP, 1 + CLIP))
    pg = torch.where(adv < 0, torch.minimum(pg, -adv * 3.0), pg) if case.get("mode") != "gspo" else pg

    def total(x, by_row):
        return ((x * m).sum(-1) / m.sum(-1)).mean() if by_row else (x * m).sum() / m.sum()
    # the sequence-level objective averages all of its terms sequence by sequence
    by_row = case.get("mode") == "gspo" or case.get("agg") == "seq-mean-token-mean"
    k = (ref - logp).clamp(-20, 20)
    loss = total(pg, by_row) + KL_COEF * total((k.exp() - k - 1).clamp(-10, 10), by_row)
    return loss - ENTROPY_COEF * total(entropy, by_row) if entropy is not None else loss


def _exact_gae(t):
    r, v, m = (t[k].double() for k in ("rewards", "values", "mask"))
    nxt = torch.zeros_like(r[:, 0])
    last, adv = torch.zeros_like(nxt), torch.zeros_like(r)
    for i in reversed(range(r.shape[1])):
        now = r[:, i] + nxt - v[:, i] + 0.95 * last
        nxt = torch.where(m[:, i] > 0, v[:, i], nxt)
        last = torch.where(m[:, i] > 0, now, last)
        adv[:, i] = last
    return adv


def exact(case, seed):
    kind = case["kind"]
    if kind == "loss":
        t = _token_values(case["rows"], case["response"], seed, _response_lengths(case))
        logp = t["logp"].double().requires_grad_()
        entropy = t["entropy"].double().requires_grad_() if case["entropy"] else None
        adv = _exact_gae(t) if case["adv"] == "gae" else _exact_advantages(t, int(t["group"].max()) + 1)
        loss = _exact_loss(case, t, logp, t["old"].double(), adv, entropy, t["ref"].double())
        loss.backward()
        out = {"advantages": adv, "grad": logp.grad}
        return dict(out, grad_entropy=entropy.grad) if case["entropy"] else out
    if kind == "prefill":
        with torch.no_grad():
            model = _Plain(case, seed, False)
            rows = _prompts(case, model.cfg, seed)
            lens = [len(x) for x in rows]
            x = model.hidden(torch.tensor([t for x in rows for t in x], device="cuda"), lens)
            last = torch.tensor([sum(lens[:i + 1]) - 1 for i in range(len(lens))], device="cuda")
            return {"logits": x[last] @ model.get("lm_head").T}
    if kind == "rollout":
        with torch.no_grad():
            model = _Plain(case, seed, False)
            succ, new = _successors(model.cfg).tolist(), case["new"]
            rows = _prompts(case, model.cfg, seed)
            lens = [len(x) for x in rows]
            for x in rows:
                for _ in range(new):
                    x.append(succ[x[-1]])
            ids = torch.tensor([t for x in rows for t in x[:-1]], device="cuda")
            labels = torch.tensor([x[n:] for x, n in zip(rows, lens)], device="cuda")
            x = model.hidden(ids, [n + new - 1 for n in lens])
            at = torch.cat([torch.arange(n - 1, n + new - 1) + sum(lens[:i]) + i * (new - 1) for i, n in enumerate(lens)])
            logp, _, best = model.scores(x[at.cuda()], labels.reshape(-1))
            spread = lambda v: v.reshape(-1, new).repeat_interleave(case["samples"], 0)  # noqa: E731
            return {"tokens": spread(best), "logprobs": spread(logp)}
    model = _Plain(case, seed, kind == "update")
    ids, attention = _padded(case, model.cfg, seed)
    p, r, P = _prompt_lengths(case), _response_lengths(case), case["prompt"]
    lens = [a + b for a, b in zip(p, r)]
    starts = [sum(lens[:i]) for i in range(len(lens))]
    sel = torch.cat([torch.arange(s + a - 1, s + a + b - 1) for s, a, b in zip(starts, p, r)]).cuda()
    labels = torch.cat([ids[i, P:P + b] for i, b in enumerate(r)])
    inside = torch.arange(case["response"], device="cuda")[None] < torch.tensor(r, device="cuda")[:, None]

    def place(v):
        return torch.zeros(inside.shape, dtype=v.dtype, device="cuda").masked_scatter(inside, v)
    with torch.set_grad_enabled(kind == "update"):
        logp, ent, _ = model.scores(model.hidden(ids[attention.bool()], lens)[sel], labels)
        logp, ent = place(logp), place(ent) if case["entropy"] else None
    if kind == "score":
        return {"logp": logp} if ent is None else {"logp": logp, "entropy": ent}
    t = _token_values(case["rows"], case["response"], seed, _response_lengths(case))
    ref = (0.3 * t["logp"] - math.log(model.cfg.vocab_size)) * t["mask"]
    adv = _exact_advantages(t, int(t["group"].max()) + 1)
    _exact_loss(case, t, logp, logp.detach(), adv, ent, ref.double()).backward()
    flat, weights = [], []
    for name in list(model.w):
        x = model.w.pop(name)
        pad = -x.numel() % 128
        flat.append(F.pad(x.grad.reshape(-1), (0, pad)))
        weights.append(F.pad(x.detach().to(torch.bfloat16).reshape(-1), (0, pad)))
        del x
    grad, weights = torch.cat(flat), torch.cat(weights)
    del flat
    norm = grad.norm()
    # the first AdamW step: both moments' corrections cancel their factors
    w = weights.double()
    del weights
    w *= 1 - LR * 0.01
    step = grad * min(1.0, 1.0 / (float(norm) + 1e-6))
    w -= LR * step / (step.abs() + 1e-8)
    return {"logp": logp.detach(), "grad": grad, "weights": w}
