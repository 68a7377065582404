"""What serving with this framework spends its time on: one engine step of each served model family.

A case is one scheduled batch - decode rows, prompt portions, or both - that `ModelRunner.execute` runs as the engine's loop
does: pack the inputs into pinned memory, copy them over, embedding, layers, final norm, logits.  The families are the ones
the engine is configured for: a dense GQA decoder (the Qwen3-8B preset's sizes), a sparse mixture of experts (the
Qwen3-30B-A3B preset's), a hybrid of gated delta nets and gated attention (the Qwen3-Next layout at the width the design
benchmark uses) and latent attention with experts in block-scaled fp8 (the DeepSeek-V3 preset's widths).  A few layers stand
for a model's many, which repeat them; the vocabulary is the design benchmark's.

`exact` is the same step in 64 bits and plain torch from the same weights.
"""
import dataclasses
import math

import numpy as np
import torch

VOCAB, BLOCK, MAX_LEN = 32768, 16, 8448
EXPERTS_FP8 = 32          # routed experts of the fp8 model: the number kernel_bench.py measures this layer with


# ----------------------------------------------------------------------------- the cases
def listed():
    def case(name, family, decode=0, context=0, prompts=0, prompt=0, behind=0):
        return {"name": name, "family": family, "decode": decode, "context": context, "prompts": prompts, "prompt": prompt,
                "behind": behind}
    return [
        case("dense_decode_1", "dense", decode=1, context=777),                       # one user at a chat prompt: latency
        case("dense_decode_64", "dense", decode=64, context=4000),                    # a busy server between prompts
        case("dense_mixed", "dense", decode=48, context=2000, prompts=1, prompt=500, behind=1024),    # a portion joins decoding
        case("dense_prefill", "dense", prompts=5, prompt=2048),                       # offline prompts, several a step
        case("moe_decode_16", "moe", decode=16, context=2500),                        # few rows, most experts touched
        case("moe_prefill", "moe", prompts=3, prompt=1300),                           # prompts over all experts
        case("hybrid_decode_2", "hybrid", decode=2, context=300),                     # two users of a hybrid model
        case("hybrid_decode_64", "hybrid", decode=64, context=700),                   # a busy server, hybrid model
        case("hybrid_prefill", "hybrid", prompts=4, prompt=1024),                     # prompts of a hybrid model
        case("latent_decode_16", "latent", decode=16, context=8000),                  # long contexts on a latent cache
        case("latent_decode_64", "latent", decode=64, context=3000),                  # a busy server, latent cache
        case("latent_prefill", "latent", prompts=2, prompt=600),                      # prompts on a latent cache
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    family = rng.choice(["dense", "moe", "hybrid", "latent"])
    kind = rng.choice(["decode", "prefill", "decode", "prefill", "mixed"])
    c = {"family": family, "decode": 0, "context": 0, "prompts": 0, "prompt": 0, "behind": 0}
    if kind != "prefill":
        c["decode"] = log(1, 64)
        c["context"] = log(40, 900 if family == "hybrid" else min(8000, 4000 * 64 // c["decode"]))
    if kind != "decode":
        most = {"dense": 8000, "moe": 6000, "hybrid": 4000, "latent": 1200}[family] if kind == "prefill" else 600
        c["prompts"] = rng.randint(1, 4) if kind == "prefill" else rng.randint(1, 2)
        c["prompt"] = log(17, min(2048, most // c["prompts"]))
        c["behind"] = rng.choice([0, 0, log(30, 600 if family == "hybrid" else 1500)])
    return c


def _lengths(n, most):
    """Ragged lengths up to `most`, the first one the longest."""
    return [max(2, int(round(most * (1.0 - 0.75 * ((i * 0.6180339887) % 1.0))))) for i in range(n)]


def _sequences(case):
    """[(tokens already in the cache, tokens of this step)]: decode rows first."""
    return [(n, 1) for n in _lengths(case["decode"], case["context"])] + \
           [(case["behind"], n) for n in _lengths(case["prompts"], case["prompt"])]


# ----------------------------------------------------------------------------- models and weights
def _args(family):
    from xllm_b200.models import ModelArgs, preset
    if family == "dense":
        return dataclasses.replace(preset("qwen3-8b"), num_hidden_layers=4, vocab_size=VOCAB)
    if family == "moe":
        return dataclasses.replace(preset("qwen3-30b-a3b"), num_hidden_layers=2, vocab_size=VOCAB)
    if family == "latent":
        return dataclasses.replace(preset("deepseek-v3"), num_hidden_layers=2, first_k_dense_replace=1, vocab_size=VOCAB,
                                   num_experts=EXPERTS_FP8, num_nextn_predict_layers=0, max_position_embeddings=32768)
    return ModelArgs(model_type="qwen3_next", vocab_size=VOCAB, hidden_size=2048, num_hidden_layers=4, num_attention_heads=16,
                     num_key_value_heads=4, head_dim=128, intermediate_size=6144, qk_norm=True, rope_theta=1e6,
                     partial_rotary_factor=0.25, max_position_embeddings=32768, tie_word_embeddings=False,
                     extra=dict(linear_num_value_heads=32, linear_num_key_heads=16, linear_key_head_dim=128,
                                linear_value_head_dim=128, linear_conv_kernel_dim=4, full_attention_interval=4))


class _Weights:
    """A checkpoint of the family by tensor name, each tensor made from the seed and its own name."""

    def __init__(self, family, seed):
        self.a, self.family, self.seed = _args(family), family, seed
        self.dev = torch.device("cuda", torch.cuda.current_device())

    def gen(self, name):
        g = torch.Generator(device=self.dev)
        h = 0
        for ch in name:
            h = (h * 131 + ord(ch)) % (1 << 31)
        g.manual_seed((self.seed * 1000003 + h) % (1 << 62))
        return g

    def normal(self, name, *shape, std=0.02, mean=0.0):
        return torch.empty(shape, dtype=torch.bfloat16, device=self.dev).normal_(mean, std, generator=self.gen(name))

    def uniform(self, name, *shape, lo=0.0, hi=1.0):
        return torch.empty(shape, dtype=torch.float32, device=self.dev).uniform_(lo, hi, generator=self.gen(name))

    def fp8(self, name, rows, cols):
        """{name: e4m3 weight, name + _scale_inv: its scales by blocks of 128 x 128}."""
        q = torch.empty(rows, cols, dtype=torch.bfloat16, device=self.dev).normal_(0.0, 96.0, generator=self.gen(name))
        s = self.uniform(name + "_s", (rows + 127) // 128, (cols + 127) // 128, lo=0.5, hi=1.5) * (0.02 / 96.0)
        return {name: q.clamp_(-448, 448).to(torch.float8_e4m3fn), name + "_scale_inv": s}

    def linear(self, name, rows, cols):
        if self.family == "latent" and "kv_b_proj" not in name:
            return self.fp8(name, rows, cols)
        return {name: self.normal(name, rows, cols)}

    def _routed(self):
        """Columns of the residual stream that only the embedding writes and the routers read: a trained router decides
        with a margin, one of random numbers on ties that any rounding turns."""
        return self.a.num_experts if self.family in ("moe", "latent") else 0

    def embedding(self):
        name, E = "model.embed_tokens.weight", self._routed()
        w = self.normal(name, VOCAB, self.a.hidden_size, std=0.5)
        if E:
            top = self.a.num_experts_per_tok
            level = torch.empty(VOCAB, E, device=self.dev).uniform_(-1.0, 0.5, generator=self.gen("levels"))
            rank = torch.rand(VOCAB, E, device=self.dev, generator=self.gen("chosen"))
            if self.family == "latent":      # the chosen experts lie in `topk_group` groups, equally many in each
                G, keep = self.a.n_group, self.a.topk_group
                groups = torch.rand(VOCAB, G, device=self.dev, generator=self.gen("groups")).topk(keep, dim=1).indices
                inside = rank.view(VOCAB, G, E // G).topk(top // keep, dim=2).indices
                chosen = (torch.arange(G, device=self.dev)[None, :, None] * (E // G) + inside)
                chosen = chosen.gather(1, groups[:, :, None].expand(-1, -1, top // keep)).reshape(VOCAB, top)
            else:
                chosen = rank.topk(top, dim=1).indices
            high = torch.empty(VOCAB, top, device=self.dev).uniform_(1.5, 3.0, generator=self.gen("high"))
            w[:, :E] = level.scatter(1, chosen, high).to(w.dtype)
        return w

    def out_rows(self, tensors):
        """A projection into the residual stream: the routers' columns get nothing."""
        for n, w in tensors.items():
            E = self._routed()
            if E and not n.endswith("_scale_inv"):
                w.view(torch.uint8 if w.dtype.itemsize == 1 else torch.int16)[:E] = 0
        return tensors

    def layer(self, i):
        """Name without the layer's prefix -> tensor."""
        a, p = self.a, f"{i}."
        H, nq, nkv, d = a.hidden_size, a.num_attention_heads, a.num_key_value_heads, a.head_dim
        t, zero_centred = {}, self.family == "hybrid"

        def norm(name, n, zero=zero_centred):
            t[name] = self.normal(p + name, n, std=0.1, mean=0.0 if zero else 1.0)

        def lin(name, rows, cols, out=False):
            w = self.linear(p + name, rows, cols)
            t.update({n[len(p):]: x for n, x in (self.out_rows(w) if out else w).items()})

        norm("input_layernorm.weight", H)
        norm("post_attention_layernorm.weight", H)
        if self.family == "latent":
            nope, rope, vd, L = a.qk_nope_head_dim, a.qk_rope_head_dim, a.v_head_dim, a.kv_lora_rank
            lin("self_attn.q_a_proj.weight", a.q_lora_rank, H)
            norm("self_attn.q_a_layernorm.weight", a.q_lora_rank)
            lin("self_attn.q_b_proj.weight", nq * (nope + rope), a.q_lora_rank)
            lin("self_attn.kv_a_proj_with_mqa.weight", L + rope, H)
            norm("self_attn.kv_a_layernorm.weight", L)
            lin("self_attn.kv_b_proj.weight", nq * (nope + vd), L)
            lin("self_attn.o_proj.weight", H, nq * vd, out=True)
        elif self.family == "hybrid" and (i + 1) % a.extra["full_attention_interval"]:
            e = a.extra
            nk, nv, dk, dv = (e[k] for k in ("linear_num_key_heads", "linear_num_value_heads", "linear_key_head_dim",
                                             "linear_value_head_dim"))
            lin("linear_attn.in_proj_qkvz.weight", 2 * nk * dk + 2 * nv * dv, H)
            lin("linear_attn.in_proj_ba.weight", 2 * nv, H)
            t["linear_attn.conv1d.weight"] = self.normal(p + "conv", 2 * nk * dk + nv * dv, 1, e["linear_conv_kernel_dim"], std=0.3)
            t["linear_attn.dt_bias"] = self.uniform(p + "dt", nv, lo=-4.0, hi=0.0).bfloat16()
            t["linear_attn.A_log"] = self.uniform(p + "A", nv, lo=0.5, hi=16.0).log().bfloat16()
            norm("linear_attn.norm.weight", dv, zero=False)
            lin("linear_attn.out_proj.weight", H, nv * dv, out=True)
        else:
            lin("self_attn.q_proj.weight", nq * d * (2 if self.family == "hybrid" else 1), H)
            lin("self_attn.k_proj.weight", nkv * d, H)
            lin("self_attn.v_proj.weight", nkv * d, H)
            norm("self_attn.q_norm.weight", d)
            norm("self_attn.k_norm.weight", d)
            lin("self_attn.o_proj.weight", H, nq * d, out=True)
        if a.is_moe_layer(i):
            gate = torch.zeros(a.num_experts, H, dtype=torch.bfloat16, device=self.dev)
            gate[:, :a.num_experts] = torch.eye(a.num_experts, device=self.dev) * (1.0 if self.family == "latent" else 0.7)
            t["mlp.gate.weight"] = gate
            if self.family == "latent":
                t["mlp.gate.e_score_correction_bias"] = self.uniform(p + "bias", a.num_experts, lo=0.0, hi=0.02)
            I, names = a.moe_intermediate_size, [f"mlp.experts.{e}." for e in range(a.num_experts)]
            names += ["mlp.shared_experts."] * (1 if self.family == "latent" else 0)
        else:
            I, names = a.intermediate_size, ["mlp."]
        for n in names:
            lin(n + "gate_proj.weight", I, H)
            lin(n + "up_proj.weight", I, H)
            lin(n + "down_proj.weight", H, I, out=True)
        return t

    def final_norm(self):
        return self.normal("norm", self.a.hidden_size, std=0.1, mean=0.0 if self.family == "hybrid" else 1.0)

    def lm_head(self):
        return self.normal("lm_head", VOCAB, self.a.hidden_size)

    def checkpoint(self):
        yield "model.embed_tokens.weight", self.embedding()
        for i in range(self.a.num_hidden_layers):
            for n, w in self.layer(i).items():
                yield f"model.layers.{i}.{n}", w
        yield "model.norm.weight", self.final_norm()
        yield "lm_head.weight", self.lm_head()

    # what the cache holds for the tokens in front of the step, by layer: [tokens, heads, size] each, in sequence order.  Keys
    # are normed and rotated, latents normed, values as projected.
    def cached(self, i, tokens):
        a = self.a
        if self.family == "latent":
            c = self.normal(f"{i}.c", tokens, 1, a.kv_lora_rank, std=1.0)
            return [torch.cat([c, self.normal(f"{i}.pe", tokens, 1, a.qk_rope_head_dim, std=1.7)], dim=-1)]
        shape = (tokens, a.num_key_value_heads, a.head_dim)
        return [self.normal(f"{i}.k", *shape, std=1.0), self.normal(f"{i}.v", *shape, std=1.2)]


def _tokens(case, seed):
    """Per sequence: (ids in front of the step, ids of the step)."""
    rng = np.random.default_rng(seed)
    return [(rng.integers(0, VOCAB, b), rng.integers(0, VOCAB, n)) for b, n in _sequences(case)]


# ----------------------------------------------------------------------------- the step
def prepare(case, seed):
    """An engine with the checkpoint loaded and the sequences' earlier tokens in its cache, and the scheduled batch."""
    from xllm_b200 import EngineConfig, LLMEngine
    w = _Weights(case["family"], seed)
    seqs, toks = _sequences(case), _tokens(case, seed)
    total = sum(-(-(b + n) // BLOCK) + 1 for b, n in seqs)
    step = sum(n for _, n in seqs)
    hybrid = case["family"] == "hybrid"
    engine = LLMEngine(EngineConfig(
        model="perf", device="cuda:0", dtype="bfloat16", block_size=BLOCK, num_blocks=total + 8, max_seqs_per_batch=max(len(seqs), 8),
        max_tokens_per_batch=max(step, 2304), max_model_len=MAX_LEN, random_weights=True, enable_prefix_cache=False,
        max_running_seqs=len(seqs), mla_latent_cache=case["family"] == "latent"), model_args=w.a)
    engine.update_weights(w.checkpoint())
    sched, runner, none = engine.scheduler, engine.runner, np.empty(0, dtype=np.int64)
    ids = [f"r{i}" for i in range(len(seqs))]
    # earlier tokens, in portions by turns, so that the sequences' pages lie mixed as they do on a running server
    portion = 2048 if hybrid else 256
    for at in range(0, max(b for b, _ in seqs), portion):
        group, size = [], 0
        for r, part in [(r, before[at:at + portion]) for r, (before, _) in zip(ids, toks)] + [(None, None)]:
            if group and (r is None or size + len(part) > 2048):
                batch = sched.schedule_replay([g[0] for g in group], [g[1].tolist() for g in group], [[] for _ in group])
                if hybrid:                      # recurrent states come from the tokens themselves
                    runner.execute(batch, want_host=False, want_logits=True)
                sched.process_output(batch.batch_id, none, None)
                group, size = [], 0
            if r is not None and len(part):
                group.append((r, part))
                size += len(part)
    batch = sched.schedule_replay(ids, [t.tolist() for _, t in toks], [[len(t) - 1] for _, t in toks])
    earlier = sum(b for b, _ in seqs)
    if earlier and not hybrid:
        row = {batch.request_id(i): i for i in range(batch.n_seqs)}
        table = np.asarray(batch.block_tables)
        page = torch.from_numpy(np.concatenate([table[row[r]][np.arange(b) // BLOCK] for r, (b, _) in zip(ids, seqs)])).cuda().long()
        place = torch.from_numpy(np.concatenate([np.arange(b) % BLOCK for b, _ in seqs])).cuda()
        for i, planes in enumerate(runner.kv_caches):
            for plane, values in zip(planes, w.cached(i, earlier)):
                plane[page, :, place] = values
    key = runner.graph_key(batch, "logits")
    if key is not None:
        runner.capture_graph(key)
    return {"engine": engine, "runner": runner, "batch": batch}


def run(state):
    """One step.  Logits at every sequence's last token, rows in the batch's order, and the caches it wrote to."""
    runner = state["runner"]
    logits = runner.execute(state["batch"], want_host=False, want_logits=True)
    return {"logits": logits, "cache": [k for k, _ in runner.kv_caches if k is not None],
            "values": [v for k, v in runner.kv_caches if k is not None and v.data_ptr() != k.data_ptr()]}


def work(case):
    """Weights once (of the experts those that random routing reaches), every sequence's cache once, the logits."""
    a, seqs = _args(case["family"]), _sequences(case)
    T, H, d = sum(n for _, n in seqs), a.hidden_size, a.head_dim
    pairs = sum(n * b + n * (n + 1) / 2 for b, n in seqs)
    context = sum(b + n for b, n in seqs)
    byte = 1 if case["family"] == "latent" else 2
    nbytes, flops = T * H * 2.0, 0.0
    for i in range(a.num_hidden_layers):
        linear = case["family"] == "hybrid" and (i + 1) % a.extra["full_attention_interval"] != 0
        if case["family"] == "latent":
            nh, nope, rope, vd, L = a.num_attention_heads, a.qk_nope_head_dim, a.qk_rope_head_dim, a.v_head_dim, a.kv_lora_rank
            w = a.q_lora_rank * (H + nh * (nope + rope)) + (L + rope) * H + H * nh * vd
            nbytes += w + 2 * nh * (nope + vd) * L + 2 * context * (L + rope)
            fresh = sum(n for b, n in seqs if n > 1)          # prompts expand what they attend to, decoding absorbs instead
            expanded = sum(b + n for b, n in seqs if n > 1)
            pre = sum(n * b + n * (n + 1) / 2 for b, n in seqs if n > 1)
            flops += 2 * T * w + 2 * (T - fresh + expanded) * nh * (nope + vd) * L
            flops += 2 * pre * nh * (nope + rope + vd) + 2 * (pairs - pre) * nh * (2 * L + rope)
        elif linear:
            e = a.extra
            kd, vdim = e["linear_num_key_heads"] * e["linear_key_head_dim"], e["linear_num_value_heads"] * e["linear_value_head_dim"]
            w = H * (2 * kd + 2 * vdim + 2 * e["linear_num_value_heads"]) + H * vdim
            state = vdim * e["linear_key_head_dim"]
            fresh = sum(1 for b, _ in seqs if b == 0)
            nbytes += 2 * w + 4 * state * (2 * len(seqs) - fresh)
            flops += 2 * T * w + 6 * T * state
        else:
            gate = 2 if case["family"] == "hybrid" else 1
            w = H * d * (a.num_attention_heads * (gate + 1) + 2 * a.num_key_value_heads)
            nbytes += 2 * w + 4 * context * a.num_key_value_heads * d
            flops += 2 * T * w + 4 * pairs * a.num_attention_heads * d
        if a.is_moe_layer(i):
            E, k, one = a.num_experts, a.num_experts_per_tok, 3 * H * a.moe_intermediate_size
            shared = a.n_shared_experts
            nbytes += byte * one * (E * (1 - (1 - k / E) ** T) + shared) + 2 * E * H
            flops += 2 * T * one * (k + shared) + 2 * T * E * H
        else:
            one = 3 * H * a.intermediate_size
            nbytes += byte * one
            flops += 2 * T * one
    nbytes += 2 * VOCAB * H + 2 * len(seqs) * VOCAB
    flops += 2 * len(seqs) * VOCAB * H
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """bf16 activations throughout: against 64 bits a step is off by 0.005 (experts: the routers' margins carry the embedding
    through), 0.011 (dense), 0.017 (hybrid) and 0.05 (latent, whose fp8 products also round activations to e4m3), and another
    correct order of sums or roundings by about as much from this one, except that roundings of the same inputs are shared."""
    return {"rel": 0.02 if case["family"] == "moe" else 0.03, "max": 0.3}


# ----------------------------------------------------------------------------- the same in 64 bits
def _rms(x, w, eps, zero=False):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps) * (w.double() + 1.0 if zero else w.double())


def _rope(x, pos, theta, dims, adjacent):
    """x [n, heads, size], the first `dims` of which are rotated."""
    half = dims // 2
    ang = pos.double()[:, None] * theta ** (-torch.arange(half, device=x.device, dtype=torch.float64) * 2 / dims)
    c, s = ang.cos()[:, None], ang.sin()[:, None]
    r = x[..., :dims]
    x1, x2 = (r[..., 0::2], r[..., 1::2]) if adjacent else (r[..., :half], r[..., half:])
    y1, y2 = x1 * c - x2 * s, x2 * c + x1 * s
    y = torch.stack([y1, y2], dim=-1).flatten(-2) if adjacent else torch.cat([y1, y2], dim=-1)
    return torch.cat([y, x[..., dims:]], dim=-1)


def _attend(q, k, v, scale, before):
    """q [n, h, d] behind `before` tokens of k, v [before + n, h or fewer, d]."""
    n, h, out = q.shape[0], q.shape[1], []
    group = h // k.shape[1]
    rows = max(1, int(2e8 // (h * k.shape[0])))
    for a in range(0, n, rows):
        b = min(n, a + rows)
        seen = before + b
        qq = q[a:b].view(b - a, k.shape[1], group, -1)
        s = torch.einsum("nkgd,tkd->kgnt", qq, k[:seen]) * scale
        hide = torch.arange(seen, device=q.device)[None] > before + torch.arange(a, b, device=q.device)[:, None]
        p = torch.softmax(s.masked_fill(hide, -math.inf), dim=-1)
        out.append(torch.einsum("kgnt,tkd->nkgd", p, v[:seen]).reshape(b - a, h, -1))
    return torch.cat(out)


def _dequant(t, name):
    w = t[name].double()
    s = t.get(name + "_scale_inv")
    if s is None:
        return w
    s = s.double().repeat_interleave(128, 0)[:w.shape[0]].repeat_interleave(128, 1)[:, :w.shape[1]]
    return w * s


def _delta_net(x, t, a, bounds):
    """Gated delta net over whole sequences (they start from nothing)."""
    e = a.extra
    nk, nv, dk, dv, K = (e[k] for k in ("linear_num_key_heads", "linear_num_value_heads", "linear_key_head_dim",
                                        "linear_value_head_dim", "linear_conv_kernel_dim"))
    r, T, F = nv // nk, x.shape[0], torch.nn.functional
    y = (x @ _dequant(t, "linear_attn.in_proj_qkvz.weight").T).view(T, nk, -1)
    q, k, v, z = torch.split(y, [dk, dk, r * dv, r * dv], dim=-1)
    b, al = torch.split((x @ _dequant(t, "linear_attn.in_proj_ba.weight").T).view(T, nk, 2 * r), [r, r], dim=-1)
    beta = torch.sigmoid(b.reshape(T, nv))
    decay = torch.exp(-t["linear_attn.A_log"].double().exp() * F.softplus(al.reshape(T, nv) + t["linear_attn.dt_bias"].double()))
    mixed = torch.cat([q.reshape(T, -1), k.reshape(T, -1), v.reshape(T, -1)], dim=-1)
    cw = t["linear_attn.conv1d.weight"].double()[:, 0]
    most = max(e1 - e0 for e0, e1 in bounds)
    B = len(bounds)
    pad = x.new_zeros(B, most + K - 1, mixed.shape[1])
    dd, bb = x.new_ones(B, most, nv), x.new_zeros(B, most, nv)
    for i, (e0, e1) in enumerate(bounds):
        pad[i, K - 1:K - 1 + e1 - e0] = mixed[e0:e1]
        dd[i, :e1 - e0], bb[i, :e1 - e0] = decay[e0:e1], beta[e0:e1]
    conv = F.silu(sum(pad[:, j:j + most] * cw[:, j] for j in range(K)))
    q, k, v = torch.split(conv, [nk * dk, nk * dk, nv * dv], dim=-1)

    def unit(u):
        u = u.reshape(B, most, nk, dk)
        return (u * torch.rsqrt(u.pow(2).sum(-1, keepdim=True) + 1e-6)).repeat_interleave(r, dim=2)

    q, k, v = unit(q) * dk ** -0.5, unit(k), v.reshape(B, most, nv, dv)
    S, out = x.new_zeros(B, nv, dk, dv), x.new_empty(B, most, nv, dv)
    for j in range(most):
        S = S * dd[:, j, :, None, None]
        delta = (v[:, j] - torch.einsum("bhkv,bhk->bhv", S, k[:, j])) * bb[:, j, :, None]
        S = S + k[:, j, :, :, None] * delta[:, :, None]
        out[:, j] = torch.einsum("bhkv,bhk->bhv", S, q[:, j])
    o = torch.cat([out[i, :e1 - e0] for i, (e0, e1) in enumerate(bounds)])
    o = _rms(o, t["linear_attn.norm.weight"], a.rms_norm_eps) * F.silu(z.reshape(T, nv, dv))
    return o.reshape(T, -1) @ _dequant(t, "linear_attn.out_proj.weight").T


def _mlp(x, t, n):
    return (torch.nn.functional.silu(x @ _dequant(t, n + "gate_proj.weight").T) * (x @ _dequant(t, n + "up_proj.weight").T)) \
        @ _dequant(t, n + "down_proj.weight").T


def _experts(x, t, a):
    logits = x @ t["mlp.gate.weight"].double().T
    T, E, k = x.shape[0], a.num_experts, a.num_experts_per_tok
    if a.scoring_func == "sigmoid":
        score = torch.sigmoid(logits)
        biased = score + t["mlp.gate.e_score_correction_bias"].double()
        best = biased.view(T, a.n_group, -1).topk(2, dim=-1).values.sum(-1).topk(a.topk_group, dim=-1).indices
        keep = torch.zeros(T, a.n_group, dtype=torch.bool, device=x.device).scatter_(1, best, True)
        chosen = biased.masked_fill(~keep.repeat_interleave(E // a.n_group, 1), -math.inf).topk(k, dim=-1).indices
    else:
        score = torch.softmax(logits, dim=-1)
        chosen = score.topk(k, dim=-1).indices
    weight = score.gather(1, chosen)
    weight = weight / weight.sum(-1, keepdim=True) * a.routed_scaling_factor
    y = _mlp(x, t, "mlp.shared_experts.") if a.n_shared_experts else torch.zeros_like(x)
    for e in range(E):
        row, place = (chosen == e).nonzero(as_tuple=True)
        if len(row):
            y.index_add_(0, row, _mlp(x[row], t, f"mlp.experts.{e}.") * weight[row, place, None])
    return y


@torch.no_grad()
def exact(case, seed):
    w = _Weights(case["family"], seed)
    a, seqs, toks, hybrid = w.a, _sequences(case), _tokens(case, seed), case["family"] == "hybrid"
    eps = a.rms_norm_eps
    # what the model runs on: a hybrid's states come from the earlier tokens, the others' caches are given
    rows = [np.concatenate([b, n]) if hybrid else n for b, n in toks]
    begin = [0 if hybrid else b for b, _ in seqs]
    ends = np.cumsum([len(r) for r in rows])
    bounds = [(int(e - len(r)), int(e)) for r, e in zip(rows, ends)]
    ids = torch.from_numpy(np.concatenate(rows)).cuda()
    pos = torch.from_numpy(np.concatenate([np.arange(b, b + len(r)) for b, r in zip(begin, rows)])).cuda()
    x = w.embedding()[ids].double()
    for i in range(a.num_hidden_layers):
        t = w.layer(i)
        h = _rms(x, t["input_layernorm.weight"], eps, hybrid)
        if "linear_attn.A_log" in t:
            y = _delta_net(h, t, a, bounds)
        else:
            y = _attention(w, i, h, t, a, bounds, begin, pos)
        x = x + y
        h = _rms(x, t["post_attention_layernorm.weight"], eps, hybrid)
        x = x + (_experts(h, t, a) if a.is_moe_layer(i) else _mlp(h, t, "mlp."))
    last = torch.tensor([e - 1 for _, e in bounds], device=x.device)
    logits = _rms(x[last], w.final_norm(), eps, hybrid) @ w.lm_head().double().T
    return {"logits": logits, "cache": None, "values": None}


def _attention(w, i, h, t, a, bounds, begin, pos):
    T, nq, d, theta, eps = h.shape[0], a.num_attention_heads, a.head_dim, a.rope_theta, a.rms_norm_eps
    earlier = w.cached(i, sum(begin)) if sum(begin) else None
    gate = None
    if w.family == "latent":
        nope, rd, vd, L = a.qk_nope_head_dim, a.qk_rope_head_dim, a.v_head_dim, a.kv_lora_rank
        q = _rms(h @ _dequant(t, "self_attn.q_a_proj.weight").T, t["self_attn.q_a_layernorm.weight"], eps)
        q = (q @ _dequant(t, "self_attn.q_b_proj.weight").T).view(T, nq, nope + rd)
        kv = h @ _dequant(t, "self_attn.kv_a_proj_with_mqa.weight").T
        c = _rms(kv[:, :L], t["self_attn.kv_a_layernorm.weight"], eps)
        new = torch.cat([c, _rope(kv[:, None, L:], pos, theta, rd, True)[:, 0]], dim=-1)[:, None]
        kvb = t["self_attn.kv_b_proj.weight"].double().view(nq, nope + vd, L)
        q = torch.cat([torch.einsum("thn,hnl->thl", q[..., :nope], kvb[:, :nope]), _rope(q[..., nope:], pos, theta, rd, True)], dim=-1)
        new, scale = [new], (nope + rd) ** -0.5
    else:
        q = h @ _dequant(t, "self_attn.q_proj.weight").T
        if w.family == "hybrid":
            q, gate = q.view(T, nq, 2 * d).split(d, dim=-1)
        zero = w.family == "hybrid"
        q = _rope(_rms(q.reshape(T, nq, d), t["self_attn.q_norm.weight"], eps, zero), pos, theta, a.rotary_dim, False)
        k = _rms((h @ _dequant(t, "self_attn.k_proj.weight").T).view(T, -1, d), t["self_attn.k_norm.weight"], eps, zero)
        new = [_rope(k, pos, theta, a.rotary_dim, False), (h @ _dequant(t, "self_attn.v_proj.weight").T).view(T, -1, d)]
        scale = d ** -0.5
    out, at = [], 0
    for (e0, e1), b in zip(bounds, begin):
        kv = [torch.cat([earlier[j][at:at + b].double(), n[e0:e1]]) if b else n[e0:e1] for j, n in enumerate(new)]
        at += b
        out.append(_attend(q[e0:e1], kv[0], kv[0][..., :a.kv_lora_rank] if len(kv) == 1 else kv[1], scale, b))
    o = torch.cat(out)
    if w.family == "latent":
        o = torch.einsum("thl,hvl->thv", o, kvb[:, nope:])
    if gate is not None:
        o = o * torch.sigmoid(gate)
    return o.reshape(T, -1) @ _dequant(t, "self_attn.o_proj.weight").T
