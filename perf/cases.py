"""What the engine's speed is measured on: whole passes through `AutoModel`, as a program that serves a model makes them.

A pass is one of three things:

* ``replay``    a batch of prompts goes in (`set_input_cb`, `forward_cb`: logits of the first new token), then `new` - 1 further
                tokens of each sequence, one step at a time (the trace replay of a serving log: the tokens are known, the
                logits of every step are wanted), then the sequences leave (`free_seqs`);
* ``greedy``    the same with tokens chosen on the device (`forward_cb_greedy`), fed back by the host, and the logits of one
                last step;
* ``generate``  `generate()` for a rectangle of prompts, then the logits of every position of what came out (`model(ids)`);
* ``score``     `model(ids)` alone.

Weights are the random ones that the engine draws on the device by tensor name (XFT_FAKE_MODEL=2).  Random weights
answer every rounding with a larger change, and choose tokens and experts by differences below one, as trained models do not; so
the embedding is as large as what the layers add to it, where tokens are chosen the head's rows follow it, and where experts are
chosen it carries the directions of a token's experts.  A program loads its
model once: the states of one architecture share it.  Prompts come from the seed.
"""
import math
import os
import tempfile
import weakref
import zlib

import numpy as np
import torch

import xfastertransformer_b200 as xft
from xfastertransformer_b200.tools.synthetic import config_only, preset
from xfastertransformer_b200.utils.flags import Env


def _case(mode, model, layers, batch, prompt, new, dtype="bf16", kv="bf16", ragged=False, name=None):
    c = {"mode": mode, "model": model, "layers": layers, "batch": batch, "prompt": prompt, "new": new, "dtype": dtype, "kv": kv,
         "ragged": ragged}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest model and call: launches and host work are all there is
        _case("generate", "tiny-llama", 2, 2, 32, 16, name="tiny-generate"),
        # a small chat model behind a server: short ragged prompts, heads of 64, greedy tokens chosen on the device
        _case("greedy", "qwen2-0_5b", 24, 8, 200, 32, ragged=True, name="small-greedy-b8"),
        # one user of a 7B model (half its layers): every step streams all weights for one row
        _case("replay", "llama-2-7b", 16, 1, 512, 32, name="7b-b1"),
        # a full batch on a quarter of the 7B model: the keys and values outweigh the weights
        _case("replay", "llama-2-7b", 8, 32, 1024, 48, ragged=True, name="7b-b32-long"),
        # the same widths with int8 weights and activations, and with 4-bit weights
        _case("replay", "llama-2-7b", 8, 32, 128, 32, dtype="w8a8", name="7b-b32-w8a8"),
        _case("replay", "llama-2-7b", 8, 16, 100, 32, dtype="int4", ragged=True, name="7b-b16-int4"),
        # first token of 70B layers: 2048-token prompts in passes of 8192 tokens
        _case("replay", "llama-2-70b", 2, 8, 2048, 1, name="70b-prompts"),
        # decode steps of 70B layers
        _case("replay", "llama-2-70b", 4, 16, 128, 48, ragged=True, name="70b-steps"),
        # experts: 8 wide ones, two per token
        _case("replay", "mixtral-8x7b", 2, 64, 160, 32, ragged=True, name="mixtral-b64"),
        # latent attention and 256 fp8 experts: one dense and one expert layer
        _case("replay", "deepseek-v3", 2, 32, 128, 16, dtype="fp8_e4m3", ragged=True, name="deepseek-b32"),
        # long contexts in an int8 cache
        _case("replay", "llama-3-8b", 8, 8, 3000, 32, kv="int8", ragged=True, name="8b-long-int8kv"),
        # perplexity of a text: logits of every position, heads of 256, a vocabulary of 256000
        _case("score", "gemma-2b", 18, 2, 389, 0, name="gemma-score"),
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    kind = rng.choice(["prompts", "steps", "steps", "mixed", "quant", "small", "moe", "score"])
    kv, dtype = "bf16", "bf16"
    if kind == "score":
        return _case("score", rng.choice(["gemma-2b", "llama-2-7b"]), rng.randint(2, 6), rng.randint(1, 3), _log(rng, 16, 600), 0)
    if kind == "small":
        return _case("greedy", "qwen2-0_5b", rng.randint(4, 24), _log(rng, 1, 40), _log(rng, 3, 700), rng.randint(4, 24), ragged=rng.random() < 0.5)
    if kind == "moe":
        model, layers = rng.choice([("mixtral-8x7b", 2), ("mixtral-8x7b", 1), ("deepseek-v3", 2)])
        batch, prompt, new = _log(rng, 1, 64), _log(rng, 4, 200), rng.randint(1, 24)
        dtype = "fp8_e4m3" if model == "deepseek-v3" else "bf16"
    else:
        model, layers = rng.choice([("llama-2-7b", 4), ("llama-2-70b", 2), ("llama-3-8b", 4), ("llama-2-7b", 8)])
        batch = _log(rng, 1, 64)
        if kind == "prompts":
            batch = min(batch, 16)
            prompt, new = _log(rng, 200, min(4000, 16384 // batch)), 1
        elif kind == "steps":
            prompt, new = _log(rng, 4, 256), rng.randint(16, 48)
        else:
            prompt, new = _log(rng, 64, min(3000, 20000 // batch)), rng.randint(4, 32)
            if kind == "quant":
                dtype = rng.choice(["w8a8", "int8", "int4"])
            else:
                kv = rng.choice(["bf16", "int8"])
    return _case("replay", model, layers, batch, prompt, new, dtype, kv, rng.random() < 0.6)


def _config(case):
    over = {"num_layer": case["layers"]}
    if case["model"] == "deepseek-v3":
        over["first_k_dense_replace"] = 1          # one dense layer, then experts
    cfg = preset(case["model"], **over)
    cfg.max_pos_seq_len = max(cfg.max_pos_seq_len, case["prompt"] + case["new"] + 64) if case["model"] != "deepseek-v3" else 8192
    return cfg


def _lens(case):
    """Prompt lengths; ragged ones lie between half of `prompt` and `prompt`."""
    n = case["prompt"]
    return [max(1, n - i * 37 % max(n // 2, 1)) if case["ragged"] else n for i in range(case["batch"])]


def _tokens(case, seed):
    """Prompts, and the tokens of the steps after them [new - 1][batch]."""
    r = np.random.RandomState(seed & 0x7FFFFFFF)
    V = _config(case).vocab_size
    prompts = [r.randint(0, V, n).tolist() for n in _lens(case)]
    return prompts, [r.randint(0, V, case["batch"]).tolist() for _ in range(case["new"] - 1)]


# -- weights --------------------------------------------------------------------------------------------------------
_CHOOSING = ("greedy", "generate")
_MOE = ("mixtral", "deepseek_moe")


def _normal(name, shape, std=0.02, dtype=torch.bfloat16):
    """The tensor of that name: N(0, std), drawn on the device from a seed that is the name's CRC."""
    g = torch.Generator(device="cuda")
    g.manual_seed(zlib.crc32(name.encode()) & 0x7FFFFFFF)
    return torch.empty(shape, dtype=dtype, device="cuda").normal_(0.0, std, generator=g)


def _ends(case, cfg):
    """Embedding and head.  Where tokens are chosen, row t + 1 of the head is the embedding of token t in small.  Where experts
    are, an embedding is noise plus the directions of the experts that its token goes to, some stronger than others."""
    shape = (cfg.vocab_size, cfg.hidden_size)
    if case["mode"] in _CHOOSING:
        wte = _normal("model.wte.bin", shape, 4.0)
        return wte, (wte.roll(1, 0).float() * 0.005).bfloat16()
    head = _normal("model.lm_head.weight.bin", shape)
    if cfg.model_type not in _MOE:
        return _normal("model.wte.bin", shape, 6.0), head
    E, k = cfg.sparse_experts, cfg.num_experts_per_tok
    g = torch.Generator(device="cuda")
    g.manual_seed(7)
    groups = max(cfg.n_group, 1)
    at = torch.rand(cfg.vocab_size, groups, E // groups, device="cuda", generator=g)
    if groups > 1:                                       # the experts of a token lie in as many groups as it may use
        far = torch.rand(cfg.vocab_size, groups, device="cuda", generator=g).topk(groups - cfg.topk_group, 1)[1]
        per = at.topk(k // cfg.topk_group, -1)[0][..., -1:]
        at = torch.where(at >= per, at, -1.0).scatter(1, far[..., None].expand(-1, -1, E // groups), -1.0)
    chosen = at.flatten(1).topk(k, -1)[1]
    strength = torch.linspace(1.5, 0.8, k, device="cuda")
    d = _directions(cfg)
    wte = _normal("model.wte.bin", shape, 2.0)
    for j in range(k):
        for r in range(0, cfg.vocab_size, 16384):
            wte[r:r + 16384] += 2 * strength[j] * d[chosen[r:r + 16384, j]]
    return wte, head


def _directions(cfg):
    return _normal("directions", (cfg.sparse_experts, cfg.hidden_size), 1.0).sign()


def _router(cfg):
    """One direction per expert, scaled so that a chosen expert scores about 4."""
    rms = math.sqrt(1 + cfg.num_experts_per_tok * 1.35)
    return (_directions(cfg).float() * (4 * rms / cfg.hidden_size)).bfloat16()


_models = weakref.WeakValueDictionary()


def _model(case):
    key = (case["model"], case["layers"], case["dtype"], case["kv"], case["mode"] in _CHOOSING)
    m = _models.get(key)
    if m is None:
        cfg = _config(case)
        os.environ["XFT_FAKE_MODEL"] = "2"
        Env.get().reload()
        with tempfile.TemporaryDirectory(prefix="xft_cases_") as path:
            config_only(path, cfg)
            m = _models[key] = xft.AutoModel.from_pretrained(path, dtype=case["dtype"], kv_cache_dtype=case["kv"])
        decoder = m.model.decoder
        wte, head = _ends(case, cfg)
        decoder.wte.copy_(wte)
        decoder.lm_head.w.copy_(head)
        for layer in decoder.layers:
            if hasattr(layer, "router"):
                layer.router.w.copy_(_router(cfg))
        del wte, head
        # what a server does before it opens: one short request (scratch memory, layouts of packed experts)
        ids = m.set_input_cb([[1, 2, 3]], None, 8)
        m.forward_cb()
        m.free_seqs(ids)
    return m


def prepare(case, seed):
    prompts, steps = _tokens(case, seed)
    if case["mode"] in ("generate", "score"):
        prompts = torch.tensor(prompts)
    return {"model": _model(case), "mode": case["mode"], "prompts": prompts, "steps": steps, "new": case["new"],
            "max_length": case["prompt"] + case["new"] + 1}


def run(state):
    m = state["model"]
    if state["mode"] == "score":
        return m(state["prompts"])
    if state["mode"] == "generate":
        out = m.generate(state["prompts"], max_length=state["max_length"] - 1, eos_token_id=-2, pad_token_id=0)
        return out, m(out)
    greedy = state["mode"] == "greedy"
    ids = m.set_input_cb(state["prompts"], None, state["max_length"], greedy=greedy).tolist()
    if greedy:
        chosen = [m.forward_cb_greedy()]
        for _ in range(state["new"] - 1):
            m.set_input_cb(chosen[-1].tolist(), ids, greedy=True)
            chosen.append(m.forward_cb_greedy())
        m.set_input_cb(chosen[-1].tolist(), ids)
        out = torch.stack(chosen), m.forward_cb()
    else:
        out = [m.forward_cb()]
        for step in state["steps"]:
            m.set_input_cb(step, ids)
            out.append(m.forward_cb())
    m.free_seqs(ids)
    return out


# -- what a pass cannot do without --------------------------------------------------------------------------------------
_BYTES = {"bf16": 2.0, "w8a8": 1.0, "int8": 1.0, "int4": 0.5, "fp8_e4m3": 1.0}


def _passes(case):
    """(new tokens, contexts after them, rows of logits) of each forward of a pass."""
    lens, B = _lens(case), case["batch"]
    if case["mode"] == "score":
        return [(lens, lens, sum(lens))]
    out = [(lens, lens, B)]
    steps = case["new"] - 1 + (case["mode"] == "greedy")
    out += [([1] * B, [n + s + 1 for n in lens], B) for s in range(steps)]
    if case["mode"] == "generate":
        full = [n + case["new"] for n in lens]
        out.append((full, full, sum(full)))
    return out


def work(case):
    cfg = _config(case)
    H, V, L, heads = cfg.hidden_size, cfg.vocab_size, cfg.num_layer, cfg.head_num
    wb = _BYTES[case["dtype"]]
    bytes_, flops = 0.0, 0.0
    for new, ctx, rows in _passes(case):
        T = sum(new)
        pairs = sum(n * c - n * (n - 1) / 2 for n, c in zip(new, ctx))       # (query, visible key) pairs
        for i in range(L):
            if case["model"] == "deepseek-v3":
                nope, rot, vd, r, ql = cfg.qk_nope_head_dim, cfg.qk_rope_head_dim, cfg.v_head_dim, cfg.kv_lora_rank, cfg.q_lora_rank
                w = H * (ql + r + rot) + ql * heads * (nope + rot) + r * heads * (nope + vd) + heads * vd * H
                kv, score = (r + rot) * 2.0, 2.0 * heads * (nope + rot + vd)
            else:
                D = cfg.size_per_head
                w = H * (heads + 2 * cfg.kv_head_num) * D + heads * D * H
                kv = 2.0 * cfg.kv_head_num * (D * 2.0 if case["kv"] == "bf16" else D + 4.0)
                score = 4.0 * heads * D
            read = mults = w
            if cfg.model_type in _MOE and not (case["model"] == "deepseek-v3" and i < cfg.first_k_dense_replace):
                E, k, I = cfg.sparse_experts, cfg.num_experts_per_tok, cfg.moe_intermediate_size or cfg.inter_size
                read += 3.0 * H * I * (E * (1 - (1 - k / E) ** T) + cfg.dense_experts) + H * E
                mults += 3.0 * H * I * (k + cfg.dense_experts) + H * E
            else:
                read += 3.0 * H * cfg.inter_size
                mults += 3.0 * H * cfg.inter_size
            bytes_ += read * wb + kv * (sum(ctx) + T)
            flops += 2.0 * mults * T + score * pairs
        bytes_ += 2.0 * H * T + 2.0 * V * H + (4.0 * V * rows)
        flops += 2.0 * V * H * rows
    return {"bytes": bytes_, "flops": flops}


# -- the same numbers in 64 bits ----------------------------------------------------------------------------------------
def _quantised(w, dtype):
    """The values that a quantised product stands for: one scale and offset per output row, or per 128 x 128 block (e4m3)."""
    if dtype == "bf16":
        return w.double()
    w = w.float()
    if dtype == "fp8_e4m3":
        o, i = w.shape
        p = torch.zeros((o + 127) // 128 * 128, (i + 127) // 128 * 128, device=w.device)
        p[:o, :i] = w
        b = p.view(p.shape[0] // 128, 128, p.shape[1] // 128, 128)
        s = b.abs().amax(dim=(1, 3), keepdim=True).clamp_min(1e-12) / 448.0
        return ((b / s).to(torch.float8_e4m3fn).double() * s.double()).view(p.shape)[:o, :i]
    hi, lo = w.amax(1, keepdim=True), w.amin(1, keepdim=True)
    if dtype == "int4":
        s, z, a, e = (hi - lo) / 15.0, lo, 0, 15
    else:
        s = (hi - lo) / 255.0
        z, a, e = (hi + lo) / 2.0 + 0.5 * s, -128, 127
    return torch.round((w - z) / s).clamp_(a, e).double() * s.double() + z.double()


class _Exact:
    """The model in plain torch and 64 bits, weights drawn again by name."""

    def __init__(self, case):
        self.c, self.cfg = case, _config(case)
        self.kind = case["dtype"]

    def w(self, name, o, k, kind=None):
        return _quantised(_normal(name, (o, k)), kind or self.kind)

    def norm(self, x):
        return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + self.cfg.layernorm_eps)

    def angles(self, pos, dim):
        r, half = self.cfg.rope, dim // 2
        f = r.theta ** (-torch.arange(0, dim, 2, dtype=torch.float64, device="cuda") / dim)
        if r.scaling_type == "yarn":
            at = lambda turns: dim * math.log(r.original_max_pos / (turns * 2 * math.pi)) / (2 * math.log(r.theta))
            lo, hi = max(math.floor(at(r.beta_fast)), 0), min(math.ceil(at(r.beta_slow)), dim - 1)
            keep = 1 - ((torch.arange(half, dtype=torch.float64, device="cuda") - lo) / max(hi - lo, 1e-3)).clamp(0, 1)
            f = f / r.scaling_factor * (1 - keep) + f * keep
        a = pos.double()[:, None] * f
        return a.cos()[:, None], a.sin()[:, None]

    def turn(self, x, cs, interleaved=False):
        c, s = cs
        if interleaved:
            a, b = x[..., 0::2], x[..., 1::2]
            return torch.stack([a * c - b * s, b * c + a * s], -1).flatten(-2)
        a, b = x.chunk(2, -1)
        return torch.cat([a * c - b * s, b * c + a * s], -1)

    def attend(self, q, k, v, scale):
        """q [n, h, d], k and v [n, h', d]: causal."""
        out = torch.empty(q.shape[0], q.shape[1], v.shape[2], dtype=torch.float64, device="cuda")
        g = q.shape[1] // k.shape[1]
        for h in range(q.shape[1]):
            for r in range(0, q.shape[0], 4096):
                s = q[r:r + 4096, h] @ k[:r + 4096, h // g].T * scale
                s.masked_fill_(torch.ones_like(s, dtype=torch.bool).triu_(r + 1), float("-inf"))
                out[r:r + 4096, h] = torch.softmax(s, -1) @ v[:r + 4096, h // g]
        return out.flatten(1)

    def gated(self, x, g, u, d, act="silu"):
        out = torch.empty(x.shape[0], d.shape[0], dtype=torch.float64, device="cuda")
        for r in range(0, x.shape[0], 8192):
            y = x[r:r + 8192]
            a = y @ g.T
            a = torch.nn.functional.silu(a) if act == "silu" else torch.nn.functional.gelu(a, approximate="tanh")
            out[r:r + 8192] = (a * (y @ u.T)) @ d.T
        return out

    def experts(self, p, h):
        cfg, E = self.cfg, self.cfg.sparse_experts
        H, I = cfg.hidden_size, cfg.moe_intermediate_size or cfg.inter_size
        if cfg.model_type == "mixtral":
            logits = h @ _router(cfg).double().T
            val, idx = logits.topk(cfg.num_experts_per_tok, -1)
            wt = torch.softmax(val, -1)
            names = lambda e: [p + f"moe.sparse_experts.{e}.w{j}.0.bin" for j in (1, 2, 3)]
        else:
            score = torch.sigmoid(h @ _router(cfg).double().T)
            sel = score + _normal(p + "mlp.gate.e_score_correction_bias.bin", (E,), dtype=torch.float32).double()
            groups = sel.view(-1, cfg.n_group, E // cfg.n_group)
            best = groups.topk(2, -1)[0].sum(-1).topk(cfg.topk_group, -1)[1]
            mask = torch.zeros(groups.shape[:2], dtype=torch.bool, device="cuda").scatter_(1, best, True)
            sel = groups.masked_fill(~mask[..., None], float("-inf")).flatten(1)
            idx = sel.topk(cfg.num_experts_per_tok, -1)[1]
            wt = score.gather(1, idx)
            wt = wt / wt.sum(-1, keepdim=True) * cfg.routed_scaling_factor
            names = lambda e: [p + f"mlp.experts.{e}.{n}_proj.weight.bin" for n in ("gate", "up", "down")]
        out = torch.zeros_like(h)
        for e in range(E):
            t, j = (idx == e).nonzero(as_tuple=True)
            if t.numel():
                g, u, d = names(e)
                y = self.gated(h[t], self.w(g, I, H), self.w(u, I, H), self.w(d, H, I))
                out.index_add_(0, t, y * wt[t, j][:, None])
        if cfg.dense_experts:
            n = [p + f"mlp.shared_experts.{x}_proj.weight.bin" for x in ("gate", "up", "down")]
            S = cfg.dense_experts * I
            out += self.gated(h, self.w(n[0], S, H), self.w(n[1], S, H), self.w(n[2], H, S))
        return out

    def layer(self, i, x, pos, spans):
        cfg, p = self.cfg, f"model.layers.{i}."
        H, heads = cfg.hidden_size, cfg.head_num
        h = self.norm(x)
        if cfg.model_type == "deepseek_moe":
            nope, rot, vd, r, ql = cfg.qk_nope_head_dim, cfg.qk_rope_head_dim, cfg.v_head_dim, cfg.kv_lora_rank, cfg.q_lora_rank
            a = p + "self_attn."
            cs = self.angles(pos, rot)
            q = (self.norm(h @ self.w(a + "q_a_proj.weight.bin", ql, H).T) @ self.w(a + "q_b_proj.weight.bin", heads * (nope + rot), ql).T)
            q = q.view(-1, heads, nope + rot)
            lat = h @ self.w(a + "kv_a_proj_with_mqa.weight.bin", r + rot, H).T
            kvb = (self.norm(lat[:, :r]) @ self.w(a + "kv_b_proj.weight.bin", heads * (nope + vd), r).T).view(-1, heads, nope + vd)
            q = torch.cat([q[..., :nope], self.turn(q[..., nope:], cs, True)], -1)
            k = torch.cat([kvb[..., :nope], self.turn(lat[:, None, r:], cs, True).expand(-1, heads, -1)], -1)
            m = 0.1 * cfg.rope.mscale_all_dim * math.log(cfg.rope.scaling_factor) + 1.0
            o = torch.cat([self.attend(q[s:e], k[s:e], kvb[s:e, :, nope:], (nope + rot) ** -0.5 * m * m) for s, e in spans])
            x = x + o @ self.w(p + "attention.dense.weight.bin", H, heads * vd).T
        else:
            D, kvh = cfg.size_per_head, cfg.kv_head_num
            y = h @ self.w(p + "attention.query_key_value.weight.0.bin", (heads + 2 * kvh) * D, H).T
            if cfg.model_type == "qwen2":
                y = y + _normal(p + "attention.query_key_value.bias.0.bin", ((heads + 2 * kvh) * D,), dtype=torch.float32).double()
            q, k, v = y.view(-1, heads + 2 * kvh, D).split([heads, kvh, kvh], 1)
            cs = self.angles(pos, D)
            q, k = self.turn(q, cs), self.turn(k, cs)
            o = torch.cat([self.attend(q[s:e], k[s:e], v[s:e], D ** -0.5) for s, e in spans])
            x = x + o @ self.w(p + "attention.dense.weight.0.bin", H, heads * D).T
        h = self.norm(x)
        if cfg.model_type in _MOE and not (cfg.model_type == "deepseek_moe" and i < cfg.first_k_dense_replace):
            return x + self.experts(p, h)
        end = ".weight.bin" if cfg.model_type == "deepseek_moe" else ".weight.0.bin"
        g, u, d = (self.w(p + f"mlp.{n}_proj" + end, *((H, cfg.inter_size) if n == "down" else (cfg.inter_size, H))) for n in ("gate", "up", "down"))
        return x + self.gated(h, g, u, d, "gelu" if cfg.activation_type == "gelu" else "silu")

    def logits(self, seqs, rows):
        """Logits of the places `rows[i]` of sequence i, sequence after sequence."""
        cfg = self.cfg
        wte, head = _ends(self.c, cfg)
        spans, pos, at, want = [], [], 0, []
        for s, r in zip(seqs, rows):
            spans.append((at, at + len(s)))
            pos += range(len(s))
            want += [at + j for j in r]
            at += len(s)
        pos = torch.tensor(pos, device="cuda")
        x = wte[torch.tensor([t for s in seqs for t in s], device="cuda")].double()
        if cfg.model_type == "gemma":
            x = x * math.sqrt(cfg.hidden_size)
        for i in range(cfg.num_layer):
            x = self.layer(i, x, pos, spans)
        return self.norm(x[torch.tensor(want, device="cuda")]) @ head.double().T


@torch.no_grad()
def exact(case, seed):
    prompts, steps = _tokens(case, seed)
    m, B, V = _Exact(case), case["batch"], _config(case).vocab_size
    if case["mode"] == "score":
        y = m.logits(prompts, [range(len(p)) for p in prompts])
        return y.view(B, -1, V)
    if case["mode"] in _CHOOSING:
        seqs = [p + [(p[-1] + 1 + j) % V for j in range(case["new"])] for p in prompts]      # the head's order
        if case["mode"] == "generate":
            return torch.tensor(seqs), m.logits(seqs, [range(len(s)) for s in seqs]).view(B, -1, V)
        return torch.tensor([s[-case["new"]:] for s in seqs]).t().contiguous(), m.logits(seqs, [[len(s) - 1] for s in seqs])
    seqs = [p + [s[i] for s in steps] for i, p in enumerate(prompts)]
    y = m.logits(seqs, [range(len(p) - 1, len(q)) for p, q in zip(prompts, seqs)]).view(B, case["new"], V)
    return list(y.transpose(0, 1))


def tolerance(case):
    return {"rel": 0.03, "max": 0.5, "differ": 0.0}
