"""The work a user of this engine has it do, as cases that can be timed and checked.

A case names a design, its layer sizes (those of ``bench.py``'s configurations and of the tests' tiny model), a data
type, a number of requests with lengths between ``shortest`` and ``longest``, and one of two ways to call the engine:

* ``prompt``: ``Engine.step`` on whole prompts, as a program does that scores text or fills a cache; the logits of
  ``wanted`` places a request come back.
* ``serve``: the requests are submitted together and ``Engine.run_step`` is called until all have ended, as a serving
  program does: prompts in portions beside decoded tokens, replayed decode steps, sampling.  The tokens of every
  request and the logits behind each request's last token come back.

Weights are drawn here, in distributions like a trained model's where that matters: the residual stream is dominated
by the embedding, the router's rows are directions the embeddings hold (so a token's experts are clear, and all
experts are used), an output matrix that gives each token a clear successor (so greedy and sampled text is the same
for every correct implementation), decay parameters over the ranges such layers are initialised and trained in.
"""
import math
import random
import re
import zlib

import numpy as np
import torch

from dlm_b200.engine import Engine, make_runtime
from dlm_b200.parts.model import DecoderModel
from dlm_b200.registry import resolve
from dlm_b200.sampling import SamplingParams

PAGE = 64
STEP = 2048          # the engine's default budget of tokens a step


# ------------------------------------------------------------------------------------------------- the cases
def listed():
    moe = {"design": "qwen2_moe", "width": 2048, "dtype": "bfloat16"}
    return [
        # the smallest call: the tiny configuration in 32-bit, four ragged prompts in one step (launches and host only)
        dict(name="tiny_f32_prompts", design="qwen2_moe", width=64, layers=2, dtype="float32", how="prompt", requests=4,
             shortest=1, longest=33, wanted=1),
        # one user at a terminal: a short prompt, then single-row decode steps (latency)
        dict(moe, name="chat_1", layers=4, how="serve", requests=1, shortest=128, longest=128, new=48, temperature=0.0),
        # the headline: all 24 layers, eight requests of 1,024 tokens, decoded together
        dict(moe, name="decode_8_all_layers", layers=24, how="serve", requests=8, shortest=1024, longest=1024, new=64,
             temperature=0.0),
        # a busy server: 64 short ragged prompts, sampled
        dict(moe, name="serve_64_sampled", layers=4, how="serve", requests=64, shortest=16, longest=256, new=32,
             temperature=0.8),
        # one prompt of the default step budget
        dict(moe, name="prompt_2048", layers=4, how="prompt", requests=1, shortest=2048, longest=2048, wanted=1),
        # ragged prompts of odd lengths batched in one step
        dict(moe, name="prompts_ragged", layers=4, how="prompt", requests=6, shortest=17, longest=601, wanted=1),
        # long documents in portions of the step budget beside decoding requests; the last layer looks through a window
        dict(moe, name="long_documents", layers=4, how="serve", requests=3, shortest=2311, longest=10240, new=16,
             temperature=0.0),
        # the 32-bit path at real layer sizes: a few ragged prompts and some decoded tokens
        dict(moe, name="f32_requests", dtype="float32", layers=2, how="serve", requests=4, shortest=33, longest=400,
             new=8, temperature=0.0),
        # state-space scan, latent attention with a window, delta rule: a prompt of the default step budget
        dict(design="zesapel", width=2048, dtype="bfloat16", layers=3, name="zesapel_prompt", how="prompt", requests=1,
             shortest=2048, longest=2048, wanted=8),
        # selective scan, retention beside attention with a distance penalty, experts: three ragged prompts
        dict(design="zasazen", width=2048, dtype="bfloat16", layers=3, name="zasazen_prompts", how="prompt", requests=3,
             shortest=203, longest=1101, wanted=8),
        # gated delta rule, latent attention over everything, chunked attention beside gated linear attention
        dict(design="salolorn", width=2048, dtype="bfloat16", layers=3, name="salolorn_prompt", how="prompt",
             requests=1, shortest=1900, longest=1900, wanted=8),
        # eight requests of a recurrent design through the scheduler: ragged prompts, then decode steps
        dict(design="salolorn", width=1024, dtype="bfloat16", layers=3, name="salolorn_serve", how="serve", requests=8,
             shortest=60, longest=500, new=32, temperature=0.0),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["tiny", "prompt", "prompt", "serve", "serve", "serve", "f32", "zesapel", "zasazen", "salolorn",
                       "recurrent_serve"])
    if kind == "tiny":
        n = rng.randint(1, 8)
        return dict(design="qwen2_moe", width=64, layers=2, dtype=rng.choice(["float32", "bfloat16"]), how="prompt",
                    requests=n, shortest=rng.randint(1, 5), longest=_log_uniform(rng, 6, 120), wanted=1)
    if kind in ("prompt", "zesapel", "zasazen", "salolorn"):
        total = _log_uniform(rng, 100, 2048)
        n = min(rng.choice([1, 1, 2, 3, 5, 12]), total // 17)
        longest = total if n == 1 else min(total, max(17, int(1.5 * total / n)))
        shortest = longest if n == 1 else max(1, 2 * total // n - longest)
        if kind == "prompt":
            return dict(design="qwen2_moe", width=2048, layers=rng.choice([2, 4]), dtype="bfloat16", how="prompt",
                        requests=n, shortest=shortest, longest=longest, wanted=1)
        return dict(design=kind, width=rng.choice([1024, 2048]), layers=3, dtype="bfloat16", how="prompt", requests=n,
                    shortest=shortest, longest=longest, wanted=8)
    if kind == "f32":
        return dict(design="qwen2_moe", width=2048, layers=2, dtype="float32", how="serve", requests=rng.randint(1, 4),
                    shortest=rng.randint(1, 33), longest=_log_uniform(rng, 40, 400), new=rng.randint(2, 8),
                    temperature=0.0)
    if kind == "recurrent_serve":
        return dict(design=rng.choice(["zesapel", "zasazen", "salolorn"]), width=1024, layers=3, dtype="bfloat16",
                    how="serve", requests=_log_uniform(rng, 1, 16), shortest=_log_uniform(rng, 20, 60),
                    longest=_log_uniform(rng, 64, 500), new=rng.randint(8, 32), temperature=0.0)
    n = _log_uniform(rng, 1, 64)
    longest = _log_uniform(rng, 32, min(10240, 16384 // n))
    return dict(design="qwen2_moe", width=2048, layers=rng.choice([2, 4]), dtype="bfloat16", how="serve", requests=n,
                shortest=max(1, longest // rng.randint(1, 9)), longest=longest, new=rng.randint(8, 48),
                temperature=rng.choice([0.0, 0.0, 0.8]))


def lengths(case):
    """The requests' prompt lengths: evenly spread from the longest to the shortest, interleaved."""
    n = case["requests"]
    out = [case["longest"] if n == 1 else round(case["longest"] + (case["shortest"] - case["longest"]) * i / (n - 1))
           for i in range(n)]
    return out[::2] + out[1::2]


def wanted_places(case, n):
    w = min(case["wanted"], n)
    return sorted({n - 1 - (n * i) // w for i in range(w)})


# ---------------------------------------------------------------------------------- configurations and tensors
def config(case):
    """The ``config.json`` of a case, as a dict."""
    W, L = case["width"], case["layers"]
    if case["design"] == "qwen2_moe":
        base = dict(architectures=["Qwen2MoeForCausalLM"], model_type="qwen2_moe", num_hidden_layers=L, hidden_size=W,
                    decoder_sparse_step=1, norm_topk_prob=False, rms_norm_eps=1e-6, tie_word_embeddings=False,
                    max_position_embeddings=16384)
        if W == 64:
            return dict(base, num_attention_heads=4, num_key_value_heads=2, head_dim=16, num_experts=8,
                        num_experts_per_tok=2, moe_intermediate_size=32, shared_expert_intermediate_size=64,
                        intermediate_size=128, vocab_size=256, rope_theta=10000.0, use_sliding_window=False)
        return dict(base, num_attention_heads=16, num_key_value_heads=16, head_dim=128, num_experts=60,
                    num_experts_per_tok=4, moe_intermediate_size=1408, shared_expert_intermediate_size=5632,
                    intermediate_size=5632, vocab_size=151936, rope_theta=1e6, use_sliding_window=True,
                    sliding_window=4096, max_window_layers=max(1, L * 7 // 8))
    base = {"vocab": 32768, "width": W, "max_positions": 8192}
    if case["design"] == "zesapel":
        mlp = {"kind": "moe", "router": {"experts": W // 64, "top": 2}, "expert": {"ff": W}}
        return dict(base, architecture="Zesapel", streams=4, embedding={"scale": 1.0}, norm={"eps": 1e-5},
                    canon={"taps": 4}, layers=[
                        {"type": "general_delta", "mixer": {"heads": W // 64, "dim": 64}, "mlp": mlp},
                        {"type": "mamba2", "mlp": mlp, "mixer": {"heads": W // 32, "vdim": 64, "state": 128, "groups": 1,
                                                                 "conv": 4, "norm_groups": 1}},
                        {"type": "latent_attention", "mlp": mlp, "mixer": {
                            "heads": W // 128, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": 512, "q_rank": 768,
                            "mask": {"size": 1024}, "rot": {"base": 10000.0, "dims": 64}, "scale": 192 ** -0.5}}])
    if case["design"] == "zasazen":
        hr = W // 128
        pair = {"type": "parallel", "mixer": {
            "left": {"heads": W // 64, "kv_heads": W // 256, "dim": 64, "vdim": 64, "scale": 0.125,
                     "q_temp": {"coef": 0.5, "every": 512}},
            "right": {"heads": hr, "dim": 64, "vdim": 128, "rot": {"base": 1e6, "dims": 64},
                      "decay": [1.0 - 2.0 ** (-5 - 5 * i / (hr - 1)) for i in range(hr)]}}}
        scan = {"type": "mamba1", "mixer": {"inner": 2 * W, "state": 16, "dt_rank": W // 16, "conv": 4}}
        moe = {"kind": "moe", "router": {"experts": 16, "top": 2}, "expert": {"ff": W // 2}, "shared": {"ff": W}}
        dense = {"kind": "dense", "ff": 4 * W}
        return dict(base, architecture="Zasazen", embedding={"scale": 1.0}, norm={"eps": 1e-5},
                    loop={"start": 1, "stop": 3, "times": 2},
                    layers=[dict(pair, mlp=dense), dict(pair, mlp=moe), dict(scan, mlp=moe)])
    dense = {"kind": "dense", "ff": 3 * W}
    return dict(base, architecture="Salolorn", norm={"eps": 1e-6}, logit_scale=W ** -0.5,
                loop={"start": 1, "stop": 3, "times": 2}, layers=[
                    {"type": "delta", "mlp": dense, "mixer": {"heads": W // 128, "kv_heads": W // 256, "dim": 128,
                                                              "vdim": 128, "conv": 4}},
                    {"type": "latent_attention", "mlp": dense, "mixer": {
                        "heads": W // 128, "dim": 128, "rot_dim": 64, "vdim": 128, "kv_rank": 512, "scale": 192 ** -0.5,
                        "rot": {"base": 10000.0, "dims": 64}}},
                    {"type": "parallel", "mlp": dense, "mixer": {
                        "left": {"heads": W // 64, "kv_heads": W // 256, "dim": 64, "vdim": 64, "scale": 0.125,
                                 "mask": {"size": 2048}, "rot": {"base": 1e6, "dims": 64}},
                        "right": {"heads": W // 128, "dim": 64, "vdim": 128, "tau": 16.0},
                        "left_scale": 1.0, "right_scale": 1.0}}])


def vocabulary(cfg):
    return cfg.get("vocab_size") or cfg["vocab"]


def shapes(cfg):
    """Name -> shape of every tensor of a model folder with this configuration."""
    out = {}
    if cfg.get("model_type") == "qwen2_moe":
        H, V, E = cfg["hidden_size"], cfg["vocab_size"], cfg["num_experts"]
        Q, KV = cfg["num_attention_heads"] * cfg["head_dim"], cfg["num_key_value_heads"] * cfg["head_dim"]
        ffs = [(f"experts.{e}", cfg["moe_intermediate_size"]) for e in range(E)]
        ffs.append(("shared_expert", cfg["shared_expert_intermediate_size"]))
        for i in range(cfg["num_hidden_layers"]):
            p = f"model.layers.{i}."
            for n, o in (("q", Q), ("k", KV), ("v", KV)):
                out[f"{p}self_attn.{n}_proj.weight"], out[f"{p}self_attn.{n}_proj.bias"] = (o, H), (o,)
            out[p + "self_attn.o_proj.weight"] = (H, Q)
            out[p + "input_layernorm.weight"] = out[p + "post_attention_layernorm.weight"] = (H,)
            out[p + "mlp.gate.weight"], out[p + "mlp.shared_expert_gate.weight"] = (E, H), (1, H)
            for n, f in ffs:
                out[f"{p}mlp.{n}.gate_proj.weight"] = out[f"{p}mlp.{n}.up_proj.weight"] = (f, H)
                out[f"{p}mlp.{n}.down_proj.weight"] = (H, f)
        return dict(out, **{"model.embed_tokens.weight": (V, H), "model.norm.weight": (H,), "lm_head.weight": (V, H)})
    W, V, design = cfg["width"], cfg["vocab"], cfg["architecture"]
    out.update({"embed": (V, W), "final.norm": (W,)})
    if design != "Salolorn":
        out["head"] = (V, W)
    if design == "Zesapel":
        out["pos"] = (cfg["max_positions"], W)
    if cfg.get("loop"):
        out["loop.step"] = (cfg["loop"]["times"], W)
        if design == "Zasazen":
            out["loop.in"] = (W, 2 * W)
    for i, layer in enumerate(cfg["layers"]):
        m, p, mlp = layer["mixer"], f"l{i}.", layer["mlp"]
        x = p + "mix."
        out[p + "norm1"] = out[p + "norm2"] = (W,)
        if design == "Salolorn":
            out[p + "norm1b"] = out[p + "norm2b"] = (W,)
        if design == "Zesapel":
            S = cfg["streams"]
            for q in "12":
                out[f"{p}hc{q}.in"] = out[f"{p}hc{q}.out"] = (S,)
                out[f"{p}hc{q}.mix"] = (S, S)
            out[p + "canon1"] = (W, cfg["canon"]["taps"])
        if layer["type"] == "general_delta":
            D = m["heads"] * m["dim"]
            out.update({x + n: (D, W) for n in ("r", "k", "v", "a", "g")})
            out.update({x + "a.b": (D,), x + "w1": (16, W), x + "w2": (D, 16), x + "w0": (D,), x + "norm": (D,),
                        x + "o": (W, D)})
        elif layer["type"] == "mamba2":
            D, C = m["heads"] * m["vdim"], m["heads"] * m["vdim"] + 2 * m["groups"] * m["state"]
            out.update({x + "in": (D + C + m["heads"], W), x + "conv": (C, m["conv"]), x + "conv.b": (C,),
                        x + "dt_bias": (m["heads"],), x + "A_log": (m["heads"],), x + "D": (m["heads"],),
                        x + "norm": (D,), x + "o": (W, D)})
        elif layer["type"] == "mamba1":
            D, N, R = m["inner"], m["state"], m["dt_rank"]
            out.update({x + "in": (2 * D, W), x + "conv": (D, m["conv"]), x + "conv.b": (D,), x + "x": (R + 2 * N, D),
                        x + "dt": (D, R), x + "dt.b": (D,), x + "A_log": (D, N), x + "D": (D,), x + "o": (W, D)})
        elif layer["type"] == "latent_attention":
            H, d, r, dv, rank = m["heads"], m["dim"], m["rot_dim"], m["vdim"], m["kv_rank"]
            if "q_rank" in m:
                out.update({x + "dq": (m["q_rank"], W), x + "dq.norm": (m["q_rank"],),
                            x + "uq": (H * (d + r), m["q_rank"]), x + "sink": (H,), x + "g": (H, W)})
            else:
                out[x + "q"] = (H * (d + r), W)
            out.update({x + "dkv": (rank + r, W), x + "dkv.norm": (rank,), x + "uk": (H * d, rank),
                        x + "uv": (H * dv, rank), x + "o": (W, H * dv)})
        elif layer["type"] == "delta":
            H, G, d, dv = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
            for n, o in (("q", G * d), ("k", G * d), ("v", H * dv)):
                out[x + n], out[x + n + ".conv"] = (o, W), (o, m["conv"])
            out.update({x + "b": (H, W), x + "a": (H, W), x + "A_log": (H,), x + "dt_bias": (H,), x + "norm": (dv,),
                        x + "g": (H * dv, W), x + "o": (W, H * dv)})
        else:
            for side in ("left", "right"):
                s, y = m[side], f"{x}{side}."
                H, G = s["heads"], s.get("kv_heads", s["heads"])
                out.update({y + "q": (H * s["dim"], W), y + "k": (G * s["dim"], W), y + "v": (G * s["vdim"], W),
                            y + "o": (W, H * s["vdim"])})
                if side == "right":
                    out[y + "g"] = (H * s["vdim"], W)
                if design == "Zasazen":
                    out[y + "out"] = (W,)
                    if side == "left":
                        out.update({y + "q.b": (H * s["dim"],), y + "k.b": (G * s["dim"],), y + "v.b": (G * s["vdim"],),
                                    y + "q.norm": (H * s["dim"],), y + "k.norm": (G * s["dim"],)})
                elif side == "left":
                    out.update({y + "q.norm": (s["dim"],), y + "k.norm": (s["dim"],), y + "sink": (H,), y + "g": (H, W)})
                else:
                    out.update({y + "a1": (16, W), y + "a2": (H * s["dim"], 16), y + "a2.b": (H * s["dim"],),
                                y + "norm": (s["vdim"],)})
        y = p + "mlp."
        if mlp["kind"] == "dense":
            out[y + "up"], out[y + "down"] = (mlp["ff"], W), (W, mlp["ff"])
            if design == "Salolorn":
                out[y + "gate"] = (mlp["ff"], W)
            continue
        E, f = mlp["router"]["experts"], mlp["expert"]["ff"]
        for e in range(E):
            out[f"{y}e{e}.up"], out[f"{y}e{e}.down"] = (f, W), (W, f)
            if design == "Zasazen":
                out[f"{y}e{e}.gate"] = (f, W)
        if design == "Zesapel":
            out[y + "table"] = (V, mlp["router"]["top"])
        else:
            f = mlp["shared"]["ff"]
            out.update({y + "router": (E, W), y + "router.b": (E,), y + "shared.gate": (f, W), y + "shared.up": (f, W),
                        y + "shared.down": (W, f), y + "shared.sg": (1, W)})
    return out


class Weights:
    """``w(name)``: the tensor of that name, made on the GPU from the seed and the name alone, in the case's type."""

    def __init__(self, case, seed):
        self.case, self.seed, self.cfg = case, int(seed), config(case)
        self.shapes = shapes(self.cfg)
        self.dtype = torch.bfloat16 if case["dtype"] == "bfloat16" else torch.float32
        self.vocab = vocabulary(self.cfg)

    def _gen(self, name):
        return torch.Generator(device="cuda").manual_seed((self.seed * 1000003 + zlib.crc32(name.encode())) % (1 << 62))

    def _randn(self, name, shape, dtype=None):
        return torch.randn(shape, generator=self._gen(name), device="cuda", dtype=dtype or self.dtype)

    def _uniform(self, name, shape, lo, hi):
        return torch.rand(shape, generator=self._gen(name), device="cuda", dtype=torch.float64) * (hi - lo) + lo

    def _topics(self, E):
        W = self.case["width"]
        return self._randn("topics", (E, W), torch.float32) * W ** -0.5

    def successors(self):
        """The token that follows each token (a tied output matrix makes a token follow itself)."""
        if self.cfg.get("architecture") == "Salolorn":
            return torch.arange(self.vocab, device="cuda")
        return torch.argsort(torch.rand(self.vocab, generator=self._gen("successors"), device="cuda"))

    def __call__(self, name):
        return self._values(name, self.shapes[name]).to(self.dtype)

    def _values(self, name, shape):
        if name in ("embed", "model.embed_tokens.weight"):
            x = self._randn(name, shape, torch.float32)
            E, top = self.cfg.get("num_experts"), self.cfg.get("num_experts_per_tok")
            if self.cfg.get("architecture") == "Zasazen":
                E, top = 16, 2
            if E:
                chosen = torch.argsort(torch.rand((shape[0], E), generator=self._gen("chosen"), device="cuda"), dim=1)
                u = self._topics(E)
                for j in range(top):
                    x += 10.0 * u[chosen[:, j]]
            return x.to(self.dtype)
        if name in ("head", "lm_head.weight"):
            e = self("embed" if name == "head" else "model.embed_tokens.weight").float() * shape[1] ** -0.5
            out = torch.empty_like(e)
            out[self.successors()] = e
            return out
        if name.endswith((".mlp.gate.weight", ".router")):        # every layer's experts in another order
            return self._topics(shape[0])[torch.randperm(shape[0], generator=self._gen(name), device="cuda")]
        if name.endswith(".table"):
            E = self.cfg["layers"][0]["mlp"]["router"]["experts"]
            return torch.argsort(torch.rand((shape[0], E), generator=self._gen(name), device="cuda"), dim=1)[:, :shape[1]]
        if name.endswith("A_log"):
            if len(shape) == 2:
                return torch.log(torch.arange(1, shape[1] + 1, device="cuda", dtype=torch.float64)).expand(shape)
            return torch.log(self._uniform(name, shape, 1.0, 16.0))
        if name.endswith((".dt_bias", ".dt.b")):                  # softplus of it: 0.001 to 0.1
            step = torch.exp(self._uniform(name, shape, math.log(1e-3), math.log(1e-1)))
            return step + torch.log(-torch.expm1(-step))
        if name.endswith(".w0"):
            return self._uniform(name, shape, -6.0, -1.0)
        if name.endswith(".a2.b"):
            return self._uniform(name, shape, 0.0, 4.0)
        if name == "loop.in":
            eye = torch.eye(shape[0], device="cuda")
            return torch.cat([eye, 0.5 * eye], dim=1) + 0.25 * shape[1] ** -0.5 * self._randn(name, shape, torch.float32)
        if name.endswith(".mix") and len(shape) == 2 and shape[0] == shape[1]:
            return torch.eye(shape[0], device="cuda") + 0.02 * self._randn(name, shape, torch.float32)
        if re.search(r"(norm\d?|layernorm\.weight|model\.norm\.weight|\.D|hc\d\.(in|out)|(left|right)\.out)$", name):
            return 1.0 + 0.02 * self._randn(name, shape, torch.float32)
        if name.endswith(("norm1b", "norm2b")):
            return 0.3 + 0.02 * self._randn(name, shape, torch.float32)
        if name.endswith(("conv", "canon1")):
            return (0.3 if name.endswith("conv") else 0.1) * self._randn(name, shape)
        if len(shape) == 1 or name in ("pos", "loop.step"):
            return (0.5 if name.endswith("sink") else 0.02) * self._randn(name, shape)
        return shape[-1] ** -0.5 * self._randn(name, shape)

    def prompts(self):
        ids = [torch.randint(0, self.vocab, (n,), generator=self._gen(f"prompt {i}"), device="cuda").tolist()
               for i, n in enumerate(lengths(self.case))]
        return ids


# ------------------------------------------------------------------------------------------- prepare and run
def prepare(case, seed):
    w = Weights(case, seed)
    rt = make_runtime(case["dtype"])
    _, cfg, spec = resolve(w.cfg)
    model = DecoderModel(spec, rt)

    def get(name):
        t = w(name) if not name.endswith(".table") else w._values(name, w.shapes[name])
        return t.to(torch.int32) if name.endswith(".table") else t

    model.load(get, list(w.shapes))
    n, longest = case["requests"], max(lengths(case)) + case.get("new", 0)
    held = sum(-(-(k + case.get("new", 0)) // PAGE) * PAGE for k in lengths(case))
    eng = Engine(cfg, model, page_size=PAGE, max_tokens=held + (n + 2) * PAGE, max_requests=n, max_step_tokens=STEP,
                 max_context=max(256, longest + 1))
    return {"engine": eng, "case": case, "prompts": w.prompts()}


def run(state):
    eng, case, prompts = state["engine"], state["case"], state["prompts"]
    if case["how"] == "prompt":
        slots = [eng.cache.open() for _ in prompts]
        logits = eng.step([(s, p, wanted_places(case, len(p))) for s, p in zip(slots, prompts)])
        for s in slots:
            eng.cache.close(s)
        return {"logits": logits}
    hot = case["temperature"] > 0
    params = dict(temperature=case["temperature"], top_p=0.9 if hot else 1.0, top_k=50 if hot else 0, seed=1)
    ids = [eng.submit(p, SamplingParams(**params), max_new_tokens=case["new"]) for p in prompts]
    seen, last = dict.fromkeys(ids, 0), {}
    while eng.scheduler.has_work():
        for row, (rid, _) in enumerate(eng.run_step()):
            seen[rid] += 1
            if seen[rid] == case["new"]:
                last[rid] = eng.last_logits[row].clone()
    return {"tokens": np.array([eng.result(i) for i in ids], dtype=np.int64), "logits": torch.stack([last[i] for i in ids])}


# ------------------------------------------------------------------------------------------------- work, tolerance
def _runs(cfg):
    """Layers in the order they are run."""
    n = cfg.get("num_hidden_layers") or len(cfg["layers"])
    loop = cfg.get("loop")
    if not loop:
        return list(range(n))
    return [*range(loop["start"]), *list(range(loop["start"], loop["stop"])) * loop["times"], *range(loop["stop"], n)]


def _window(cfg, i):
    if cfg.get("model_type") == "qwen2_moe":
        return cfg["sliding_window"] if cfg.get("use_sliding_window") and i >= cfg["max_window_layers"] else None
    m = cfg["layers"][i]["mixer"]
    return ((m.get("left") or m).get("mask") or {}).get("size")


def work(case):
    """Bytes: every weight a step needs once per step (experts: as many as its tokens choose on average), cached keys
    and states read and written, the logits.  Flops: two per weight and token, scores and mixes of attention, state
    updates and read-outs."""
    cfg = config(case)
    size = 2 if case["dtype"] == "bfloat16" else 4
    prompt, new, V = lengths(case), case.get("new", 1), vocabulary(cfg)
    qwen = cfg.get("model_type") == "qwen2_moe"
    dense, experts = {}, {}
    for name, shape in shapes(cfg).items():
        layer = re.match(r"(?:model\.layers\.|l)(\d+)\.", name)
        if layer and not name.endswith(".table"):
            part = experts if re.search(r"\.(experts\.\d+|e\d+)\.", name) else dense
            part[int(layer.group(1))] = part.get(int(layer.group(1)), 0) + math.prod(shape)

    def layer_sizes(i):
        """(experts, chosen, cached numbers a token, flops a visible key, numbers of state)"""
        if qwen:
            Q, KV = (cfg[k] * cfg["head_dim"] for k in ("num_attention_heads", "num_key_value_heads"))
            return cfg["num_experts"], cfg["num_experts_per_tok"], 2 * KV, 4 * Q, 0
        m, r = cfg["layers"][i]["mixer"], cfg["layers"][i]["mlp"].get("router") or {"experts": 0, "top": 0}
        kind, E, k = cfg["layers"][i]["type"], r["experts"], r["top"]
        if kind == "latent_attention":
            return E, k, m["kv_rank"] + m["rot_dim"], 2 * m["heads"] * (m["dim"] + m["rot_dim"] + m["vdim"]), 0
        if kind == "parallel":
            a, b = m["left"], m["right"]
            return (E, k, a["kv_heads"] * (a["dim"] + a["vdim"]), 2 * a["heads"] * (a["dim"] + a["vdim"]),
                    b["heads"] * b["dim"] * b["vdim"])
        return E, k, 0, 0, (m["inner"] * m["state"] if kind == "mamba1" else
                            m["heads"] * m.get("state", m.get("dim", 0)) * m.get("vdim", m.get("dim", 0)))

    def visible(i, n, first=0):
        w = _window(cfg, i)
        return sum(min(p + 1, w) if w else p + 1 for p in range(first, n))

    steps = [STEP] * (sum(prompt) // STEP) + ([sum(prompt) % STEP] if sum(prompt) % STEP else [])
    if case["how"] == "serve":
        steps += [len(prompt)] * (new - 1)
    logits = sum(len(wanted_places(case, n)) for n in prompt) if case["how"] == "prompt" else len(prompt) * new
    b = f = 0.0
    extra = new - 1 if case["how"] == "serve" else 0
    for i in _runs(cfg):
        E, k, kv, per_key, state = layer_sizes(i)
        for T in steps:
            touched = E * (1.0 - (1.0 - k / E) ** T) if E else 0.0
            b += size * (dense.get(i, 0) + (experts.get(i, 0) / E * touched if E else 0.0))
            f += 2.0 * T * (dense.get(i, 0) + (experts.get(i, 0) / E * k if E else 0.0))
        for n in prompt:
            w = _window(cfg, i)
            b += size * kv * (n + extra) + size * kv * sum(min(n + t, w or n + t) for t in range(1, extra + 1))
            b += 8.0 * state * (1 + extra)
            f += per_key * visible(i, n + extra) + 4.0 * state * (n + extra)
    b += size * V * case["width"] * len([T for T in steps if T]) if case["how"] == "serve" else size * V * case["width"]
    b += 4.0 * logits * V
    f += 2.0 * logits * V * case["width"]
    return {"bytes": b, "flops": f}


def tolerance(case):
    # relative error of the logits, four times what the engine's error against 64 bits was measured to be over all cases
    # (1.3e-6 in 32-bit, 4.5e-3 in bfloat16); tokens are whole numbers that a clear successor decides
    if case["dtype"] == "float32":
        return {"rel": 5e-6, "differ": 0.0}
    return {"rel": 1.8e-2, "differ": 0.005}


# ------------------------------------------------------------------------------------------- exact, in 64 bits
def _rms(x, w, eps):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w


def _silu(x):
    return x * torch.sigmoid(x)


def _conv(x, w):
    out, taps = torch.zeros_like(x), w.shape[1]
    for j in range(taps):
        back = taps - 1 - j
        if back < x.shape[0]:
            out[back:] += x[:x.shape[0] - back] * w[:, j]
    return out


def _rotate(x, base, dims, neighbours=False):
    """x: [T, heads, D]; frequencies and angles are rounded to 32 bits, as the designs say."""
    f = torch.tensor([float(base) ** (-2.0 * i / dims) for i in range(dims // 2)], dtype=torch.float64, device=x.device).float()
    a = (torch.arange(x.shape[0], device=x.device).float()[:, None] * f)[:, None, :].double()
    c, s = torch.cos(a), torch.sin(a)
    if neighbours:
        u, v = x[..., 0:dims:2], x[..., 1:dims:2]
        r = torch.stack([u * c - v * s, v * c + u * s], dim=-1).reshape(*x.shape[:-1], dims)
    else:
        u, v = x[..., :dims // 2], x[..., dims // 2:dims]
        r = torch.cat([u * c - v * s, v * c + u * s], dim=-1)
    return torch.cat([r, x[..., dims:]], dim=-1)


def _attend(q, k, v, scale, window=None, chunk=None, slopes=None, sink=None):
    """q: [T, H, d]; k, v: [T, G, d / dv]; causal.  -> [T, H, dv]"""
    T, H = q.shape[:2]
    G = k.shape[1]
    out = torch.empty(T, H, v.shape[2], dtype=q.dtype, device=q.device)
    j = torch.arange(T, device=q.device)
    rows = max(1, 2048 * 512 // T)
    for a in range(0, T, rows):
        i = torch.arange(a, min(T, a + rows), device=q.device)[:, None]
        see = j[None] <= i
        if window:
            see &= i - j[None] < window
        if chunk:
            see &= i // chunk == j[None] // chunk
        for h in range(H):
            s = q[a:a + rows, h] @ k[:, h * G // H].T * scale
            if slopes is not None:
                s = s - slopes[h] * (i - j[None])
            s = s.masked_fill(~see, float("-inf"))
            m = s.max(-1, keepdim=True).values
            if sink is not None:
                m = torch.maximum(m, sink[h])
            e = torch.exp(s - m)
            den = e.sum(-1, keepdim=True)
            if sink is not None:
                den = den + torch.exp(sink[h] - m)
            out[a:a + rows, h] = e / den @ v[:, h * G // H]
    return out


def _linear_state(q, k, v, decay):
    """S <- decay * S + k v^T; o = S^T q.  q, k: [T, H, d]; v: [T, H, dv]; decay: [T or 1, H, d or 1]."""
    T, H, d = q.shape
    S = torch.zeros(H, d, v.shape[2], dtype=q.dtype, device=q.device)
    o = torch.empty_like(v)
    for t in range(T):
        S = S * decay[t if decay.shape[0] > 1 else 0][:, :, None]
        S += k[t][:, :, None] * v[t][:, None, :]
        o[t] = (q[t][:, None, :] @ S)[:, 0]
    return o


class _Exact:
    def __init__(self, case, seed):
        self.w, self.cfg = Weights(case, seed), config(case)

    def t(self, name):
        return self.w(name).double()

    def logits(self, seqs, places):
        """The logits at ``places[r]`` of every sequence, side by side.  Layer by layer over all sequences, so that a
        layer's weights are made once."""
        w, cfg = self.w, self.cfg
        qwen = cfg.get("model_type") == "qwen2_moe"
        design = "qwen" if qwen else cfg["architecture"]
        emb = self.w("model.embed_tokens.weight" if qwen else "embed")
        ids = [torch.tensor(s, device="cuda") for s in seqs]
        cut = [len(s) for s in seqs]
        x = torch.cat([emb[i].double() for i in ids])
        if design == "Zesapel":
            pos = self.t("pos")
            x = x + torch.cat([pos[:n] for n in cut])
            x = x[None].repeat(cfg["streams"], 1, 1)
        x0, loop, passes = x, cfg.get("loop"), 0
        for i in _runs(cfg):
            if loop and i == loop["start"]:
                step = self.t("loop.step")[passes]
                if design == "Zasazen":
                    x = torch.cat([x, x0], dim=-1) @ self.t("loop.in").T + step
                else:
                    x = (x + x0 if passes else x) + step
                passes += 1
            x = getattr(self, "_" + design.lower())(i, x, cut, torch.cat(ids))
        x = x.sum(0) if design == "Zesapel" else x
        eps = cfg["rms_norm_eps"] if qwen else cfg["norm"]["eps"]
        at = torch.tensor([sum(cut[:r]) + p for r, ps in enumerate(places) for p in ps], device="cuda")
        x = _rms(x[at], self.t("model.norm.weight" if qwen else "final.norm"), eps)
        head = emb if design == "Salolorn" else w("lm_head.weight" if qwen else "head")
        return torch.cat([x @ part.double().T for part in head.split(16384)], dim=1) * cfg.get("logit_scale", 1.0)

    @staticmethod
    def _each(cut, fn, *rows):
        """fn on every sequence's rows by itself."""
        return torch.cat([fn(*p) for p in zip(*(r.split(cut) for r in rows))])

    def _gated(self, h, name, act=_silu, names=("gate_proj.weight", "up_proj.weight", "down_proj.weight")):
        return (act(h @ self.t(name + names[0]).T) * (h @ self.t(name + names[1]).T)) @ self.t(name + names[2]).T

    def _qwen(self, i, x, cut, ids):
        cfg, p = self.cfg, f"model.layers.{i}."
        nh, nkv, hd, eps = (cfg[k] for k in ("num_attention_heads", "num_key_value_heads", "head_dim", "rms_norm_eps"))
        h = _rms(x, self.t(p + "input_layernorm.weight"), eps)
        q, k, v = (h @ self.t(f"{p}self_attn.{n}_proj.weight").T + self.t(f"{p}self_attn.{n}_proj.bias") for n in "qkv")

        def one(q, k, v):
            q, k = (_rotate(a.view(a.shape[0], -1, hd), cfg["rope_theta"], hd) for a in (q, k))
            return _attend(q, k, v.view(-1, nkv, hd), hd ** -0.5, _window(cfg, i)).reshape(-1, nh * hd)

        x = x + self._each(cut, one, q, k, v) @ self.t(p + "self_attn.o_proj.weight").T
        h = _rms(x, self.t(p + "post_attention_layernorm.weight"), eps)
        prob, idx = torch.softmax(h @ self.t(p + "mlp.gate.weight").T, -1).topk(cfg["num_experts_per_tok"], dim=-1)
        y = torch.sigmoid(h @ self.t(p + "mlp.shared_expert_gate.weight").T) * self._gated(h, p + "mlp.shared_expert.")
        for e in range(cfg["num_experts"]):
            row, slot = (idx == e).nonzero(as_tuple=True)
            if row.numel():
                y.index_add_(0, row, prob[row, slot][:, None] * self._gated(h[row], f"{p}mlp.experts.{e}."))
        return x + y

    def _latent(self, h, cut, m, p, eps, neighbours):
        H, d, r, rank = m["heads"], m["dim"], m["rot_dim"], m["kv_rank"]
        q = h @ self.t(p + "q").T if "q_rank" not in m else \
            _rms(h @ self.t(p + "dq").T, self.t(p + "dq.norm"), eps) @ self.t(p + "uq").T
        low = h @ self.t(p + "dkv").T
        c = _rms(low[:, :rank], self.t(p + "dkv.norm"), eps)
        k, v = c @ self.t(p + "uk").T, c @ self.t(p + "uv").T
        sink = self.t(p + "sink") if "q_rank" in m else None

        def one(q, k, v, kr):
            q = q.view(-1, H, d + r)
            rot = [_rotate(a, m["rot"]["base"], r, neighbours) for a in (q[..., d:], kr[:, None])]
            q = torch.cat([q[..., :d], rot[0]], -1)
            k = torch.cat([k.view(-1, H, d), rot[1].expand(-1, H, -1)], -1)
            return _attend(q, k, v.view(-1, H, m["vdim"]), m["scale"], (m.get("mask") or {}).get("size"),
                           sink=sink).reshape(-1, H * m["vdim"])

        o = self._each(cut, one, q, k, v, low[:, rank:])
        if "q_rank" in m:
            o = (o.view(-1, H, m["vdim"]) * torch.sigmoid(h @ self.t(p + "g").T)[:, :, None]).reshape(o.shape)
        return o @ self.t(p + "o").T

    def _zesapel(self, i, xs, cut, ids):
        cfg, p = self.cfg, f"l{i}."
        eps, layer = cfg["norm"]["eps"], cfg["layers"][i]
        m, x = layer["mixer"], p + "mix."

        def ssm(h):
            H, P, N = m["heads"], m["vdim"], m["state"]
            inner, proj = H * P, h @ self.t(x + "in").T
            z, xbc, dt = proj.split([inner, inner + 2 * N, H], dim=1)
            conv = self.t(x + "conv")
            xbc = _silu(self._each(cut, lambda a: _conv(a, conv), xbc) + self.t(x + "conv.b"))
            dt = torch.nn.functional.softplus(dt + self.t(x + "dt_bias"), threshold=100.0)
            A, D = -torch.exp(self.t(x + "A_log")), self.t(x + "D")

            def one(xbc, dt):
                T = xbc.shape[0]
                v = xbc[:, :inner].view(T, H, P)
                B, C = (a[:, None].expand(T, H, N) for a in (xbc[:, inner:inner + N], xbc[:, inner + N:]))
                o = _linear_state(C, dt[:, :, None] * B, v, torch.exp(A * dt)[:, :, None])
                return (o + D[:, None] * v).reshape(T, inner)

            return _rms(self._each(cut, one, xbc, dt) * _silu(z), self.t(x + "norm"), eps) @ self.t(x + "o").T

        def delta(h):
            H, d = m["heads"], m["dim"]
            r, k, v, a, g = (h @ self.t(x + n).T for n in "rkvag")
            a = torch.sigmoid(a + self.t(x + "a.b"))
            lw = torch.tanh(h @ self.t(x + "w1").T) @ self.t(x + "w2").T + self.t(x + "w0")
            w = torch.exp(-math.exp(-0.5) * torch.sigmoid(lw))

            def one(r, k, v, a, w):
                T = r.shape[0]
                r, k, v, a, w = (b.view(T, H, d) for b in (r, k, v, a, w))
                u = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
                S, o = torch.zeros(H, d, d, dtype=h.dtype, device=h.device), torch.empty_like(v)
                for t in range(T):
                    S = w[t][:, :, None] * S - (a[t] * u[t])[:, :, None] * (u[t][:, None, :] @ S) + k[t][:, :, None] * v[t][:, None, :]
                    o[t] = (r[t][:, None, :] @ S)[:, 0]
                return _rms(o, 1.0, eps).reshape(T, H * d)

            o = self._each(cut, one, r, k, v, a, w) * self.t(x + "norm") * torch.sigmoid(g)
            return o @ self.t(x + "o").T

        def mixer(h):
            canon = self.t(p + "canon1")
            h = h + self._each(cut, lambda a: _conv(a, canon), h)
            if layer["type"] == "latent_attention":
                return self._latent(h, cut, m, x, eps, False)
            return ssm(h) if layer["type"] == "mamba2" else delta(h)

        def experts(h):
            mlp, y = layer["mlp"], torch.zeros_like(h)
            table = self.w._values(p + "mlp.table", self.w.shapes[p + "mlp.table"])[ids]
            for e in range(mlp["router"]["experts"]):
                row = (table == e).any(-1).nonzero()[:, 0]
                if row.numel():
                    up = torch.nn.functional.gelu(h[row] @ self.t(f"{p}mlp.e{e}.up").T)
                    y[row] += up @ self.t(f"{p}mlp.e{e}.down").T / mlp["router"]["top"]
            return y

        for q, fn in (("1", mixer), ("2", experts)):
            u = torch.einsum("s,stw->tw", self.t(f"{p}hc{q}.in"), xs)
            y = fn(_rms(u, self.t(f"{p}norm{q}"), eps))
            xs = torch.einsum("sr,stw->rtw", self.t(f"{p}hc{q}.mix"), xs) + self.t(f"{p}hc{q}.out")[:, None, None] * y
        return xs

    def _zasazen(self, i, res, cut, ids):
        cfg, p = self.cfg, f"l{i}."
        eps, layer = cfg["norm"]["eps"], cfg["layers"][i]
        m, mlp, x = layer["mixer"], layer["mlp"], p + "mix."
        h = _rms(res, self.t(p + "norm1"), eps)
        if layer["type"] == "mamba1":
            D, N, R = m["inner"], m["state"], m["dt_rank"]
            xin, z = (h @ self.t(x + "in").T).split(D, dim=1)
            conv = self.t(x + "conv")
            xin = _silu(self._each(cut, lambda a: _conv(a, conv), xin) + self.t(x + "conv.b"))
            low, B, C = (xin @ self.t(x + "x").T).split([R, N, N], dim=1)
            dt = torch.nn.functional.softplus(low @ self.t(x + "dt").T + self.t(x + "dt.b"), threshold=100.0)
            A, skip = -torch.exp(self.t(x + "A_log")), self.t(x + "D")

            def one(xin, B, C, dt):
                S, y = torch.zeros(D, N, dtype=h.dtype, device=h.device), torch.empty_like(xin)
                for t in range(xin.shape[0]):
                    S = torch.exp(dt[t][:, None] * A) * S + (dt[t] * xin[t])[:, None] * B[t]
                    y[t] = S @ C[t]
                return y + skip * xin

            y = (self._each(cut, one, xin, B, C, dt) * _silu(z)) @ self.t(x + "o").T
        else:
            a, b = m["left"], m["right"]
            q, k, v = (h @ self.t(f"{x}left.{n}").T + self.t(f"{x}left.{n}.b") for n in "qkv")
            q, k = _rms(q, self.t(x + "left.q.norm"), eps), _rms(k, self.t(x + "left.k.norm"), eps)
            slopes = [2.0 ** (-8.0 * (n + 1) / a["heads"]) for n in range(a["heads"])]

            def attention(q, k, v):
                T = q.shape[0]
                at = torch.arange(T, dtype=h.dtype, device=h.device)
                q = q * (1.0 + a["q_temp"]["coef"] * torch.log(torch.floor((at + 1) / a["q_temp"]["every"]) + 1.0))[:, None]
                return _attend(q.view(T, -1, a["dim"]), k.view(T, -1, a["dim"]), v.view(T, -1, a["vdim"]), a["scale"],
                               slopes=slopes).reshape(T, -1)

            left = self._each(cut, attention, q, k, v) @ self.t(x + "left.o").T
            q, k, v, g = (h @ self.t(f"{x}right.{n}").T for n in "qkvg")
            decay = torch.tensor(b["decay"], dtype=torch.float64, device=h.device).float().double()[None, :, None]

            def retention(q, k, v):
                T = q.shape[0]
                q, k = (_rotate(c.view(T, -1, b["dim"]), b["rot"]["base"], b["rot"]["dims"]) for c in (q, k))
                return _rms(_linear_state(q, k * b["dim"] ** -0.5, v.view(T, -1, b["vdim"]), decay), 1.0, eps).reshape(T, -1)

            right = (self._each(cut, retention, q, k, v) * _silu(g)) @ self.t(x + "right.o").T
            y = 0.5 * (_rms(left, self.t(x + "left.out"), eps) + _rms(right, self.t(x + "right.out"), eps))
        h, f = _rms(res, self.t(p + "norm2"), eps), p + "mlp."
        if mlp["kind"] == "dense":
            return res + y + torch.nn.functional.gelu(h @ self.t(f + "up").T, approximate="tanh") @ self.t(f + "down").T
        names = ("gate", "up", "down")
        top, idx = (h @ self.t(f + "router").T + self.t(f + "router.b")).topk(mlp["router"]["top"], dim=-1)
        prob = torch.softmax(top, -1)
        y = y + torch.sigmoid(h @ self.t(f + "shared.sg").T) * self._gated(h, f + "shared.", names=names)
        for e in range(mlp["router"]["experts"]):
            row, slot = (idx == e).nonzero(as_tuple=True)
            if row.numel():
                y.index_add_(0, row, prob[row, slot][:, None] * self._gated(h[row], f"{f}e{e}.", names=names))
        return res + y

    def _salolorn(self, i, res, cut, ids):
        cfg, p = self.cfg, f"l{i}."
        eps, layer = cfg["norm"]["eps"], cfg["layers"][i]
        m, x = layer["mixer"], p + "mix."
        h = _rms(res, self.t(p + "norm1"), eps)
        if layer["type"] == "latent_attention":
            y = self._latent(h, cut, m, x, eps, True)
        elif layer["type"] == "delta":
            H, G, d, dv = m["heads"], m["kv_heads"], m["dim"], m["vdim"]
            taps = [self.t(f"{x}{n}.conv") for n in "qkv"]
            q, k, v = (_silu(self._each(cut, lambda a, c=c: _conv(a, c), h @ self.t(x + n).T)) for n, c in zip("qkv", taps))
            beta = torch.sigmoid(h @ self.t(x + "b").T)
            g = torch.exp(-torch.exp(self.t(x + "A_log"))
                          * torch.nn.functional.softplus(h @ self.t(x + "a").T + self.t(x + "dt_bias"), threshold=100.0))

            def one(q, k, v, beta, g):
                T = q.shape[0]
                q, k = (a.view(T, G, d) / torch.sqrt((a.view(T, G, d) ** 2).sum(-1, keepdim=True) + 1e-6) for a in (q, k))
                q, k = (a.repeat_interleave(H // G, dim=1) for a in (q * d ** -0.5, k))
                v = v.view(T, H, dv)
                S, o = torch.zeros(H, d, dv, dtype=h.dtype, device=h.device), torch.empty_like(v)
                for t in range(T):
                    S = g[t][:, None, None] * S
                    u = beta[t][:, None] * (v[t] - (k[t][:, None, :] @ S)[:, 0])
                    S = S + k[t][:, :, None] * u[:, None, :]
                    o[t] = (q[t][:, None, :] @ S)[:, 0]
                return _rms(o, 1.0, eps).reshape(T, H * dv)

            o = self._each(cut, one, q, k, v, beta, g) * self.t(x + "norm").repeat(H) * _silu(h @ self.t(x + "g").T)
            y = o @ self.t(x + "o").T
        else:
            a, b = m["left"], m["right"]
            q, k, v = (h @ self.t(f"{x}left.{n}").T for n in "qkv")
            qn, kn, sink = self.t(x + "left.q.norm"), self.t(x + "left.k.norm"), self.t(x + "left.sink")

            def attention(q, k, v):
                T = q.shape[0]
                q, k = (_rotate(_rms(c.view(T, -1, a["dim"]), n, eps), a["rot"]["base"], a["rot"]["dims"])
                        for c, n in ((q, qn), (k, kn)))
                return _attend(q, k, v.view(T, -1, a["vdim"]), a["scale"], chunk=a["mask"]["size"], sink=sink)

            o = self._each(cut, attention, q, k, v) * torch.sigmoid(h @ self.t(x + "left.g").T)[:, :, None]
            y = m["left_scale"] * o.reshape(h.shape[0], -1) @ self.t(x + "left.o").T
            q, k, v, g = (h @ self.t(f"{x}right.{n}").T for n in "qkvg")
            z = (h @ self.t(x + "right.a1").T) @ self.t(x + "right.a2").T + self.t(x + "right.a2.b")
            alpha = torch.exp(torch.nn.functional.logsigmoid(z) / b["tau"])
            weight = self.t(x + "right.norm")

            def linear(q, k, v, alpha):
                T = q.shape[0]
                q, k, alpha = (c.view(T, -1, b["dim"]) for c in (q, k, alpha))
                return _rms(_linear_state(q * b["dim"] ** -0.5, k, v.view(T, -1, b["vdim"]), alpha), weight, eps).reshape(T, -1)

            y = y + m["right_scale"] * (self._each(cut, linear, q, k, v, alpha) * _silu(g)) @ self.t(x + "right.o").T
        res = res + _rms(y, self.t(p + "norm1b"), eps)
        h = _rms(res, self.t(p + "norm2"), eps)
        return res + _rms(self._gated(h, p + "mlp.", names=("gate", "up", "down")), self.t(p + "norm2b"), eps)


def exact(case, seed):
    with torch.no_grad():
        e = _Exact(case, seed)
        prompts = e.w.prompts()
        if case["how"] == "prompt":
            return {"logits": e.logits(prompts, [wanted_places(case, len(p)) for p in prompts])}
        follow = e.w.successors().tolist()
        seqs = []
        for p in prompts:
            p = list(p)
            for _ in range(case["new"] - 1):
                p.append(follow[p[-1]])
            seqs.append(p)
        return {"tokens": None, "logits": e.logits(seqs, [[len(s) - 1] for s in seqs])}


if __name__ == "__main__":
    rng = random.Random(0)
    for c in listed() + [dict(draw(rng), name=f"drawn {i}") for i in range(6)]:
        print(c["name"], work(c), lengths(c)[:8])
