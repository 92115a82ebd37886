"""The work whose speed is watched: decode steps and prompt portions, as a serving program has them done.

A case is either one decode step of a whole model through ``ModelRunner.step`` (captured, as the engine runs it; the
logits come back) or one layer's mixer, feed-forward or block on a flat batch of tokens (``parts.base.build``, the step
from ``StepInputBuilder``, pages and state slots from ``CacheManager``).  Sizes are those of the benchmark's model
shapes.  Weights, inputs and everything the cache holds are drawn from the seed; ``exact`` works the same formulas in
64 bits with plain torch.
"""

from __future__ import annotations

import math

import torch
import torch.nn.functional as F

from turingserve_b200.cache.manager import CacheManager, RunNeeds
from turingserve_b200.config.registry import get_architecture
from turingserve_b200.engine.batch import StepEntry, StepInputBuilder
from turingserve_b200.engine.runner import ModelRunner, run_needs
from turingserve_b200 import kernels
from turingserve_b200.models import fetedra, gugezen, komirax, pizunex, qwen2
from turingserve_b200.parts.base import BuildContext, build, build_block
from turingserve_b200.parts.model import DecoderModel

DEV = "cuda"
BF16 = torch.bfloat16
EPS = 1e-6

# the widths of the benchmark: Qwen2.5 shapes and layers of the other designs at the widths of 1.5B and 7B models
QWEN = {"0.5b": dict(hidden_size=896, intermediate_size=4864, num_heads=14, num_kv_heads=2, head_dim=64, vocab_size=151936),
        "1.5b": dict(hidden_size=1536, intermediate_size=8960, num_heads=12, num_kv_heads=2, head_dim=128, vocab_size=151936),
        "7b": dict(hidden_size=3584, intermediate_size=18944, num_heads=28, num_kv_heads=4, head_dim=128, vocab_size=152064)}
WIDTH = {"1.5b": 1536, "7b": 3584}
HEADS = {"1.5b": (12, 2), "7b": (28, 4)}                    # query heads, key/value heads of 128
LATENT = {"1.5b": dict(H=12, q_rank=768), "7b": dict(H=28, q_rank=1536)}        # plain 128, rotated 64, values 128, latent 512
DELTA = {"1.5b": (12, 6), "7b": (28, 14)}                   # heads, query/key heads of 128 x 128, 4 taps
STATE_SPACE = {"1.5b": 48, "7b": 112}                       # heads of 64, state 128, 2 groups, 4 taps, 2 norm parts
LINEAR = {"1.5b": 6, "7b": 14}                              # linear attention heads of 128 x 128
ROUTED = {"1.5b": (2688, 1344), "7b": (7104, 3552)}         # 8 experts, top 2; a shared one
DENSE = {"1.5b": 13440, "7b": 28416}
ROT_BANDED = {"base": 500000.0, "dims": 128, "scaling": {"factor": 8.0, "low": 1.0, "high": 4.0, "original": 8192}}
ROT_YARN = {"base": 10000.0, "dims": 64, "scaling": {"factor": 8.0, "original": 4096, "fast": 16.0, "slow": 2.0}}
ROT_PLAIN = {"base": 500000.0, "dims": 64}


def listed() -> list[dict]:
    layer = dict(context=0, prompts=1, singles=0, singles_context=0, page=64)
    return [
        # one user alone with a small model: a step is a chain of short kernels
        dict(name="qwen_decode_1", model="qwen", size="0.5b", layers=4, batch=1, context=517, page=16),
        # the benchmark's own step: eight users at 2,048 tokens
        dict(name="qwen_decode_8", model="qwen", size="1.5b", layers=4, batch=8, context=2048, page=16),
        # the same step of a design that mixes windowed attention, latent attention and the delta rule
        dict(name="pizunex_decode_8", model="pizunex", size="1.5b", layers=4, batch=8, context=2048, page=64),
        # a prompt of 2,048 tokens through one whole layer (the largest case)
        dict(name="qwen_layer_prompt", layer="qwen", size="1.5b", tokens=2048, **layer),
        # two prompts of odd lengths that arrive in portions, behind 1,300 tokens each: capped scores, bias, window
        dict(name="capped_attention_portions", layer="capped", size="1.5b", tokens=1023, **{**layer, "prompts": 2, "context": 1300}),
        # a prompt through latent attention
        dict(name="latent_attention_prompt", layer="latent", size="1.5b", tokens=2048, **layer),
        # a scheduler's mixed step at the 7B width: eight decoding users beside a portion of 512 of a long prompt
        dict(name="latent_window_mixed", layer="latent_window", size="7b", tokens=512,
             **{**layer, "context": 3000, "singles": 8, "singles_context": 2048}),
        # a prompt through attention with a sink and linear attention, side by side
        dict(name="sink_and_linear_prompt", layer="pair", size="1.5b", tokens=2048, **layer),
        # a prompt through the state-space mixer
        dict(name="state_space_prompt", layer="state_space", size="1.5b", tokens=2048, **layer),
        # an odd prompt through the delta rule
        dict(name="delta_rule_prompt", layer="delta", size="1.5b", tokens=1537, **layer),
        # a prompt through attention with two score maps a head
        dict(name="two_map_prompt", layer="two_map", size="1.5b", tokens=2048, **{**layer, "page": 16}),
        # a prompt through a routed feed-forward with a shared expert
        dict(name="routed_prompt", layer="routed", size="1.5b", tokens=2048, **layer),
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return max(lo, min(hi, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng) -> dict:
    kind = rng.choice(["qwen_step", "pizunex_step", "qwen", "capped", "latent", "latent_window", "pair", "state_space", "delta",
                       "two_map", "routed"])
    page = rng.choice([16, 64])
    if kind == "qwen_step":
        return dict(model="qwen", size=rng.choice(["0.5b", "1.5b"]), layers=rng.choice([2, 3, 4]), batch=_log_int(rng, 1, 48),
                    context=_log_int(rng, 16, 3000), page=page)
    if kind == "pizunex_step":
        return dict(model="pizunex", size="1.5b", layers=4, batch=_log_int(rng, 1, 32), context=_log_int(rng, 16, 3000), page=page)
    size = "1.5b" if kind == "qwen" else rng.choice(["1.5b", "1.5b", "7b"])
    prompts = rng.choice([1, 1, 2, 3])
    tokens = _log_int(rng, 17, (2047 if size == "1.5b" else 700) // prompts)
    keeps = kind not in ("qwen", "routed")
    singles = rng.choice([0, 0, _log_int(rng, 1, 16)]) if keeps else 0
    context = rng.choice([0, _log_int(rng, 5, 2000)]) if keeps else 0
    return dict(layer=kind, size=size, tokens=tokens, prompts=prompts, context=context, singles=singles,
                singles_context=_log_int(rng, 5, 2500) if singles else 0, page=page)


# -- what a case is made of: tensors by name, from the seed alone -----------------------------------------------------
class _Draws:
    def __init__(self, seed: int) -> None:
        self.g = torch.Generator(device=DEV).manual_seed(seed)

    def normal(self, *shape, std: float = 0.02, mean: float = 0.0, dtype=BF16) -> torch.Tensor:
        return torch.empty(shape, dtype=torch.float32, device=DEV).normal_(mean, std, generator=self.g).to(dtype)

    def uniform(self, *shape, lo: float, hi: float) -> torch.Tensor:
        return torch.empty(shape, dtype=torch.float32, device=DEV).uniform_(lo, hi, generator=self.g)

    def scale(self, *shape) -> torch.Tensor:
        return self.normal(*shape, std=0.1, mean=1.0, dtype=torch.float32)


def _mixer_config(kind: str, size: str) -> dict:
    """The layer's entry as the family's configuration file has it."""
    H, G = HEADS[size]
    if kind == "capped":
        return {"type": "attention", "mixer": {"heads": H, "kv_heads": G, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "softcap": 30.0,
                                               "mask": {"size": 1024}, "q_temp": {"coef": 0.1, "every": 128}}}
    if kind in ("latent", "latent_window"):
        m = {"heads": LATENT[size]["H"], "dim": 128, "rot_dim": 64, "vdim": 128, "q_rank": LATENT[size]["q_rank"], "kv_rank": 512,
             "scale": 192 ** -0.5, "rot": ROT_YARN if kind == "latent" else ROT_PLAIN}
        if kind == "latent_window":
            m["mask"] = {"size": 1024}
        return {"type": "latent_attention", "mixer": m}
    if kind == "delta":
        return {"type": "delta", "mixer": {"heads": DELTA[size][0], "kv_heads": DELTA[size][1], "dim": 128, "vdim": 128, "conv": 4}}
    if kind == "state_space":
        return {"type": "mamba2", "mixer": {"heads": STATE_SPACE[size], "vdim": 64, "state": 128, "groups": 2, "conv": 4, "norm_groups": 2}}
    if kind == "pair":
        L = LINEAR[size]
        return {"type": "parallel", "mixer": {
            "left": {"heads": H, "kv_heads": G, "dim": 128, "vdim": 128, "scale": 128 ** -0.5, "rot": ROT_BANDED},
            "right": {"heads": L, "dim": 128, "vdim": 128, "decay": _decays(L)}, "left_scale": 0.7, "right_scale": 1.1}}
    if kind == "two_map":
        return {"type": "attention", "mixer": {"heads": H, "kv_heads": G, "dim": 64, "vdim": 128, "diff": 0.5, "scale": 0.125}}
    raise ValueError(kind)


def _decays(n: int) -> list[float]:
    return [1.0 - 2.0 ** -(2 + 6 * i / max(1, n - 1)) for i in range(n)]


def _mixer_weights(kind: str, size: str, d: _Draws) -> dict[str, torch.Tensor]:
    h = WIDTH[size]
    H, G = HEADS[size]
    if kind == "capped":
        return {"q": d.normal(H * 128, h), "k": d.normal(G * 128, h), "q.norm": d.scale(H * 128), "k.norm": d.scale(G * 128),
                "o": d.normal(h, H * 128)}
    if kind in ("latent", "latent_window"):
        H, r = LATENT[size]["H"], LATENT[size]["q_rank"]
        w = {"dq": d.normal(r, h), "dq.norm": d.scale(r), "uq": d.normal(H * 192, r), "dkv": d.normal(576, h), "dkv.norm": d.scale(512),
             "uk": d.normal(H * 128, 512), "uv": d.normal(H * 128, 512), "o": d.normal(h, H * 128)}
        if kind == "latent_window":
            w.update({"sink": d.normal(H, std=1.0, dtype=torch.float32), "g": d.normal(H, h)})
        return w
    if kind == "delta":
        H, G = DELTA[size]
        c = lambda n: d.normal(n, 4, std=0.5, dtype=torch.float32)
        return {"q": d.normal(G * 128, h), "k": d.normal(G * 128, h), "v": d.normal(H * 128, h), "g": d.normal(H * 128, h),
                "b": d.normal(H, h), "a": d.normal(H, h), "q.conv": c(G * 128), "k.conv": c(G * 128), "v.conv": c(H * 128),
                "A_log": d.uniform(H, lo=0.0, hi=1.5), "dt_bias": d.uniform(H, lo=-4.5, hi=-2.0), "norm": d.scale(128),
                "o": d.normal(h, H * 128)}
    if kind == "state_space":
        H = STATE_SPACE[size]
        C = H * 64 + 512
        return {"in": d.normal(2 * H * 64 + 512 + H, h), "conv": d.normal(C, 4, std=0.5, dtype=torch.float32),
                "conv.b": d.normal(C, std=0.1, dtype=torch.float32), "dt_bias": d.uniform(H, lo=-4.5, hi=-2.0),
                "A_log": d.uniform(H, lo=0.0, hi=2.5), "D": d.scale(H), "norm": d.scale(H * 64), "o": d.normal(h, H * 64)}
    if kind == "pair":
        L = LINEAR[size] * 128
        left = {"q": d.normal(H * 128, h), "k": d.normal(G * 128, h), "v": d.normal(G * 128, h), "g": d.normal(H * 128, h),
                "q.b": d.normal(H * 128), "k.b": d.normal(G * 128), "v.b": d.normal(G * 128),
                "sink": d.normal(H, std=1.0, dtype=torch.float32), "o": d.normal(h, H * 128)}
        right = {"q": d.normal(L, h), "k": d.normal(L, h), "v": d.normal(L, h), "g": d.normal(L, h), "norm": d.scale(L), "o": d.normal(h, L)}
        return {**{"left." + k: v for k, v in left.items()}, **{"right." + k: v for k, v in right.items()}}
    if kind == "two_map":
        w = {"q": d.normal(H * 128, h), "k": d.normal(G * 128, h), "v": d.normal(G * 128, h), "q.b": d.normal(H * 128),
             "k.b": d.normal(G * 128), "v.b": d.normal(G * 128), "o": d.normal(h, H * 128)}
        w.update({n: d.normal(64, std=0.1, dtype=torch.float32) for n in ("lq1", "lk1", "lq2", "lk2")})
        return w
    raise ValueError(kind)


def _memory(kind: str, size: str, context: int, d: _Draws) -> dict[str, torch.Tensor]:
    """What one request's earlier tokens left behind: cached rows {k, v}, or {state, inputs} (the filter's last inputs)."""
    G = HEADS[size][1] if size in HEADS else 0
    out = {}
    if kind in ("capped", "pair", "two_map"):
        out.update(k=d.normal(context, G, 128, std=1.0), v=d.normal(context, G, 128, std=0.8))
    if kind in ("latent", "latent_window"):
        out.update(k=d.normal(context, 1, 576, std=1.0))
    some = 0.3 if context else 0.0                          # (a request's first tokens find a zeroed slot)
    if kind == "delta":
        H, G = DELTA[size]
        out.update(state=d.normal(H, 128, 128, std=some / 8, dtype=torch.float32),
                   inputs=d.normal(3, 2 * G * 128 + H * 128, std=some * 2).float())
    if kind == "state_space":
        H = STATE_SPACE[size]
        out.update(state=d.normal(H, 128, 64, std=some, dtype=torch.float32), inputs=d.normal(3, H * 64 + 512, std=some * 2).float())
    if kind == "pair":
        out.update(state=d.normal(LINEAR[size], 128, 128, std=some * 5, dtype=torch.float32))
    return out


def _routed_weights(size: str, d: _Draws) -> dict[str, torch.Tensor]:
    h, (ff, shared) = WIDTH[size], ROUTED[size]
    w = {"router": d.normal(8, h, dtype=torch.float32)}
    for e in range(8):
        w[f"e{e}.up"], w[f"e{e}.down"] = d.normal(ff, h), d.normal(h, ff)
    w["shared.up"], w["shared.down"] = d.normal(shared, h), d.normal(h, shared)
    return w


def _qwen_weights(size: str, d: _Draws) -> dict[str, torch.Tensor]:
    """One layer's tensors, by the checkpoint's names behind 'model.layers.i.'."""
    z = QWEN[size]
    h, ff, D = z["hidden_size"], z["intermediate_size"], z["head_dim"]
    q, kv = z["num_heads"] * D, z["num_kv_heads"] * D
    at, ml = "self_attn.", "mlp."
    return {at + "q_proj.weight": d.normal(q, h), at + "k_proj.weight": d.normal(kv, h), at + "v_proj.weight": d.normal(kv, h),
            at + "q_proj.bias": d.normal(q), at + "k_proj.bias": d.normal(kv), at + "v_proj.bias": d.normal(kv),
            at + "o_proj.weight": d.normal(h, q), ml + "gate_proj.weight": d.normal(ff, h), ml + "up_proj.weight": d.normal(ff, h),
            ml + "down_proj.weight": d.normal(h, ff), "input_layernorm.weight": d.normal(h, std=0.1, mean=1.0),
            "post_attention_layernorm.weight": d.normal(h, std=0.1, mean=1.0)}


PIZUNEX_LAYERS = ("capped", "latent", "delta", "delta")     # with a dense feed-forward, but for the third


def _qwen_config(size: str, layers: int):
    return qwen2.make_config(num_layers=layers, rope_theta=1e6, rms_norm_eps=EPS, tie_word_embeddings=True,
                             max_position_embeddings=32768, **QWEN[size])


def _lengths(case: dict) -> list[tuple[int, int]]:
    """(tokens this step, tokens before) per request, single tokens first; prompts of a step differ in length."""
    return ([(1, case["singles_context"] + 7 * i) for i in range(case["singles"])]
            + [(max(2, case["tokens"] - 61 * i), case["context"]) for i in range(case["prompts"])])


def _inputs(case: dict, seed: int) -> dict:
    """Weights, input rows and every request's memory."""
    d = _Draws(seed)
    if "model" in case:
        n, B, ctx = case["layers"], case["batch"], case["context"]
        if case["model"] == "qwen":
            z = QWEN[case["size"]]
            h, kinds = z["hidden_size"], ["qwen"] * n
            w = {f"model.layers.{i}.{k}": v for i in range(n) for k, v in _qwen_weights(case["size"], d).items()}
            w.update({"model.embed_tokens.weight": d.normal(z["vocab_size"], h), "model.norm.weight": d.normal(h, std=0.1, mean=1.0)})
            vocab = z["vocab_size"]
            memory = [[dict(k=d.normal(ctx + 3 * b, z["num_kv_heads"], z["head_dim"], std=1.0),
                            v=d.normal(ctx + 3 * b, z["num_kv_heads"], z["head_dim"], std=0.8)) for _ in kinds] for b in range(B)]
        else:
            h, kinds, vocab, w = WIDTH[case["size"]], PIZUNEX_LAYERS[:n], 32000, {}
            for i, kind in enumerate(kinds):
                w.update({f"l{i}.mix.{k}": v for k, v in _mixer_weights(kind, case["size"], d).items()})
                w[f"l{i}.norm1"] = d.scale(h)
                if i != 2:
                    w.update({f"l{i}.norm2": d.scale(h), f"l{i}.mlp.up": d.normal(DENSE[case["size"]], h),
                              f"l{i}.mlp.down": d.normal(h, DENSE[case["size"]])})
            w.update({"embed": d.normal(vocab, h, std=1.0), "head": d.normal(vocab, h), "final.norm": d.scale(h)})
            memory = [[_memory(k, case["size"], ctx + 3 * b, d) for k in kinds] for b in range(B)]
        tokens = torch.randint(0, vocab, (B,), generator=d.g, device=DEV).tolist()
        return dict(w=w, memory=memory, tokens=tokens, vocab=vocab, kinds=kinds)
    kind, size = case["layer"], case["size"]
    reqs = _lengths(case)
    h = QWEN[size]["hidden_size"]
    x = d.normal(sum(n for n, _ in reqs), h, std=1.0)
    if kind == "routed":
        return dict(w=_routed_weights(size, d), x=x, reqs=reqs, memory=[{} for _ in reqs])
    if kind == "qwen":
        return dict(w=_qwen_weights(size, d), x=x, reqs=reqs, memory=[{} for _ in reqs])
    return dict(w=_mixer_weights(kind, size, d), x=x, reqs=reqs, memory=[_memory(kind, size, c, d) for _, c in reqs])


# -- prepare and run ---------------------------------------------------------------------------------------------------
def _fill(manager: CacheManager, view, state, rc, context: int, memory: dict) -> None:
    """Puts a request's earlier tokens where the run's mixer keeps them."""
    if view is not None and "k" in memory and context:
        pos = torch.arange(context, device=DEV)
        table = torch.tensor(rc.tables[view.group], device=DEV)
        pages, at = table[pos // manager.page_size], pos % manager.page_size
        view.k[pages, :, at] = memory["k"]
        if "v" in memory:
            view.v[pages, :, at] = memory["v"]
    if state is not None and "state" in memory:
        rows = [memory["state"].reshape(-1)] + ([memory["inputs"].reshape(-1)] if "inputs" in memory else [])
        state[rc.slot] = torch.cat(rows).view(state[rc.slot].shape)


def _part(kind: str, size: str, ctx: BuildContext):
    """The layer's mixer (or feed-forward), built from its family's configuration."""
    family = {"capped": pizunex, "latent": pizunex, "delta": pizunex, "latent_window": fetedra, "state_space": gugezen,
              "pair": gugezen, "routed": gugezen, "two_map": komirax}[kind]
    entry = _mixer_config("capped" if kind == "routed" else kind, size) if kind != "routed" else _mixer_config("state_space", size)
    mlp = {"kind": "dense", "ff": 256}
    if kind == "routed":
        ff, shared = ROUTED[size]
        mlp = {"kind": "moe", "expert": {"ff": ff}, "router": {"experts": 8, "top": 2}, "shared": {"ff": shared}}
    more = {"streams": 2} if family in (gugezen, fetedra) else {}
    cfg = family.make_config(width=WIDTH[size], vocab=512, layers=[{**entry, "mlp": mlp}], eps=EPS, **more)
    spec = cfg.layers[0]
    return build("feed_forward", spec.feed_forward, ctx) if kind == "routed" else build("mixer", spec.mixer, ctx)


def prepare(case: dict, seed: int) -> dict:
    data = _inputs(case, seed)
    page = case["page"]
    if "model" in case:
        B, most = case["batch"], case["context"] + 3 * case["batch"] + 2 * page
        if case["model"] == "qwen":
            cfg, build_model = _qwen_config(case["size"], case["layers"]), DecoderModel
        else:
            entries = []
            for i, kind in enumerate(data["kinds"]):
                entries.append({**_mixer_config(kind, case["size"]), "mlp": None if i == 2 else {"kind": "dense", "ff": DENSE[case["size"]]}})
            cfg = pizunex.make_config(width=WIDTH[case["size"]], vocab=data["vocab"], layers=entries, eps=EPS)
        arch = get_architecture(cfg.architecture)
        model = (arch.build_model or DecoderModel)(cfg, BF16, DEV, most)
        model.load(arch.tensor_names(cfg), data["w"])
        pages = B * (-(-most // page)) + 8
        manager = CacheManager(run_needs(model), page, pages, B, BF16, torch.device(DEV, 0))
        runner = ModelRunner(model, manager, max(B, 16), B, most, (B,))
        entries = []
        for b in range(B):
            rc = manager.admit(f"r{b}")
            context = case["context"] + 3 * b
            manager.grow(rc, context)
            for r, memory in enumerate(data["memory"][b]):
                _fill(manager, runner.views[r], manager.states[r], rc, context, memory)
            manager.advance(rc, context)
            entries.append(StepEntry(rc, [data["tokens"][b]], [0]))
        return dict(case=case, runner=runner, entries=entries)
    kind, x = case["layer"], data["x"]
    most = max(n + c for n, c in data["reqs"])
    ctx = BuildContext(hidden_size=x.shape[1], dtype=BF16, device=torch.device(DEV, 0), max_positions=most)
    if kind == "routed":
        part = _part(kind, case["size"], ctx)
        part.load(data["w"])
        return dict(case=case, part=part, x=x)
    if kind == "qwen":
        part = build_block(_qwen_config(case["size"], 1).layers[0], ctx)
        prefix = {"mixer": "self_attn.", "feed_forward": "mlp.", "mixer_norm": "input_layernorm.", "ffn_norm": "post_attention_layernorm."}
        for role, sub in part.parts().items():
            sub.load({name: data["w"][prefix[role] + name] for name in sub.parameters()})
        mixer = part.mixer
    else:
        part = mixer = _part(kind, case["size"], ctx)
        part.load({name: data["w"][name] for name in part.parameters()})
    needs = RunNeeds(mixer.cache_need(), mixer.state_need())
    n_req = len(data["reqs"])
    manager = CacheManager([needs], page, sum(-(-(n + c) // page) for n, c in data["reqs"]) + 8, n_req, BF16, torch.device(DEV, 0))
    view, state = manager.view(0), manager.states[0]
    entries = []
    for i, ((n, context), memory) in enumerate(zip(data["reqs"], data["memory"])):
        rc = manager.admit(f"r{i}")
        manager.grow(rc, context)
        _fill(manager, view, state, rc, context, memory)
        manager.advance(rc, context)
        manager.grow(rc, n)
        entries.append(StepEntry(rc, [0] * n, [n - 1]))
    builder = StepInputBuilder(manager, x.shape[0], n_req, -(-most // page), torch.device(DEV, 0))
    return dict(case=case, part=part, x=x, manager=manager, view=view, state=state, builder=builder, step=builder.build(entries),
                before=None if state is None else state.clone())


def run(s: dict):
    case = s["case"]
    if "model" in case:
        logits = s["runner"].step(s["entries"])
        for e in s["entries"]:
            e.cache.num_tokens -= 1                         # the next pass tries the same position again
        runner = s["runner"]
        return {"logits": logits, "keys": [v.k for v in runner.views if v is not None],
                "values": [v.v for v in runner.views if v is not None],
                "states": [t[:-1] for t in runner.cache.states if t is not None]}
    ops = kernels.ops()
    if case["layer"] == "routed":
        return {"out": ops.materialize(s["part"].forward(s["x"]))}
    if case["layer"] == "qwen":
        h, residual = s["part"].forward(s["x"].clone(), None, s["step"], s["view"], None)
        return {"out": ops.materialize(h), "residual": residual, "keys": s["view"].k, "values": s["view"].v}
    if s["state"] is not None:
        s["state"].copy_(s["before"])                       # the requests' memory as the step finds it
    out = {"out": ops.materialize(s["part"].forward(s["x"], s["step"], s["view"], s["state"]))}
    if s["view"] is not None:
        out["keys"], out["values"] = s["view"].k, s["view"].v
    if s["state"] is not None:
        out["state"] = s["state"][:-1]
    return out


# -- what a pass cannot do without -------------------------------------------------------------------------------------
def _pairs(n: int, context: int, window: int | None) -> int:
    """(query, key) pairs of n tokens behind ``context`` others."""
    if window is None:
        return n * context + n * (n + 1) // 2
    return sum(min(context + i + 1, window) for i in range(n))


def _mixer_work(kind: str, size: str, reqs: list[tuple[int, int]]) -> tuple[float, float]:
    """(bytes of weights and memory, operations); the input and output rows are the caller's."""
    h = WIDTH[size]
    H, G = HEADS[size]
    T, ctx = sum(n for n, _ in reqs), sum(c for _, c in reqs)
    if kind in ("latent", "latent_window"):
        H, r = LATENT[size]["H"], LATENT[size]["q_rank"]
        w = r * h + H * 192 * r + 576 * h + 2 * H * 128 * 512 + h * H * 128
        window = 1024 if kind == "latent_window" else None
        flops, seen = 0.0, 0
        for n, c in reqs:
            reach = min(c, window - 1) if window else c
            pairs = _pairs(n, c, window)
            # over the latent rows, or with every head's keys and values formed from them first
            flops += min(2.0 * pairs * H * (576 + 512) + 2.0 * n * H * 128 * 1024, 2.0 * pairs * H * 320 + 2.0 * (n + reach) * H * 256 * 512)
            seen += reach + n
        return 2.0 * w + 2.0 * seen * 576, flops + 2.0 * T * (r * h + H * 192 * r + 576 * h + h * H * 128)
    if kind in ("capped", "pair", "two_map"):
        w = 2 * H * 128 * h + G * 128 * h * (1 if kind == "capped" else 2)
        window = 1024 if kind == "capped" else None
        maps = 2 if kind == "two_map" else 1
        flops = sum(2.0 * _pairs(n, c, window) * H * (128 + 128 * maps) for n, c in reqs)
        seen = sum((min(c, 1023) if window else c) + n for n, c in reqs)
        mem = 2.0 * seen * G * 256
        if kind == "pair":
            L = LINEAR[size]
            w += H * 128 * h + 5 * L * 128 * h
            flops += 6.0 * T * L * 128 * 128
            mem += 2.0 * 4 * len(reqs) * L * 128 * 128
        return 2.0 * w + mem, flops + 2.0 * T * w
    if kind == "delta":
        H, G = DELTA[size]
        w, state = h * (2 * G * 128 + 3 * H * 128 + 2 * H), H * 128 * 128 + 3 * (2 * G + H) * 128
    else:
        H = STATE_SPACE[size]
        w, state = h * (3 * H * 64 + 512 + H), H * 128 * 64 + 3 * (H * 64 + 512)
    return 2.0 * w + 8.0 * len(reqs) * state, 2.0 * T * w + (8.0 if kind == "delta" else 6.0) * T * H * 128 * (128 if kind == "delta" else 64)


def work(case: dict) -> dict:
    if "model" in case:
        B = case["batch"]
        reqs = [(1, case["context"] + 3 * b) for b in range(B)]
        if case["model"] == "qwen":
            z = QWEN[case["size"]]
            h, D = z["hidden_size"], z["head_dim"]
            q, kv = z["num_heads"] * D, z["num_kv_heads"] * D
            w = case["layers"] * (h * (2 * q + 2 * kv) + 3 * h * z["intermediate_size"]) + z["vocab_size"] * h
            seen = sum(n + c for n, c in reqs) * case["layers"]
            return {"bytes": 2.0 * w + 4.0 * seen * kv + 4.0 * B * z["vocab_size"], "flops": 2.0 * B * w + 4.0 * seen * q}
        h = WIDTH[case["size"]]
        nbytes, flops = 2.0 * 32000 * h + 4.0 * B * 32000, 2.0 * B * 32000 * h
        for i, kind in enumerate(PIZUNEX_LAYERS[:case["layers"]]):
            a, b = _mixer_work(kind, case["size"], reqs)
            ff = 0 if i == 2 else 2 * h * DENSE[case["size"]]
            nbytes, flops = nbytes + a + 2.0 * ff, flops + b + 2.0 * B * ff
        return {"bytes": nbytes, "flops": flops}
    reqs = _lengths(case)
    T, size = sum(n for n, _ in reqs), case["size"]
    if case["layer"] == "qwen":
        z = QWEN[size]
        h, D = z["hidden_size"], z["head_dim"]
        q, kv = z["num_heads"] * D, z["num_kv_heads"] * D
        w = h * (2 * q + 2 * kv) + 3 * h * z["intermediate_size"]
        return {"bytes": 2.0 * w + 6.0 * T * h + 4.0 * T * kv, "flops": 2.0 * T * w + sum(4.0 * _pairs(n, c, None) * q for n, c in reqs)}
    h = WIDTH[size]
    if case["layer"] == "routed":
        ff, shared = ROUTED[size]
        used = min(8, 2 * T)
        return {"bytes": 4.0 * h * (used * ff + shared) + 4.0 * T * h, "flops": 4.0 * T * h * (2 * ff + shared)}
    a, b = _mixer_work(case["layer"], size, reqs)
    return {"bytes": a + 4.0 * T * h, "flops": b}


def tolerance(case: dict) -> dict:
    # bfloat16 operands and results between kernels: a layer's outputs and states were measured 0.2 to 0.6 % from the
    # 64-bit formulas, a model's logits after four layers 0.6 to 1.6 %
    if "model" in case:
        return {"rel": 0.03, "max": 0.3}
    return {"rel": 0.02, "max": 0.15}


# -- the same in 64 bits -----------------------------------------------------------------------------------------------
def _rms(x, w=None):
    y = x / torch.sqrt(x.pow(2).mean(-1, keepdim=True) + EPS)
    return y if w is None else y * w


def _softmax_attention(q, k, v, first: int, scale: float, cap=None, slopes=None, window=None, sink=None):
    """q [n, H, D] at positions first.., k [m, G, D], v [m, G, V] at positions 0.. -> [n, H, V]."""
    n, H, _ = q.shape
    per = H // k.shape[1]
    i = torch.arange(n, device=DEV)[:, None] + first
    j = torch.arange(k.shape[0], device=DEV)[None, :]
    hidden = j > i
    if window:
        hidden = hidden | (i - j >= window)
    out = []
    for h in range(H):
        s = (q[:, h] @ k[:, h // per].T) * scale
        if cap:
            s = cap * torch.tanh(s / cap)
        if slopes is not None:
            s = s - slopes[h] * (i - j)
        s = s.masked_fill(hidden, float("-inf"))
        m = s.max(-1, keepdim=True).values
        if sink is not None:
            m = torch.maximum(m, sink[h])
        e = torch.exp(s - m)
        total = e.sum(-1, keepdim=True)
        if sink is not None:
            total = total + torch.exp(sink[h] - m)
        out.append((e / total) @ v[:, h // per])
    return torch.stack(out, 1)


def _frequencies(rot: dict) -> tuple[torch.Tensor, float]:
    i = torch.arange(rot["dims"] // 2, dtype=torch.float64, device=DEV)
    f, mag, sc = rot["base"] ** (-2.0 * i / rot["dims"]), 1.0, rot.get("scaling")
    if sc and "fast" in sc:
        at = lambda turns: rot["dims"] * math.log(sc["original"] / (2 * math.pi * turns)) / (2 * math.log(rot["base"]))
        begin, end = max(math.floor(at(sc["fast"])), 0), min(math.ceil(at(sc["slow"])), rot["dims"] - 1)
        t = ((i - begin) / max(end - begin, 0.001)).clamp(0, 1)
        f, mag = (1 - t) * f + t * f / sc["factor"], 1.0 + 0.1 * math.log(sc["factor"])
    elif sc:
        turns = sc["original"] * f / (2 * math.pi)
        s = (turns - sc["low"]) / (sc["high"] - sc["low"])
        f = torch.where(turns > sc["high"], f, torch.where(turns < sc["low"], f / sc["factor"], (1 - s) * f / sc["factor"] + s * f))
    return f, mag


def _turn(x, pos, rot: dict, halves: bool):
    """x [n, ..., R]: its pairs (neighbours, or halves of the rotated dimensions) turned by position * frequency."""
    f, mag = _frequencies(rot)
    a = pos.double()[:, None] * f
    a = a.view(a.shape[0], *([1] * (x.dim() - 2)), a.shape[1])
    c, s = torch.cos(a) * mag, torch.sin(a) * mag
    if halves:
        u, v = x.chunk(2, -1)
        return torch.cat([u * c - v * s, v * c + u * s], -1)
    u, v = x[..., 0::2], x[..., 1::2]
    return torch.stack([u * c - v * s, v * c + u * s], -1).flatten(-2)


def _filtered(x, before, taps, bias=None):
    """SiLU of a causal filter over x [n, C] behind the rows ``before`` [taps - 1, C]; also the new last inputs."""
    rows = torch.cat([before, x])
    y = sum(rows[u:u + x.shape[0]] * taps[:, u] for u in range(taps.shape[1]))
    return F.silu(y if bias is None else y + bias), rows[rows.shape[0] - before.shape[0]:]


def _exact_mixer(kind: str, size: str, w: dict, x, first: int, mem: dict):
    """One request's rows through a mixer: (output, the state after them or None)."""
    n = x.shape[0]
    H, G = HEADS[size]
    pos = torch.arange(first, first + n, device=DEV)
    if kind == "capped":
        q, k = x @ w["q"].T, x @ w["k"].T
        heat = 1.0 + 0.1 * torch.log(torch.floor((pos.double() + 1) / 128) + 1.0)
        keys = torch.cat([mem["k"], _rms(k, w["k.norm"]).view(n, G, 128)])
        slopes = [2.0 ** (-8.0 * (a + 1) / H) for a in range(H)]
        a = _softmax_attention((_rms(q, w["q.norm"]) * heat[:, None]).view(n, H, 128), keys, torch.cat([mem["v"], k.view(n, G, 128)]),
                               first, 128 ** -0.5, 30.0, slopes, 1024)
        return a.reshape(n, -1) @ w["o"].T, None
    if kind in ("latent", "latent_window"):
        H, own = LATENT[size]["H"], kind == "latent_window"
        rot = ROT_PLAIN if own else ROT_YARN
        q = (_rms(x @ w["dq"].T, w["dq.norm"]) @ w["uq"].T).view(n, H, 192)
        both = x @ w["dkv"].T
        rows = torch.cat([_rms(both[:, :512], w["dkv.norm"]), _turn(both[:, 512:], pos, rot, own)], -1)
        rows = torch.cat([mem["k"][:, 0], rows])
        qa = torch.cat([torch.einsum("nhd,hdr->nhr", q[..., :128], w["uk"].view(H, 128, 512)), _turn(q[..., 128:], pos, rot, own)], -1)
        mixed = _softmax_attention(qa, rows[:, None], rows[:, None, :512], first, 192 ** -0.5, window=1024 if own else None,
                                   sink=w["sink"] if own else None)
        if own:
            mixed = mixed * torch.sigmoid(x @ w["g"].T)[..., None]
        return torch.einsum("nhr,hvr->nhv", mixed, w["uv"].view(H, 128, 512)).reshape(n, -1) @ w["o"].T, None
    if kind == "two_map":
        q = (x @ w["q"].T + w["q.b"]).view(n, H, 2, 64)
        k = torch.cat([mem["k"], (x @ w["k"].T + w["k.b"]).view(n, G, 128)]).view(-1, G, 2, 64)
        v = torch.cat([mem["v"], (x @ w["v"].T + w["v.b"]).view(n, G, 128)])
        lam = torch.exp((w["lq1"] * w["lk1"]).sum()) - torch.exp((w["lq2"] * w["lk2"]).sum()) + 0.5
        one, two = (_softmax_attention(q[:, :, m], k[:, :, m], v, first, 0.125) for m in (0, 1))
        return (_rms(one - lam * two) * 0.5).reshape(n, -1) @ w["o"].T, None
    if kind == "pair":
        u = {key[5:]: t for key, t in w.items() if key.startswith("left.")}
        q = _turn((x @ u["q"].T + u["q.b"]).view(n, H, 128), pos, ROT_BANDED, False)
        k = torch.cat([mem["k"], _turn((x @ u["k"].T + u["k.b"]).view(n, G, 128), pos, ROT_BANDED, False)])
        v = torch.cat([mem["v"], (x @ u["v"].T + u["v.b"]).view(n, G, 128)])
        a = _softmax_attention(q, k, v, first, 128 ** -0.5, sink=u["sink"]).reshape(n, -1)
        left = (a * torch.sigmoid(x @ u["g"].T)) @ u["o"].T
        u = {key[6:]: t for key, t in w.items() if key.startswith("right.")}
        L = LINEAR[size]
        q, k, v = (F.silu(x @ u[m].T).view(n, L, 128) for m in "qkv")
        lam = torch.tensor(_decays(L), dtype=torch.float64, device=DEV).view(L, 1, 1)
        S, out = mem["state"], torch.empty(n, L, 128, dtype=torch.float64, device=DEV)
        for t in range(n):
            S = lam * S + k[t, :, :, None] * v[t, :, None, :]
            out[t] = torch.einsum("hdv,hd->hv", S, q[t])
        right = (_rms(out.reshape(n, -1), u["norm"]) * torch.sigmoid(x @ u["g"].T)) @ u["o"].T
        return 0.7 * left + 1.1 * right, S
    if kind == "delta":
        H, G = DELTA[size]
        raw = torch.cat([x @ w["q"].T, x @ w["k"].T, x @ w["v"].T], -1)
        y, last = _filtered(raw, mem["inputs"], torch.cat([w["q.conv"], w["k.conv"], w["v.conv"]]))
        unit = lambda z: z / torch.sqrt(z.pow(2).sum(-1, keepdim=True) + 1e-6)
        q, k = (unit(z.view(n, G, 128)).repeat_interleave(H // G, 1) for z in y[:, :2 * G * 128].chunk(2, -1))
        v, q = y[:, 2 * G * 128:].view(n, H, 128), q * 128 ** -0.5
        b = torch.sigmoid(x @ w["b"].T)
        g = torch.exp(-torch.exp(w["A_log"]) * F.softplus(x @ w["a"].T + w["dt_bias"], threshold=40.0))
        S, out = mem["state"], torch.empty(n, H, 128, dtype=torch.float64, device=DEV)
        for t in range(n):
            S = g[t, :, None, None] * S
            e = b[t, :, None] * (v[t] - torch.einsum("hdv,hd->hv", S, k[t]))
            S = S + k[t, :, :, None] * e[:, None, :]
            out[t] = torch.einsum("hdv,hd->hv", S, q[t])
        out = _rms(out) * w["norm"] * F.silu(x @ w["g"].T).view(n, H, 128)
        return out.reshape(n, -1) @ w["o"].T, torch.cat([S.reshape(-1), last.reshape(-1)])
    H = STATE_SPACE[size]                                   # the state-space mixer
    u = x @ w["in"].T
    z, raw, dt = u[:, :H * 64], u[:, H * 64:2 * H * 64 + 512], u[:, 2 * H * 64 + 512:]
    y, last = _filtered(raw, mem["inputs"], w["conv"], w["conv.b"])
    xs, (B, C) = y[:, :H * 64].view(n, H, 64), (m.reshape(n, 2, 128).repeat_interleave(H // 2, 1) for m in y[:, H * 64:].chunk(2, -1))
    dt = F.softplus(dt + w["dt_bias"], threshold=40.0)
    a = torch.exp(-torch.exp(w["A_log"]) * dt)
    S, out = mem["state"], torch.empty(n, H, 64, dtype=torch.float64, device=DEV)
    for t in range(n):
        S = a[t, :, None, None] * S + (dt[t, :, None] * B[t])[:, :, None] * xs[t, :, None, :]
        out[t] = torch.einsum("hnp,hn->hp", S, C[t]) + w["D"][:, None] * xs[t]
    g = _rms((out.reshape(n, -1) * F.silu(z)).view(n, 2, -1)).reshape(n, -1) * w["norm"]
    return g @ w["o"].T, torch.cat([S.reshape(-1), last.reshape(-1)])


def _exact_qwen(size: str, w: dict, h, first: int, mem: dict | None):
    """One request's rows through a layer: (the feed-forward's output, the stream it is added to)."""
    z, at = QWEN[size], "self_attn."
    n, H, G, D = h.shape[0], z["num_heads"], z["num_kv_heads"], z["head_dim"]
    x = _rms(h, w["input_layernorm.weight"])
    rot = {"base": 1e6, "dims": D}
    pos = torch.arange(first, first + n, device=DEV)
    q, k, v = ((x @ w[f"{at}{m}_proj.weight"].T + w[f"{at}{m}_proj.bias"]).view(n, -1, D) for m in "qkv")
    q, k = _turn(q, pos, rot, True), _turn(k, pos, rot, True)
    if mem is not None:
        k, v = torch.cat([mem["k"], k]), torch.cat([mem["v"], v])
    h = h + _softmax_attention(q, k, v, first, D ** -0.5).reshape(n, H * D) @ w[at + "o_proj.weight"].T
    x = _rms(h, w["post_attention_layernorm.weight"])
    return (F.silu(x @ w["mlp.gate_proj.weight"].T) * (x @ w["mlp.up_proj.weight"].T)) @ w["mlp.down_proj.weight"].T, h


def _double(v):
    if isinstance(v, torch.Tensor):
        return v.double()
    if isinstance(v, dict):
        return {k: _double(x) for k, x in v.items()}
    return [_double(x) for x in v]


def exact(case: dict, seed: int):
    data = _inputs(case, seed)
    if "model" in case:
        w, rows = data["w"], []
        names = {"qwen": ("model.embed_tokens.weight", "model.norm.weight", "model.embed_tokens.weight"),
                 "pizunex": ("embed", "final.norm", "head")}[case["model"]]
        layers = [_double({k[len(p):]: v for k, v in w.items() if k.startswith(p)}) for p in
                  (f"model.layers.{i}." if case["model"] == "qwen" else f"l{i}." for i in range(case["layers"]))]
        head, norm = w[names[2]].double(), w[names[1]].double()
        for b in range(case["batch"]):
            h, first = w[names[0]][data["tokens"][b]].double()[None], case["context"] + 3 * b
            for i, kind in enumerate(data["kinds"]):
                u, mem = layers[i], _double(data["memory"][b][i])
                if kind == "qwen":
                    y, h = _exact_qwen(case["size"], u, h, first, mem)
                    h = h + y
                    continue
                mix = {k[4:]: v for k, v in u.items() if k.startswith("mix.")}
                h = h + _exact_mixer(kind, case["size"], mix, _rms(h, u["norm1"]), first, mem)[0]
                if i != 2:
                    h = h + F.relu(_rms(h, u["norm2"]) @ u["mlp.up"].T).pow(2) @ u["mlp.down"].T
            rows.append(_rms(h, norm) @ head.T)
        return {"logits": torch.cat(rows), "keys": None, "values": None, "states": None}
    w, x = _double(data["w"]), data["x"].double()
    if case["layer"] == "routed":
        score = torch.softmax(x @ w["router"].T, -1)
        val, idx = torch.topk(score, 2, dim=-1)
        val = val / val.sum(-1, keepdim=True)
        out = F.gelu(x @ w["shared.up"].T) @ w["shared.down"].T
        for e in range(8):
            weight = (val * (idx == e)).sum(-1)
            rows = weight.nonzero()[:, 0]
            out[rows] += weight[rows, None] * (F.gelu(x[rows] @ w[f"e{e}.up"].T) @ w[f"e{e}.down"].T)
        return {"out": out}
    outs, states, at = [], [], 0
    for (n, first), mem in zip(data["reqs"], data["memory"]):
        rows = x[at:at + n]
        at += n
        if case["layer"] == "qwen":
            y, h = _exact_qwen(case["size"], w, rows, first, None)
            outs.append(y)
            states.append(h)
            continue
        y, state = _exact_mixer(case["layer"], case["size"], w, rows, first, _double(mem))
        outs.append(y)
        states.append(state)
    out = {"out": torch.cat(outs)}
    if case["layer"] == "qwen":
        return {**out, "residual": torch.cat(states), "keys": None, "values": None}
    if case["layer"] in ("capped", "latent", "latent_window", "two_map", "pair"):
        out["keys"] = out["values"] = None
    if states[0] is not None:
        out["state"] = torch.stack(states)                  # (a new manager hands its slots out from 0 up)
    return out
