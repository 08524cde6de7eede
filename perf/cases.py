"""Cases that stand for the work this library does: whole prompt and single-token steps of a GPT-2 through the engine,
and the mixers', head-wise maps' and experts' kernels of the other designs through `Ops`, the door every part uses.

Sizes are those of the benchmark: GPT-2 small, and designs of width 1024 with 16 heads of 64 (4 key/value heads), latents of
256, recurrent heads of 128 x 128 or 64 x 128, 8 experts.  A prompt is 2 x 1024 tokens or a ragged batch, a single-token step has
8 rows after about 520 positions.  `lengths` and `cached` are texts of numbers, one per sequence.
"""
import json
import math
import os
import random
import struct
import tempfile

import numpy as np
import torch

from kvad_b200 import Engine, StepEntry
from kvad_b200.ops import Ops

PAGE = 64
DT = {"bfloat16": torch.bfloat16, "float32": torch.float32}


def listed():
    small = {"layers": 12, "width": 768, "heads": 12, "inner": 3072, "vocab": 50257, "positions": 1024}
    return [
        # the headline prompt step: two whole contexts in one step, the logits of the last tokens
        dict(small, name="gpt2_prompt_bf16", kind="prompt", dtype="bfloat16", lengths="1024 1024"),
        # a ragged batch of prompts in the 32-bit engine
        dict(small, name="gpt2_prompt_f32_ragged", kind="prompt", dtype="float32", lengths="64 183 302 421 540"),
        # eight sequences generating side by side
        dict(small, name="gpt2_decode_bf16_b8", kind="decode", dtype="bfloat16", lengths="96 64 33 128 97 80 111 50", steps=24),
        # one sequence generating in the 32-bit engine: the smallest step there is
        dict(small, name="gpt2_decode_f32_b1", kind="decode", dtype="float32", lengths="33", steps=24),
        # latent attention of a prompt: one shared key of 256 that is the value too, sinks, the full triangle
        dict(name="attention_latent_prompt", kind="attention", dtype="bfloat16", lengths="1024 1024", cached="0 0", heads=16, kv_heads=1, dk=256,
             dv=256, latent=True, window=0, keep_first=0, chunk=0, softcap=0.0, sinks=True, gate="none", step=False),
        # grouped heads with capped scores, a window that keeps the first tokens, an entry-wise gate
        dict(name="attention_window_prompt", kind="attention", dtype="bfloat16", lengths="1024 1024", cached="0 0", heads=16, kv_heads=4, dk=64,
             dv=64, latent=False, window=512, keep_first=4, chunk=0, softcap=30.0, sinks=False, gate="entry", step=False),
        # single-token rows over a latent cache with a rotated part
        dict(name="attention_latent_step", kind="attention", dtype="bfloat16", lengths="1 1 1 1 1 1 1 1", cached="519 511 530 522 498 540 515 527",
             heads=16, kv_heads=1, dk=288, dv=256, latent=True, window=0, keep_first=0, chunk=0, softcap=0.0, sinks=False, gate="none", step=True),
        # linear attention with a fixed decay per head, rotated queries and keys, a unit norm per head and a gate
        dict(name="retention_prompt", kind="retention", dtype="bfloat16", lengths="1024 1024", heads=8, dk=128, dv=128, rotate=True, finish=True),
        # the gated delta rule behind short convolutions: 32-bit rows
        dict(name="delta_rule_prompt", kind="recurrence", cell="delta_rule", dtype="float32", lengths="1024 1024", heads=8, dk=128, dv=128),
        # the matrix memory over a ragged batch
        dict(name="matrix_memory_prompt", kind="recurrence", cell="matrix_memory", dtype="bfloat16", lengths="1000 517 37", heads=8, dk=64, dv=128),
        # every head's query of a prompt carried into the latent's space
        dict(name="head_maps_prompt", kind="head_maps", dtype="bfloat16", rows=2048, heads=16, n_in=64, n_out=256, gate=False),
        # the chosen experts' output product of a step of 32 single-token rows
        dict(name="experts_step", kind="experts", dtype="bfloat16", rows=32, top=2, experts=16, n_in=1408, n_out=1024),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _ragged(rng, total, most):
    """Up to `most` sequences of unequal lengths, `total` rows at most, 1024 a sequence at most."""
    n, left, out = rng.randint(1, most), total, []
    for i in range(n):
        if left < 1:
            break
        out.append(max(1, min(1024, left, _log(rng, 17, 1024))))
        left -= out[-1]
    return " ".join(str(x) for x in out)


def draw(rng):
    kind = rng.choice(["prompt", "decode", "attention", "attention", "attention_step", "retention", "recurrence", "recurrence", "head_maps", "experts"])
    dtype = rng.choice(["bfloat16", "bfloat16", "bfloat16", "float32"])
    if kind in ("prompt", "decode"):
        layers = rng.randint(2, 12)
        width, heads = rng.choice([(768, 12), (768, 12), (640, 10), (512, 8)])
        c = {"kind": kind, "dtype": dtype, "layers": layers, "width": width, "heads": heads, "inner": rng.choice([4 * width, 3 * width + 64]), "vocab": 50257, "positions": 1024}
        if kind == "prompt":
            return dict(c, lengths=_ragged(rng, 2048 if dtype == "bfloat16" else 1500, 6))
        n = rng.choice([1, 2, 3, 5, 8, 12, 16])
        return dict(c, lengths=" ".join(str(_log(rng, 8, 128)) for _ in range(n)), steps=rng.randint(12, 24))
    if kind.startswith("attention"):
        latent = rng.random() < 0.4
        heads = rng.choice([8, 16])
        kv = 1 if latent else rng.choice([h for h in (2, 4, 8) if heads % h == 0])
        dv = rng.choice([64, 128, 192, 256]) if latent else rng.choice([32, 64, 64, 128])
        dk = dv + rng.choice([0, 32]) if latent else dv
        mask = rng.choice(["full", "window", "chunk"])
        size = rng.choice([100, 256, 512])
        if kind == "attention_step":
            n = rng.choice([1, 3, 8, 16])
            lengths, cached = " ".join(["1"] * n), " ".join(str(_log(rng, 40, 1000)) for _ in range(n))
        else:
            lengths = _ragged(rng, 2048, 4)
            cached = " ".join(str(rng.choice([0, 0, 0, rng.randint(1, 300)])) for _ in lengths.split())
        return {"kind": "attention", "dtype": dtype, "lengths": lengths, "cached": cached, "heads": heads, "kv_heads": kv, "dk": dk, "dv": dv, "latent": latent,
                "window": size if mask == "window" else 0, "keep_first": 4 if mask == "window" and rng.random() < 0.5 else 0, "chunk": size if mask == "chunk" else 0,
                "softcap": rng.choice([0.0, 30.0]), "sinks": rng.random() < 0.4, "gate": "none" if latent else rng.choice(["none", "entry", "head"]),
                "step": kind == "attention_step"}
    if kind == "retention":
        return {"kind": "retention", "dtype": dtype, "lengths": _ragged(rng, 2048, 4), "heads": rng.choice([4, 6, 8]), "dk": rng.choice([64, 96, 128]),
                "dv": rng.choice([64, 128]), "rotate": rng.random() < 0.5, "finish": rng.random() < 0.6}
    if kind == "recurrence":
        cell = rng.choice(["delta_rule", "matrix_memory", "gated_linear"])
        return {"kind": "recurrence", "cell": cell, "dtype": "float32" if cell == "delta_rule" else dtype, "lengths": _ragged(rng, 2048, 4),
                "heads": rng.choice([4, 6, 8]), "dk": rng.choice([64, 96, 128]), "dv": rng.choice([64, 128])}
    if kind == "head_maps":
        n_in, n_out = rng.choice([(64, 256), (256, 64), (64, 128), (128, 64), (32, 192)])
        gate = n_in > n_out and rng.random() < 0.5
        return {"kind": "head_maps", "dtype": dtype, "rows": _log(rng, 65, 2048), "heads": rng.choice([8, 16]), "n_in": n_in, "n_out": n_out, "gate": gate}
    return {"kind": "experts", "dtype": dtype, "rows": _log(rng, 1, 32), "top": rng.choice([1, 2, 4]), "experts": rng.choice([8, 16]),
            "n_in": rng.choice([704, 1024, 1408]), "n_out": rng.choice([1024, 1408])}


def _ints(text):
    return [int(x) for x in str(text).split()]


def _gen(seed, what=0):
    g = torch.Generator(device="cuda")
    g.manual_seed((int(seed) * 1000003 + what) & 0x7FFFFFFF)
    return g


def _randn(g, *shape, std=1.0, mean=0.0, dtype=torch.float32):
    return (torch.randn(*shape, generator=g, device="cuda") * std + mean).to(dtype)


def _i32(values):
    return torch.tensor(values, dtype=torch.int32, device="cuda")


def _starts(lengths):
    return [0] + [int(x) for x in np.cumsum(lengths)]


# ---- GPT-2 through the engine ------------------------------------------------------------------------------------------


def _gpt2_weights(case, seed):
    """A checkpoint's tensors on the GPU, in the compute dtype: matrices ~ N(0, 0.02), the two that write to the residual stream
    smaller, gains about one."""
    g, e, inner, n = _gen(seed, 1), case["width"], case["inner"], case["layers"]
    t = DT[case["dtype"]]
    resid = 0.02 / math.sqrt(2 * n)
    w = {"wte.weight": _randn(g, case["vocab"], e, std=0.02, dtype=t), "wpe.weight": _randn(g, case["positions"], e, std=0.02, dtype=t)}
    for i in range(n):
        p = "h.%d." % i
        for ln in ("ln_1", "ln_2"):
            w[p + ln + ".weight"], w[p + ln + ".bias"] = _randn(g, e, std=0.05, mean=1.0, dtype=t), _randn(g, e, std=0.02, dtype=t)
        for name, a, b, std in (("attn.c_attn", e, 3 * e, 0.02), ("attn.c_proj", e, e, resid), ("mlp.c_fc", e, inner, 0.02), ("mlp.c_proj", inner, e, resid)):
            w[p + name + ".weight"], w[p + name + ".bias"] = _randn(g, a, b, std=std, dtype=t), _randn(g, b, std=0.01, dtype=t)
    w["ln_f.weight"], w["ln_f.bias"] = _randn(g, e, std=0.05, mean=1.0, dtype=t), _randn(g, e, std=0.02, dtype=t)
    return w


def _gpt2_tokens(case, seed):
    g, v = torch.Generator().manual_seed(int(seed) + 17), case["vocab"]
    prompts = [torch.randint(0, v, (n,), generator=g).tolist() for n in _ints(case["lengths"])]
    more = [torch.randint(0, v, (case.get("steps", 0),), generator=g).tolist() for _ in prompts]
    return prompts, more


def _gpt2_engine(case, seed):
    weights = _gpt2_weights(case, seed)
    prompts, more = _gpt2_tokens(case, seed)
    config = {"model_type": "gpt2", "n_layer": case["layers"], "n_embd": case["width"], "n_head": case["heads"], "n_inner": case["inner"],
              "vocab_size": case["vocab"], "n_positions": case["positions"], "layer_norm_epsilon": 1e-5, "activation_function": "gelu_new"}
    with tempfile.TemporaryDirectory(prefix="gpt2-") as folder:
        with open(os.path.join(folder, "config.json"), "w") as f:
            json.dump(config, f)
        head, at = {}, 0
        for name, w in weights.items():
            size = w.numel() * w.element_size()
            head[name] = {"dtype": "BF16" if w.dtype == torch.bfloat16 else "F32", "shape": list(w.shape), "data_offsets": [at, at + size]}
            at += size
        text = json.dumps(head).encode()
        text += b" " * (-len(text) % 8)
        with open(os.path.join(folder, "model.safetensors"), "wb") as f:
            f.write(struct.pack("<Q", len(text)) + text)
            for w in weights.values():
                w.contiguous().view(torch.uint8).cpu().numpy().tofile(f)
        tokens = sum((len(p) + len(m) + PAGE) // PAGE * PAGE for p, m in zip(prompts, more))
        return Engine.from_pretrained(folder, case["dtype"], max_tokens=tokens + PAGE), prompts, more


def _run_gpt2(s):
    engine = s["engine"]
    slots = [engine.open() for _ in s["prompts"]]
    out = [engine.step([StepEntry(slot, p, (len(p) - 1,)) for slot, p in zip(slots, s["prompts"])]).clone()]
    for j in range(len(s["more"][0])):
        out.append(engine.step([StepEntry(slot, (m[j],), (0,)) for slot, m in zip(slots, s["more"])]).clone())
    for slot in slots:
        engine.close(slot)
    return out


def _exact_gpt2(case, seed):
    w = {k: v.double() for k, v in _gpt2_weights(case, seed).items()}
    prompts, more = _gpt2_tokens(case, seed)
    e, H = case["width"], case["heads"]
    norm = lambda x, p: torch.nn.functional.layer_norm(x, (e,), w[p + ".weight"], w[p + ".bias"], 1e-5)  # noqa: E731
    lin = lambda x, p: x @ w[p + ".weight"] + w[p + ".bias"]  # noqa: E731
    rows = []
    for p, m in zip(prompts, more):
        t = torch.tensor(p + m, device="cuda")
        x = w["wte.weight"][t] + w["wpe.weight"][: len(t)]
        hide = torch.triu(torch.ones(len(t), len(t), dtype=torch.bool, device="cuda"), 1)
        for i in range(case["layers"]):
            b = "h.%d." % i
            q, k, v = lin(norm(x, b + "ln_1"), b + "attn.c_attn").view(len(t), 3, H, e // H).permute(1, 2, 0, 3)
            a = ((q @ k.transpose(1, 2)) / math.sqrt(e // H)).masked_fill(hide, -math.inf).softmax(-1)
            x = x + lin((a @ v).permute(1, 0, 2).reshape(len(t), e), b + "attn.c_proj")
            x = x + lin(torch.nn.functional.gelu(lin(norm(x, b + "ln_2"), b + "mlp.c_fc"), approximate="tanh"), b + "mlp.c_proj")
        rows.append(norm(x[len(p) - 1:], "ln_f") @ w["wte.weight"].t())
    return [torch.stack([r[j] for r in rows]) for j in range(len(more[0]) + 1)]


def _work_gpt2(case):
    lengths, e, b = _ints(case["lengths"]), case["width"], 2 if case["dtype"] == "bfloat16" else 4
    steps = 1 + case.get("steps", 0)
    matrices = case["layers"] * (4 * e * e + 2 * e * case["inner"])
    head = case["vocab"] * e
    rows, keys = sum(lengths), sum(n * (n + 1) // 2 for n in lengths)
    kept = sum(lengths)
    for j in range(1, steps):
        rows += len(lengths)
        keys += sum(n + j for n in lengths)
        kept += sum(n + j for n in lengths)
    out = len(lengths) * steps * case["vocab"] * 4
    return {"bytes": steps * (matrices + head) * b + case["layers"] * 2 * e * b * kept + out,
            "flops": 2.0 * rows * matrices + 2.0 * len(lengths) * steps * head + 4.0 * case["layers"] * e * keys}


# ---- attention with shaped scores over the paged cache -------------------------------------------------------------------


def _attention(case, seed):
    t, g = DT[case["dtype"]], _gen(seed, 2)
    lengths, cached = _ints(case["lengths"]), _ints(case["cached"])
    total = [n + c for n, c in zip(lengths, cached)]
    H, G, dk, dv = case["heads"], case["kv_heads"], case["dk"], case["dv"]
    pages = [-(-n // PAGE) for n in total]
    order = torch.randperm(sum(pages), generator=torch.Generator().manual_seed(int(seed))).tolist()
    width = max(max(pages), 16)
    table, at = [], 0
    for p in pages:
        table.append(order[at:at + p] + [0] * (width - p))
        at += p
    n = sum(lengths)
    s = {"q": _randn(g, n, H * dk, dtype=t), "k_pages": _randn(g, sum(pages), G, PAGE, dk, dtype=t),
         "v_pages": None if case["latent"] else _randn(g, sum(pages), G, PAGE, dv, dtype=t), "table": _i32(table), "starts": _i32(_starts(lengths)),
         "lens": _i32(total), "gate": None, "sinks": _randn(g, H) if case["sinks"] else None}
    if case["gate"] != "none":
        s["gate"] = _randn(g, n, H * dv if case["gate"] == "entry" else H, dtype=t)
    return s, lengths, cached


def _prepare_attention(case, seed):
    s, lengths, _ = _attention(case, seed)
    t, H, G, dv = DT[case["dtype"]], case["heads"], case["kv_heads"], case["dv"]
    ops, n, group = Ops(t), sum(lengths), H // G
    splits, scratch = 1, None
    if case["step"]:
        reach = case["window"] + case["keep_first"] if case["window"] else min(case["chunk"] or 1 << 30, s["table"].shape[1] * PAGE)
        splits = ops.scored_splits(n, G, group, reach)
        scratch = torch.empty(n * H * splits * (dv + 2), device="cuda") if splits > 1 else None
    per_block = min(group, 32) if case["step"] else max(d for d in (1, 2, 4) if group % d == 0)
    s.update(ops=ops, out=torch.empty(n, H * dv, device="cuda", dtype=t), n_seqs=len(lengths), max_new=max(lengths), heads=H, scale=case["dk"] ** -0.5, value_dim=dv,
             more=dict(softcap=case["softcap"], window=case["window"], keep_first=case["keep_first"], chunk=case["chunk"], sinks=s["sinks"], gate=s["gate"],
                       heads_per_block=per_block, n_splits=splits, scratch=scratch))
    return s


def _run_attention(s):
    s["ops"].attention_scored(s["q"], s["out"], s["starts"], s["lens"], s["n_seqs"], s["max_new"], s["table"], s["k_pages"], s["v_pages"], s["heads"], s["scale"],
                              value_dim=s["value_dim"], **s["more"])
    return s["out"]


def _seen(case, past, n):
    """[rows, keys]: whether row i (position past + i) sees key j."""
    i, j = torch.arange(past, past + n, device="cuda")[:, None], torch.arange(past + n, device="cuda")[None, :]
    ok = j <= i
    if case["window"]:
        ok &= (i - j < case["window"]) | (j < case["keep_first"])
    if case["chunk"]:
        ok &= torch.div(i, case["chunk"], rounding_mode="floor") == torch.div(j, case["chunk"], rounding_mode="floor")
    return ok


def _exact_attention(case, seed):
    s, lengths, cached = _attention(case, seed)
    H, G, dk, dv = case["heads"], case["kv_heads"], case["dk"], case["dv"]
    out, at = [], 0
    for i, (n, past) in enumerate(zip(lengths, cached)):
        pages = s["table"][i, : -(-(n + past) // PAGE)].long()
        k = s["k_pages"][pages].double().permute(1, 0, 2, 3).reshape(G, -1, dk)[:, : n + past]
        v = k[..., :dv] if case["latent"] else s["v_pages"][pages].double().permute(1, 0, 2, 3).reshape(G, -1, dv)[:, : n + past]
        q = s["q"][at:at + n].double().view(n, G, H // G, dk).permute(1, 2, 0, 3)
        x = (q @ k[:, None].transpose(2, 3)) * dk ** -0.5
        if case["softcap"]:
            x = case["softcap"] * torch.tanh(x / case["softcap"])
        x = x.masked_fill(~_seen(case, past, n), -math.inf)
        if s["sinks"] is not None:
            x = torch.cat([x, s["sinks"].double().view(G, H // G, 1, 1).expand(-1, -1, n, 1)], dim=-1)
        p = x.softmax(-1)[..., : n + past]
        o = (p @ v[:, None]).permute(2, 0, 1, 3).reshape(n, H, dv)
        if s["gate"] is not None:
            o = o * torch.sigmoid(s["gate"][at:at + n].double().view(n, H, -1))
        out.append(o.reshape(n, H * dv))
        at += n
    return torch.cat(out)


def _work_attention(case):
    lengths, cached, b = _ints(case["lengths"]), _ints(case["cached"]), 2 if case["dtype"] == "bfloat16" else 4
    H, G, dk, dv = case["heads"], case["kv_heads"], case["dk"], case["dv"]
    n, pairs, keys = sum(lengths), 0, 0
    for m, past in zip(lengths, cached):
        first = past
        for i in range(past, past + m):
            lo = i - i % case["chunk"] if case["chunk"] else max(0, i - case["window"] + 1) if case["window"] else 0
            pairs += i - lo + 1 + min(lo, case["keep_first"])
            first = min(first, lo)
        keys += past + m - first + min(first, case["keep_first"])
    gate = {"none": 0, "entry": H * dv, "head": H}[case["gate"]]
    return {"bytes": b * (n * (H * (dk + dv) + gate) + keys * G * (dk + (0 if case["latent"] else dv))), "flops": 2.0 * pairs * H * (dk + dv)}


# ---- retention -----------------------------------------------------------------------------------------------------------


def _retention(case, seed):
    t, g = DT[case["dtype"]], _gen(seed, 3)
    lengths, H, dk, dv = _ints(case["lengths"]), case["heads"], case["dk"], case["dv"]
    n = sum(lengths)
    rows = _randn(g, n, H * (2 * dk + 2 * dv), dtype=t)          # q | k | v | gate, as the fused projection leaves them
    a, b, c = H * dk, 2 * H * dk, 2 * H * dk + H * dv
    s = {"q": rows[:, :a], "k": rows[:, a:b], "v": rows[:, b:c], "gate": rows[:, c:] if case["finish"] else None,
         "decay": torch.tensor([1.0 - 2.0 ** (-5 - i % 6) for i in range(H)], dtype=torch.float32, device="cuda"),
         "freq": (1e6 ** (-torch.arange(0, dk, 2, device="cuda", dtype=torch.float64) / dk)).float() if case["rotate"] else None}
    return s, lengths


def _prepare_retention(case, seed):
    s, lengths = _retention(case, seed)
    t, H, dk, dv = DT[case["dtype"]], case["heads"], case["dk"], case["dv"]
    n = sum(lengths)
    s.update(ops=Ops(t), heads=H, n_seqs=len(lengths), starts=_i32(_starts(lengths)), lens=_i32(lengths), slots=_i32(list(range(len(lengths)))),
             state=torch.zeros(len(lengths), H, dk, dv, device="cuda"), raw=torch.empty(n, H * dv, device="cuda"),
             out=torch.empty(n, H * dv, device="cuda", dtype=t) if case["finish"] else None, rot=dk if case["rotate"] else 0, key_scale=dk ** -0.5)
    return s


def _run_retention(s):
    s["ops"].zero(s["state"])          # new sequences
    finish = s["out"] is not None
    s["ops"].retention(s["q"], s["k"], s["v"], s["out"], s["state"], s["starts"], s["lens"], s["slots"], s["n_seqs"], s["decay"], s["heads"], inv_freq=s["freq"],
                       rot_dims=s["rot"], k_scale=s["key_scale"], gate=s["gate"], unit_norm_eps=1e-5 if finish else None, raw=s["raw"], raw_only=not finish)
    return {"out": s["out"] if finish else s["raw"], "state": s["state"]}


def _exact_retention(case, seed):
    s, lengths = _retention(case, seed)
    H, dk, dv = case["heads"], case["dk"], case["dv"]
    decay = s["decay"].double()
    outs, states, at = [], [], 0
    for n in lengths:
        q, k, v = (s[x][at:at + n].double().view(n, H, -1).transpose(0, 1) for x in ("q", "k", "v"))
        if case["rotate"]:
            angle = torch.arange(n, device="cuda").double()[:, None] * s["freq"].double()
            c, sn = torch.cos(angle), torch.sin(angle)
            turn = lambda x: torch.cat([x[..., : dk // 2] * c - x[..., dk // 2:] * sn, x[..., dk // 2:] * c + x[..., : dk // 2] * sn], -1)  # noqa: E731
            q, k = turn(q), turn(k)
        k = k * dk ** -0.5
        i = torch.arange(n, device="cuda").double()
        far = (i[:, None] - i[None, :])
        d = torch.where(far >= 0, decay[:, None, None] ** far.clamp(min=0), 0.0)
        o = ((q @ k.transpose(1, 2)) * d) @ v
        states.append((k * (decay[:, None] ** (n - 1 - i))[..., None]).transpose(1, 2) @ v)
        o = o.transpose(0, 1)
        if case["finish"]:
            z = s["gate"][at:at + n].double().view(n, H, dv)
            o = o / torch.sqrt(o.square().mean(-1, keepdim=True) + 1e-5) * z * torch.sigmoid(z)
        outs.append(o.reshape(n, H * dv))
        at += n
    return {"out": torch.cat(outs), "state": torch.stack(states)}


def _work_retention(case):
    n, seqs, H, dk, dv = sum(_ints(case["lengths"])), len(_ints(case["lengths"])), case["heads"], case["dk"], case["dv"]
    b = 2 if case["dtype"] == "bfloat16" else 4
    out = n * H * dv * (2 * b if case["finish"] else 4)
    return {"bytes": n * H * (2 * dk + dv) * b + out + 4 * seqs * H * dk * dv, "flops": 4.0 * n * H * dk * dv}


# ---- recurrences with gates that depend on the token -------------------------------------------------------------------------


def _recurrence(case, seed):
    t, g, cell = DT[case["dtype"]], _gen(seed, 4), case["cell"]
    lengths, H, dk, dv = _ints(case["lengths"]), case["heads"], case["dk"], case["dv"]
    n = sum(lengths)
    s = {"beta": None, "a_log": None, "dt_bias": None}
    q, k, v = _randn(g, n, H, dk), _randn(g, n, H, dk), _randn(g, n, H * dv, dtype=t)
    if cell == "delta_rule":            # unit vectors, as the convolution's kernel leaves them; decays ready, as for prompts
        q, k = torch.nn.functional.normalize(q, dim=-1) * dk ** -0.5, torch.nn.functional.normalize(k, dim=-1)
        s["a_log"], s["dt_bias"] = _randn(g, H, std=0.5, mean=-1.0), _randn(g, H * dk, std=0.5, mean=-1.0)
        s["beta"] = torch.sigmoid(_randn(g, n, H))
        s["gates"] = torch.exp(-torch.exp(s["a_log"]).repeat_interleave(dk) * torch.nn.functional.softplus(_randn(g, n, H * dk) + s["dt_bias"]))
    elif cell == "gated_linear":
        s["gates"] = torch.sigmoid(_randn(g, n, H * dk, mean=1.0)) ** (1.0 / 12.0)
    else:                               # input and forget projections, the latter leaning to remembering
        s["gates"] = _randn(g, n, 2 * H)
        s["gates"][:, H:] += 3.0
    s.update(q=q.reshape(n, H * dk).to(t), k=k.reshape(n, H * dk).to(t), v=v)
    return s, lengths


def _prepare_recurrence(case, seed):
    s, lengths = _recurrence(case, seed)
    H, dk, dv, cell = case["heads"], case["dk"], case["dv"], case["cell"]
    ops = Ops(DT[case["dtype"]])
    s.update(ops=ops, cell=cell, heads=H, dk=dk, dv=dv, starts=_i32(_starts(lengths)), slots=_i32(list(range(len(lengths)))), n_seqs=len(lengths),
             state=torch.zeros(len(lengths), ops.recurrence_state_size(cell, H, dk, dv), device="cuda"), out=torch.empty(sum(lengths), H * dv, device="cuda"),
             more={"delta_rule": dict(beta=s["beta"], a_log=s["a_log"], dt_bias=s["dt_bias"], gates_ready=True), "gated_linear": dict(gates_ready=True, tau=12.0),
                   "matrix_memory": dict(cap=15.0)}[cell], q_scale=1.0 if cell == "delta_rule" else dk ** -0.5)
    return s


def _run_recurrence(s):
    s["ops"].zero(s["state"])          # new sequences
    s["ops"].gated_recurrence(s["cell"], s["q"], s["k"], s["v"], s["gates"], s["out"], s["state"], s["starts"], s["slots"], s["n_seqs"], s["heads"], s["heads"],
                              s["dk"], s["dv"], q_scale=s["q_scale"], **s["more"])
    return {"out": s["out"], "state": s["state"]}


def _exact_recurrence(case, seed):
    s, lengths = _recurrence(case, seed)
    H, dk, dv, cell = case["heads"], case["dk"], case["dv"], case["cell"]
    n_seqs, longest = len(lengths), max(lengths)
    starts = _starts(lengths)

    def rows(x, per_head):          # [longest, sequences, heads, ...], zeros after a sequence's end
        x = x.double().view(x.shape[0], *per_head)
        y = torch.zeros(longest, n_seqs, *per_head, dtype=torch.float64, device="cuda")
        for i, m in enumerate(lengths):
            y[:m, i] = x[starts[i]:starts[i] + m]
        return y

    q, k, v = rows(s["q"], (H, dk)), rows(s["k"], (H, dk)), rows(s["v"], (H, dv))
    q = q * (1.0 if cell == "delta_rule" else dk ** -0.5)
    live = (torch.arange(longest, device="cuda")[:, None] < torch.tensor(lengths, device="cuda")).double()[:, :, None]
    S = torch.zeros(n_seqs, H, dv, dk, dtype=torch.float64, device="cuda")
    norm, m = torch.zeros(n_seqs, H, dk, dtype=torch.float64, device="cuda"), torch.zeros(n_seqs, H, dtype=torch.float64, device="cuda")
    outs = []
    if cell == "matrix_memory":
        both = rows(s["gates"], (2 * H,))
        take, keep = 15.0 * torch.tanh(both[..., :H] / 15.0), torch.nn.functional.logsigmoid(15.0 * torch.tanh(both[..., H:] / 15.0))
    else:
        g = rows(s["gates"], (H, dk))
        beta = rows(s["beta"], (H,)) if cell == "delta_rule" else None
    for i in range(longest):
        on = live[i]
        if cell == "matrix_memory":
            new = torch.maximum(keep[i] + m, take[i])
            f, w = torch.exp(keep[i] + m - new), torch.exp(take[i] - new)
            S1 = f[..., None, None] * S + w[..., None, None] * v[i][..., None] * k[i][:, :, None]
            norm1 = f[..., None] * norm + w[..., None] * k[i]
            o = (S1 @ q[i][..., None])[..., 0] / (torch.maximum((norm1 * q[i]).sum(-1).abs(), torch.exp(-new)) + 1e-6)[..., None]
            norm, m = torch.where(on[..., None] > 0, norm1, norm), torch.where(on > 0, new, m)
        else:
            S1 = S * g[i][:, :, None]
            u = v[i] if beta is None else beta[i][..., None] * (v[i] - (S1 @ k[i][..., None])[..., 0])
            S1 = S1 + u[..., None] * k[i][:, :, None]
            o = (S1 @ q[i][..., None])[..., 0]
        S = torch.where(on[..., None, None] > 0, S1, S)
        outs.append(o)
    outs = torch.stack(outs)
    state = S.reshape(n_seqs, -1)
    if cell == "matrix_memory":          # the normaliser and the running maximum are kept once per 16 value columns
        tiles = -(-dv // 16)
        state = torch.cat([state, norm[:, :, None].expand(-1, -1, tiles, -1).reshape(n_seqs, -1), m[:, :, None].expand(-1, -1, tiles).reshape(n_seqs, -1)], 1)
    return {"out": torch.cat([outs[:x, i].reshape(x, H * dv) for i, x in enumerate(lengths)]), "state": state}


def _work_recurrence(case):
    n, seqs, H, dk, dv = sum(_ints(case["lengths"])), len(_ints(case["lengths"])), case["heads"], case["dk"], case["dv"]
    b = 2 if case["dtype"] == "bfloat16" else 4
    gates = {"delta_rule": dk + 1, "gated_linear": dk, "matrix_memory": 2}[case["cell"]]
    dots = {"delta_rule": 3, "gated_linear": 2, "matrix_memory": 2}[case["cell"]]
    return {"bytes": n * H * ((2 * dk + dv) * b + 4 * gates + 4 * dv) + 4 * seqs * H * dk * dv, "flops": 2.0 * dots * n * H * dk * dv}


# ---- head-wise maps, experts --------------------------------------------------------------------------------------------------


def _head_maps(case, seed):
    t, g, H = DT[case["dtype"]], _gen(seed, 5), case["heads"]
    gate = _randn(g, case["rows"], H * case["n_out"], dtype=t) if case["gate"] else None
    return {"a": _randn(g, case["rows"], H * case["n_in"], dtype=t), "w": _randn(g, H, case["n_out"], case["n_in"], std=case["n_in"] ** -0.5, dtype=t), "gate": gate}


def _prepare_head_maps(case, seed):
    s = _head_maps(case, seed)
    s.update(ops=Ops(DT[case["dtype"]]), out=torch.empty(case["rows"], case["heads"] * case["n_out"], device="cuda", dtype=DT[case["dtype"]]), n_in=case["n_in"],
             n_out=case["n_out"])
    return s


def _run_head_maps(s):
    s["ops"].linear_heads(s["a"], s["w"], s["out"], head_stride_a=s["n_in"], head_stride_out=s["n_out"], gate=s["gate"])
    return s["out"]


def _exact_head_maps(case, seed):
    s = _head_maps(case, seed)
    o = torch.einsum("rhi,hji->rhj", s["a"].double().view(case["rows"], case["heads"], -1), s["w"].double()).reshape(case["rows"], -1)
    return o if s["gate"] is None else o * torch.sigmoid(s["gate"].double())


def _work_head_maps(case):
    b, n, H, i, o = 2 if case["dtype"] == "bfloat16" else 4, case["rows"], case["heads"], case["n_in"], case["n_out"]
    return {"bytes": b * (n * H * (i + o * (2 if case["gate"] else 1)) + H * i * o), "flops": 2.0 * n * H * i * o}


EXPERT_TILE = 32          # positions a tile of few rows holds


def _experts(case, seed):
    """Hidden rows grouped by the expert that they chose, every expert's list padded to whole tiles; which expert a tile is."""
    t, g = DT[case["dtype"]], _gen(seed, 6)
    slots, E = case["rows"] * case["top"], case["experts"]
    logits = torch.randn(case["rows"], E, generator=torch.Generator().manual_seed(int(seed)))
    chosen = logits.topk(case["top"], dim=1).indices.reshape(-1).tolist()
    valid, tile_expert = [], []
    for e in range(E):
        mine = [i for i, x in enumerate(chosen) if x == e]
        pad = -len(mine) % EXPERT_TILE
        tile_expert += [e] * ((len(mine) + pad) // EXPERT_TILE)
        valid += mine + [-1] * pad
    spare = min(slots, slots // EXPERT_TILE + E) - len(tile_expert)          # a step's lists are as long as its shape can need
    valid, tile_expert = valid + [-1] * (spare * EXPERT_TILE), tile_expert + [-1] * spare
    hidden = torch.zeros(len(valid), case["n_in"], device="cuda", dtype=t)
    places = torch.tensor([p for p, i in enumerate(valid) if i >= 0], device="cuda")
    hidden[places] = _randn(g, slots, case["n_in"], dtype=t)
    return {"hid": hidden, "w": _randn(g, E, case["n_out"], case["n_in"], std=case["n_in"] ** -0.5, dtype=t), "valid": _i32(valid), "tile_expert": _i32(tile_expert)}


def _prepare_experts(case, seed):
    s = _experts(case, seed)
    ops = Ops(DT[case["dtype"]])
    s.update(ops=ops, outs=torch.zeros(s["hid"].shape[0], case["n_out"], device="cuda"), few=case["rows"] * case["top"] <= ops.MOE_FEW_SLOTS)
    return s


def _run_experts(s):
    s["ops"].grouped_linear(s["hid"], s["w"], s["outs"], s["tile_expert"], s["valid"], few_rows=s["few"])
    return s["outs"]


def _exact_experts(case, seed):
    s = _experts(case, seed)
    out = torch.zeros(s["hid"].shape[0], case["n_out"], dtype=torch.float64, device="cuda")
    for i, e in enumerate(s["tile_expert"].tolist()):
        if e >= 0:
            rows = slice(i * EXPERT_TILE, (i + 1) * EXPERT_TILE)
            out[rows] = s["hid"][rows].double() @ s["w"][e].double().t()
    return out


def _work_experts(case):
    b, slots = 2 if case["dtype"] == "bfloat16" else 4, case["rows"] * case["top"]
    used = case["experts"] * (1.0 - (1.0 - case["top"] / case["experts"]) ** case["rows"])      # experts that at least one row chooses, on average
    return {"bytes": used * case["n_in"] * case["n_out"] * b + slots * (case["n_in"] * b + case["n_out"] * 4), "flops": 2.0 * slots * case["n_in"] * case["n_out"]}


# ---- what the measurement calls ---------------------------------------------------------------------------------------------------


_PREPARE = {"attention": _prepare_attention, "retention": _prepare_retention, "recurrence": _prepare_recurrence, "head_maps": _prepare_head_maps,
            "experts": _prepare_experts}
_RUN = {"prompt": _run_gpt2, "decode": _run_gpt2, "attention": _run_attention, "retention": _run_retention, "recurrence": _run_recurrence,
        "head_maps": _run_head_maps, "experts": _run_experts}
_EXACT = {"prompt": _exact_gpt2, "decode": _exact_gpt2, "attention": _exact_attention, "retention": _exact_retention, "recurrence": _exact_recurrence,
          "head_maps": _exact_head_maps, "experts": _exact_experts}
_WORK = {"prompt": _work_gpt2, "decode": _work_gpt2, "attention": _work_attention, "retention": _work_retention, "recurrence": _work_recurrence,
         "head_maps": _work_head_maps, "experts": _work_experts}


def prepare(case, seed):
    if case["kind"] in ("prompt", "decode"):
        engine, prompts, more = _gpt2_engine(case, seed)
        return {"kind": case["kind"], "engine": engine, "prompts": prompts, "more": more}
    return dict(_PREPARE[case["kind"]](case, seed), kind=case["kind"])


def run(state):
    return _RUN[state["kind"]](state)


def exact(case, seed):
    return _EXACT[case["kind"]](case, seed)


def work(case):
    return _WORK[case["kind"]](case)


def tolerance(case):
    """bfloat16: one rounding of the stored result; through a whole model, of every activation on the way.  float32: sums in another
    order; the recurrences carry theirs from row to row, and the matrix memory divides by a sum that can nearly cancel."""
    if case["kind"] in ("prompt", "decode"):
        return {"rel": 2e-2} if case["dtype"] == "bfloat16" else {"rel": 1e-5}
    if case["kind"] == "recurrence":
        return {"rel": 2e-4} if case["cell"] == "matrix_memory" else {"rel": 1e-5}
    if case["kind"] == "experts":
        return {"rel": 1e-5}
    return {"rel": 1e-2} if case["dtype"] == "bfloat16" else {"rel": 1e-5}


if __name__ == "__main__":
    for c in listed() + [draw(random.Random(i)) for i in range(12)]:
        print(c, work(c))
