"""Logits of the GPT-2 / Qwen2 shapes in plain torch: in float64 what decode steps are compared with, in float32 how far plain fp32
arithmetic is from it."""
import math

import numpy as np
import torch


def lm_logits(tensors, spec, ids, positions, device="cuda", dtype=torch.float64):
    """ids [rows][T] -> logits [rows][len(positions)][V] of a causal pass (reference src/gpt2.c:96-158, src/qwen.c:112-190)."""
    qwen, C, H, kv, rows = spec.kind == "qwen", spec.n_embd, spec.n_head, spec.n_kv_heads, ids.shape[0]
    hd, T = C // H, ids.shape[1]
    w = lambda n: torch.from_numpy(np.ascontiguousarray(tensors[n])).to(device, dtype)
    idx = torch.from_numpy(ids.astype(np.int64)).to(device)
    emb = w("model.embed_tokens.weight" if qwen else "wte.weight")
    x = emb[idx] if qwen else emb[idx] + w("wpe.weight")[:T]

    def norm(v, name):
        if qwen:
            return v / torch.sqrt((v * v).mean(-1, keepdim=True) + 1e-6) * w(name + ".weight")
        d = v - v.mean(-1, keepdim=True)
        return d / torch.sqrt((d * d).mean(-1, keepdim=True) + 1e-5) * w(name + ".weight") + w(name + ".bias")

    if qwen:                                                  # the tables are fp32 by definition
        inv = spec.rope_theta ** (-2.0 * torch.arange(hd // 2, device=device, dtype=torch.float64) / hd)
        a = torch.arange(T, device=device, dtype=torch.float64)[:, None] * inv
        cos, sin = (torch.cat([f(a)] * 2, 1).float().to(dtype) for f in (torch.cos, torch.sin))
        turn = lambda z: z * cos + torch.cat([-z[..., hd // 2:], z[..., :hd // 2]], -1) * sin
    else:
        turn = lambda z: z
    lin = lambda v, n, bias=True: v @ w(n + ".weight").T + (w(n + ".bias") if bias else 0)
    heads = lambda v, n: v.view(rows, T, n, hd).transpose(1, 2)
    mask = torch.full((T, T), -math.inf, device=device, dtype=dtype).triu(1)
    for i in range(spec.n_layer):
        p = f"model.layers.{i}." if qwen else f"h.{i}."
        n = norm(x, p + ("input_layernorm" if qwen else "ln_1"))
        if qwen:
            q, k, v = (lin(n, f"{p}self_attn.{c}_proj") for c in "qkv")
        else:
            q, k, v = lin(n, p + "attn.c_attn").split(C, -1)
        q, k, v = turn(heads(q, H)), turn(heads(k, kv)), heads(v, kv)
        k, v = k.repeat_interleave(H // kv, 1), v.repeat_interleave(H // kv, 1)
        o = ((q @ k.transpose(-1, -2) / math.sqrt(hd) + mask).softmax(-1) @ v).transpose(1, 2).reshape(rows, T, C)
        x = x + (lin(o, p + "self_attn.o_proj", False) if qwen else lin(o, p + "attn.c_proj"))
        n = norm(x, p + ("post_attention_layernorm" if qwen else "ln_2"))
        if qwen:
            g = lin(n, p + "mlp.gate_proj", False)
            x = x + lin(g * torch.sigmoid(g) * lin(n, p + "mlp.up_proj", False), p + "mlp.down_proj", False)
        else:
            h = lin(n, p + "mlp.c_fc")
            x = x + lin(0.5 * h * (1 + torch.tanh(math.sqrt(2 / math.pi) * (h + 0.044715 * h ** 3))), p + "mlp.c_proj")
    return (norm(x[:, positions], "model.norm" if qwen else "ln_f") @ emb.T).cpu().numpy()
