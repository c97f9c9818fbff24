"""Steps of decoder models on the model runner, the unit of work of a serving engine: one prefill step over the new tokens of a
few requests, or one decode step (a replayed CUDA graph) of a running batch.

Six families, in bf16: dense decoders (the Llama-3-8B and Qwen3-32B shapes), routed experts (the Qwen3-30B-A3B shape), latent
attention with routed and shared experts (DeepSeek-V3's layers), and the hybrids Qwen3-Next (gated delta rule and gated attention)
and Kimi-Linear (per-channel delta rule and latent attention without positions).  The last three have the sizes of the benchmark
of hybrid decoders ("latent-moe" and "moe": width 2048, 8 of 64 experts of 768).  Models are cut to four layers and a vocabulary of
32768, so that the output head keeps about its share of a step.  Weights, token ids, cached keys and values and recurrent states
are random; requests are ragged and their pages lie scattered over the pool.

A state is a runner with loaded weights, its caches filled for the requests of the case and, for decode, its captured graph.  A pass
is one `ModelRunner.forward`; it returns the logits and the caches, which hold what the step wrote (new keys and values or latents,
convolution windows, recurrent states).  The greedy token, which a step also makes, is a function of the logits: with random weights
the two largest are often nearly the same, so that tokens would say less than the logits."""

from __future__ import annotations

import math
import os
import tempfile
import zlib

import numpy as np
import torch

PAGE = 64
LAYERS = 4
VOCAB = 32768
CONTEXT = 8192                       # longest sequence, as in the benchmark of hybrid decoders
EPS = 1e-6

FAMILIES = {
    "llama": dict(width=4096, heads=32, kv_heads=8, dim=128, ff=14336, theta=5e5),
    "qwen3": dict(width=5120, heads=64, kv_heads=8, dim=128, ff=25600, theta=1e6, qk_norm=True),
    "qwen3_moe": dict(width=2048, heads=32, kv_heads=4, dim=128, ff=768, experts=128, top=8, theta=1e6, qk_norm=True),
    "deepseek": dict(width=2048, heads=16, ff=768, experts=64, top=8, shared=True, rank=512, q_rank=768, nope=128, rot=64, vdim=128,
                     theta=1e4),
    "qwen3_next": dict(width=2048, heads=16, kv_heads=4, dim=128, ff=768, experts=64, top=8, theta=1e4, rot_share=0.5,
                       d_heads=16, d_kv=8, d_dim=128, conv=4),
    "kimi": dict(width=2048, heads=16, ff=768, experts=64, top=8, rank=512, nope=128, rot=64, vdim=128, d_heads=16, d_kv=16,
                 d_dim=128, conv=4),
}
# new tokens of a prefill step, at most (the prefill step of a chunked prompt; shorter for the costlier families)
MOST = {"llama": 8192, "qwen3": 8192, "qwen3_moe": 4096, "deepseek": 4096, "qwen3_next": 4096, "kimi": 1024}


def listed():
    d = lambda name, family, seqs, context: dict(name=name, family=family, phase="decode", seqs=seqs, context=context)
    p = lambda name, family, seqs, tokens, prefix: dict(name=name, family=family, phase="prefill", seqs=seqs, tokens=tokens,
                                                        context=prefix)
    return [
        d("llama-decode-1", "llama", 1, 1024),                  # one user waits for one token
        d("qwen3-decode-128", "qwen3", 128, 2304),              # the headline workload: 128 running requests
        d("qwen3_moe-decode-64", "qwen3_moe", 64, 1536),        # routed experts under a middling load
        d("deepseek-decode-96", "deepseek", 96, 2560),          # latent attention over long contexts
        d("qwen3_next-decode-32", "qwen3_next", 32, 2048),      # hybrids: states instead of keys and values in half the layers
        d("kimi-decode-7", "kimi", 7, 1200),                    # a small batch
        p("llama-prefill-293", "llama", 1, 293, 0),             # one short prompt: time to the first token
        p("qwen3-prefill-8192", "qwen3", 7, 8192, 0),           # the headline workload: a full step of prompts
        p("qwen3_moe-prefill-4096", "qwen3_moe", 4, 4096, 0),   # prompts of about 1024 tokens
        p("deepseek-prefill-3000", "deepseek", 3, 3000, 512),   # prompts behind a shared prefix
        p("qwen3_next-prefill-2500", "qwen3_next", 3, 2500, 0),
        p("kimi-prefill-1024", "kimi", 1, 1024, 0),             # one prompt of 1024 tokens
    ]


def draw(rng):
    family = rng.choice(sorted(FAMILIES))
    logu = lambda a, b: int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))
    if rng.random() < 0.5:
        return dict(family=family, phase="decode", seqs=logu(1, 128), context=logu(64, 2304))
    tokens = logu(16, MOST[family])
    # a prompt's later chunk, or one that shares a prefix, in a third of the steps
    prefix = logu(64, 2048) if rng.random() < 0.34 and tokens <= 4096 else 0
    return dict(family=family, phase="prefill", seqs=min(logu(1, 16), max(tokens // 8, 1)), tokens=tokens, context=prefix)


# ------------------------------------------------------------------------------------------------ the requests of a case
def requests(case):
    """`(cached tokens, new tokens)` of every request, set by the sizes of the case."""
    rs = np.random.RandomState(case["seqs"] * 7919 + case["context"] * 31 + case.get("tokens", 0))
    B = case["seqs"]
    if case["phase"] == "decode":
        cached = rs.randint(case["context"] // 2, case["context"] + 1, B)
        cached[rs.randint(B)] = case["context"]
        return cached, np.ones(B, np.int64)
    share = rs.uniform(0.4, 1.6, B)
    new = np.maximum((share / share.sum() * case["tokens"]).astype(np.int64), 1)
    new[np.argmax(new)] += case["tokens"] - new.sum()
    cached = rs.randint(case["context"] // 2, case["context"] + 1, B) if case["context"] else np.zeros(B, np.int64)
    return cached, new


def layout(case, seed):
    """Scattered pages: `(pages of each request, pages in all)`; page 0 is the pool's dummy."""
    cached, new = requests(case)
    n = -(-(cached + new) // PAGE)
    order = np.random.RandomState(seed % (2 ** 31) + 1).permutation(int(n.sum())) + 1
    return np.split(order, np.cumsum(n)[:-1]), int(n.sum())


def token_ids(case, seed):
    return np.random.RandomState(seed % (2 ** 31) + 2).randint(1, VOCAB, int(requests(case)[1].sum())).astype(np.int32)


def generator(seed, name):
    return torch.Generator(device="cuda").manual_seed((seed * 1000003 + zlib.crc32(name.encode())) % (2 ** 62))


def kinds(f):
    """Kind of mixer of every layer: the hybrids alternate, recurrence first."""
    second = "mla" if "rank" in FAMILIES[f] else "attention"
    return [("delta" if i % 2 == 0 else second) if "d_heads" in FAMILIES[f] else second for i in range(LAYERS)]


# ------------------------------------------------------------------------------------------------------------ weights
def shapes(family):
    """Checkpoint tensors by their published names: `name -> (shape, kind)`."""
    s, f = {}, FAMILIES[family]
    W = f["width"]
    s["model.embed_tokens.weight"] = ((VOCAB, W), "embed")
    for i, kind in enumerate(kinds(family)):
        p = f"model.layers.{i}."
        a = p + "self_attn."
        if kind == "attention":
            H, K, D = f["heads"], f["kv_heads"], f["dim"]
            s[a + "q_proj.weight"] = ((H * D * (2 if family == "qwen3_next" else 1), W), "w")
            s[a + "k_proj.weight"] = s[a + "v_proj.weight"] = ((K * D, W), "w")
            s[a + "o_proj.weight"] = ((W, H * D), "w")
            if f.get("qk_norm") or family == "qwen3_next":
                s[a + "q_norm.weight"] = s[a + "k_norm.weight"] = ((D,), "norm")
        elif kind == "mla":
            H, qk = f["heads"], f["nope"] + f["rot"]
            if "q_rank" in f:
                s[a + "q_a_proj.weight"] = ((f["q_rank"], W), "w")
                s[a + "q_a_layernorm.weight"] = ((f["q_rank"],), "norm")
                s[a + "q_b_proj.weight"] = ((H * qk, f["q_rank"]), "w")
            else:
                s[a + "q_proj.weight"] = ((H * qk, W), "w")
            s[a + "kv_a_proj_with_mqa.weight"] = ((f["rank"] + f["rot"], W), "w")
            s[a + "kv_a_layernorm.weight"] = ((f["rank"],), "norm")
            s[a + "kv_b_proj.weight"] = ((H * (f["nope"] + f["vdim"]), f["rank"]), "w")
            s[a + "o_proj.weight"] = ((W, H * f["vdim"]), "w")
        elif family == "qwen3_next":
            d, K, V = p + "linear_attn.", f["d_kv"] * f["d_dim"], f["d_heads"] * f["d_dim"]
            s[d + "in_proj_qkvz.weight"] = ((2 * K + 2 * V, W), "w")
            s[d + "in_proj_ba.weight"] = ((2 * f["d_heads"], W), "w")
            s[d + "conv1d.weight"] = ((2 * K + V, 1, f["conv"]), "conv")
            s[d + "dt_bias"], s[d + "A_log"] = ((f["d_heads"],), "dt"), ((f["d_heads"],), "A")
            s[d + "norm.weight"] = ((f["d_dim"],), "norm")
            s[d + "out_proj.weight"] = ((W, V), "w")
        else:
            P, D = f["d_heads"] * f["d_dim"], f["d_dim"]
            for x in "qkv":
                s[a + x + "_proj.weight"] = ((P, W), "w")
                s[a + x + "_conv1d.weight"] = ((P, 1, f["conv"]), "conv")
            for x in "fg":
                s[a + x + "_a_proj.weight"], s[a + x + "_b_proj.weight"] = ((D, W), "w"), ((P, D), "w")
            s[a + "b_proj.weight"] = ((f["d_heads"], W), "w")
            s[a + "dt_bias"], s[a + "A_log"] = ((P,), "dt"), ((f["d_heads"],), "A")
            s[a + "o_norm.weight"] = ((D,), "norm")
            s[a + "o_proj.weight"] = ((W, P), "w")
        s[p + "input_layernorm.weight"] = s[p + "post_attention_layernorm.weight"] = ((W,), "norm")
        m = p + "mlp."
        if "experts" in f:
            s[m + "gate.weight"] = ((f["experts"], W), "router")
            s[m + "experts.gate_up_proj"] = ((f["experts"], 2 * f["ff"], W), "w")
            s[m + "experts.down_proj"] = ((f["experts"], W, f["ff"]), "w")
            m += "shared_experts."
        if "experts" not in f or f.get("shared"):
            s[m + "gate_proj.weight"] = s[m + "up_proj.weight"] = ((f["ff"], W), "w")
            s[m + "down_proj.weight"] = ((W, f["ff"]), "w")
    s["model.norm.weight"] = ((W,), "norm")
    s["lm_head.weight"] = ((VOCAB, W), "w")
    return s


def tensor(family, name, shape, kind, seed):
    """One checkpoint tensor.  Projections keep unit variance; routers are sharper, as trained ones are: the last of the chosen
    experts weighs little, so that a choice made by a hair does not decide the result; the decays of the recurrences lie between 0.2 and 0.999 a token."""
    g = generator(seed, name)
    if kind == "A":
        return torch.empty(shape, device="cuda").uniform_(1.0, 8.0, generator=g).log_()
    if kind == "dt":                                  # inverse softplus of a step between 0.001 and 0.1
        t = torch.empty(shape, device="cuda").uniform_(math.log(1e-3), math.log(1e-1), generator=g).exp_()
        return t + torch.log(-torch.expm1(-t))
    std = {"embed": 1.0, "norm": 0.1, "conv": 0.5, "router": 4.0 * shape[-1] ** -0.5, "w": shape[-1] ** -0.5}[kind]
    w = torch.empty(shape, dtype=torch.bfloat16, device="cuda").normal_(0.0, std, generator=g)
    if kind == "norm" and not (family == "qwen3_next" and "linear_attn" not in name):   # its other norms are stored around zero
        w += 1.0
    return w


def config(family):
    f = FAMILIES[family]
    c = dict(hidden_size=f["width"], intermediate_size=f["ff"], num_hidden_layers=LAYERS, rms_norm_eps=EPS, vocab_size=VOCAB,
             max_position_embeddings=32768, tie_word_embeddings=False, torch_dtype="bfloat16", num_attention_heads=f["heads"],
             num_key_value_heads=f.get("kv_heads", f["heads"]), rope_theta=f.get("theta", 1e4), hidden_act="silu")
    if "dim" in f:
        c["head_dim"] = f["dim"]
    if "experts" in f:
        c.update(num_experts=f["experts"], num_experts_per_tok=f["top"], moe_intermediate_size=f["ff"], norm_topk_prob=True)
    if "rank" in f:
        c.update(kv_lora_rank=f["rank"], q_lora_rank=f.get("q_rank"), qk_nope_head_dim=f["nope"], qk_rope_head_dim=f["rot"],
                 v_head_dim=f["vdim"])
    names = {"llama": ("LlamaForCausalLM", "llama"), "qwen3": ("Qwen3ForCausalLM", "qwen3"),
             "qwen3_moe": ("Qwen3MoeForCausalLM", "qwen3_moe"), "deepseek": ("DeepseekV3ForCausalLM", "deepseek_v3"),
             "qwen3_next": ("Qwen3NextForCausalLM", "qwen3_next"), "kimi": ("KimiLinearForCausalLM", "kimi_linear")}[family]
    c.update(architectures=[names[0]], model_type=names[1])
    if family == "qwen3_moe":
        c.update(decoder_sparse_step=1, mlp_only_layers=[])
    elif family == "deepseek":
        c.update(n_routed_experts=f["experts"], n_shared_experts=1, scoring_func="softmax", topk_method="noaux_tc",
                 routed_scaling_factor=1.0, first_k_dense_replace=0)
    elif family == "qwen3_next":
        c.update(full_attention_interval=2, partial_rotary_factor=f["rot_share"], linear_num_value_heads=f["d_heads"],
                 linear_num_key_heads=f["d_kv"], linear_key_head_dim=f["d_dim"], linear_value_head_dim=f["d_dim"],
                 linear_conv_kernel_dim=f["conv"])
    elif family == "kimi":
        c.update(mla_use_nope=True, n_shared_experts=0,
                 linear_attn_config={"kda_layers": [i + 1 for i, k in enumerate(kinds(family)) if k == "delta"],
                                     "num_heads": f["d_heads"], "head_dim": f["d_dim"], "short_conv_kernel_size": f["conv"]})
    return c


# ----------------------------------------------------------------------------------------------------------- the caches
def cache_shape(family, pages):
    f = FAMILIES[family]
    return (pages + 1, PAGE, f["rank"] + f["rot"]) if "rank" in f else (pages + 1, 2, f["kv_heads"], PAGE, f["dim"])


def fill_cache(t, seed, layer):
    """Cached keys and values, or latents: normalised vectors."""
    return t.normal_(0.0, 1.0, generator=generator(seed, f"cache{layer}"))


def fill_state(conv, rec, seed, layer):
    conv.normal_(0.0, 1.0, generator=generator(seed, f"conv{layer}"))
    rec.normal_(0.0, 0.05, generator=generator(seed, f"state{layer}"))


def state_shapes(family, B):
    f = FAMILIES[family]
    C = (2 * f["d_kv"] + f["d_heads"]) * f["d_dim"]
    return (B, C, f["conv"] - 1), (B, f["d_heads"], f["d_dim"], f["d_dim"])


# ----------------------------------------------------------------------------------------------------- prepare and run
def prepare(case, seed):
    from sglang_jax_b200.configs.model_config import ModelConfig
    from sglang_jax_b200.managers.schedule_batch import ForwardMode, ModelWorkerBatch, ModelWorkerSamplingInfo
    from sglang_jax_b200.model_executor.cuda_graph_runner import DEFAULT_BS_BUCKETS, CudaGraphRunner
    from sglang_jax_b200.model_executor.model_runner import ModelRunner
    from sglang_jax_b200.parallel import state as ps
    from sglang_jax_b200.server_args import ServerArgs
    from sglang_jax_b200.utils.tiny_models import write_config_only
    if not ps.get_state().initialized:
        ps.init_distributed(0, 1, "cuda")
    family, B = case["family"], case["seqs"]
    decode = case["phase"] == "decode"
    cached, new = requests(case)
    pages, total = layout(case, seed)
    path = write_config_only(os.path.join(tempfile.gettempdir(), f"perf_cases_{family}"), config(family))
    args = ServerArgs(model_path=path, load_format="dummy", device="cuda", dtype="bfloat16", page_size=PAGE,
                      max_total_tokens=total * PAGE, max_running_requests=B, context_length=CONTEXT, skip_tokenizer_init=True,
                      disable_overlap_schedule=True, disable_radix_cache=True, disable_cuda_graph=True, mem_fraction_static=0.9)
    runner = ModelRunner(ModelConfig.from_server_args(args), args)
    with torch.inference_mode():
        runner.model.load_weights((n, tensor(family, n, sh, kind, seed)) for n, (sh, kind) in shapes(family).items())
    kept = {}
    if decode:
        def keep(_module, _args, out):                 # the logits of the captured greedy step
            if torch.cuda.is_current_stream_capturing():
                kept.setdefault("logits", out.next_token_logits)
        bucket = min(b for b in DEFAULT_BS_BUCKETS if b >= B)
        args.precompile_bs_paddings, args.cuda_graph_max_bs = [bucket], bucket
        hook = runner.model.register_forward_hook(keep)
        runner.cuda_graph_runner = CudaGraphRunner(runner)
        hook.remove()
        if runner.gemm_plan is not None:
            runner.gemm_plan.save()
    pool, rows = runner.req_to_token_pool, np.arange(B, dtype=np.int32)
    for b in range(B):
        pool.write(b, 0, (pages[b][:, None] * PAGE + np.arange(PAGE)).ravel()[:cached[b] + new[b]])
    r, c, ids = (torch.from_numpy(x).cuda() for x in pool.take_page_deltas())
    pool.page_table[r.long(), c.long()] = ids
    caches = runner.token_to_kv_pool.kv_buffer
    with torch.inference_mode():
        for i, t in enumerate(caches):
            assert tuple(t.shape) == cache_shape(family, total)
            fill_cache(t, seed, i)
        outputs = [t[1:] for t in caches]
        if runner.recurrent_pool is not None:
            conv, rec = runner.recurrent_pool.conv_state, runner.recurrent_pool.recurrent_state
            shape = state_shapes(family, B)
            for i in range(len(conv)):
                x, y = torch.empty(shape[0], dtype=torch.bfloat16, device="cuda"), torch.empty(shape[1], device="cuda")
                fill_state(x, y, seed, i)
                conv[i, 1:B + 1] = x
                rec[i, 1:B + 1] = y
                outputs += [conv[i, 1:B + 1], rec[i, 1:B + 1]]
    f = lambda v: np.asarray(v, np.int32)
    where = [pool.read(b, int(cached[b] + new[b]))[int(cached[b]):] for b in range(B)]
    batch = dict(input_ids=token_ids(case, seed), req_pool_indices=rows, seq_lens=f(cached + new), out_cache_loc=f(np.concatenate(where)),
                 positions=f(np.concatenate([np.arange(c, c + n) for c, n in zip(cached, new)])),
                 sampling_info=ModelWorkerSamplingInfo(np.ones(B, np.float32), np.ones(B, np.float32), np.ones(B, np.int32),
                                                       np.zeros(B, np.float32), None, True, False, False, False))
    if not decode:
        batch.update(extend_prefix_lens=f(cached), extend_seq_lens=f(new), extend_logprob_start_lens=f(np.zeros(B)))
    mode = ForwardMode.DECODE if decode else ForwardMode.EXTEND
    return dict(runner=runner, batch=ModelWorkerBatch(bid=0, forward_mode=mode, **batch), outputs=outputs,
                logits=kept["logits"][:B] if decode else None)


def run(state):
    out, _, _ = state["runner"].forward(state["batch"])
    logits = state["logits"] if out is None else out.next_token_logits
    return {"logits": logits, "caches": state["outputs"]}


# --------------------------------------------------------------------------------------------------------------- work
def work(case):
    family, f = case["family"], FAMILIES[case["family"]]
    cached, new = requests(case)
    T, B, W = int(new.sum()), case["seqs"], FAMILIES[case["family"]]["width"]
    pairs = float(sum(n * c + n * (n + 1) / 2 for c, n in zip(cached, new)))          # (query, key) pairs of one head
    hit = f["experts"] * (1.0 - (1.0 - f["top"] / f["experts"]) ** T) / f["experts"] if "experts" in f else 1.0
    weights = flops = 0.0
    for name, (shape, _) in shapes(family).items():
        n = float(np.prod(shape))
        if name.startswith("model.embed"):
            weights += T * W
        elif name.startswith("lm_head"):
            weights, flops = weights + n, flops + 2 * n * B
        elif ".experts." in name:
            weights, flops = weights + n * hit, flops + 2 * n * T * f["top"] / f["experts"]
        elif "kv_b_proj" in name:                      # folded into the queries and the result in decode, applied to all keys else
            weights, flops = weights + n, flops + 2 * n * (T if case["phase"] == "decode" else T + float(cached.sum()))
        else:
            weights, flops = weights + n, flops + 2 * n * T
    moved = 2 * weights + 2.0 * B * VOCAB
    for kind in kinds(family):
        if kind == "delta":
            D = f["d_dim"]
            flops += 6.0 * T * f["d_heads"] * D * D                                     # decay and read, write, read-out
            states = float(np.prod(state_shapes(family, B)[1])) * 4 + float(np.prod(state_shapes(family, B)[0])) * 2
            moved += states * (2 if case["context"] else 1)
        else:
            row = f["rank"] + f["rot"] if kind == "mla" else 2 * f["kv_heads"] * f["dim"]
            moved += 2.0 * row * float((cached + new).sum())
            if kind == "attention":
                flops += 4.0 * pairs * f["heads"] * f["dim"]
            elif case["phase"] == "decode":
                flops += 2.0 * pairs * f["heads"] * (2 * f["rank"] + f["rot"])
            else:
                flops += 2.0 * pairs * f["heads"] * (f["nope"] + f["rot"] + f["vdim"])
    return {"bytes": moved, "flops": flops}


def tolerance(case):
    # bf16 activations and caches through four layers: steps of one state rounded in other places are between 0.003 and 0.008 apart.
    # Where an expert is chosen by a hair, single tokens can move further
    return {"rel": 0.03, "max": 0.9 if "experts" in FAMILIES[case["family"]] else 0.3}


# -------------------------------------------------------------------------------------------------------------- exact
def rms(x, w=None):
    x = x * torch.rsqrt(x.square().mean(-1, keepdim=True) + EPS)
    return x if w is None else x * w


def rope(x, pos, theta, rot, interleaved):
    """Rotates the first `rot` lanes of `x [T, heads, lanes]`."""
    inv = theta ** (-torch.arange(0, rot, 2, dtype=torch.float64, device=x.device) / rot)
    a = (pos.double()[:, None] * inv)[:, None]
    c, s = a.cos(), a.sin()
    y, rest = x[..., :rot], x[..., rot:]
    if interleaved:
        u, v = y[..., 0::2], y[..., 1::2]
        y = torch.stack([u * c - v * s, v * c + u * s], -1).flatten(-2)
    else:
        u, v = y.chunk(2, -1)
        y = torch.cat([u * c - v * s, v * c + u * s], -1)
    return torch.cat([y, rest], -1)


def attend(q, k, v, cached, scale):
    """Causal attention of one request: `q [n, H, d]`, `k [s, K, d]`, `v [s, K, e]`, one group of heads at a time."""
    n, H, r = q.shape[0], q.shape[1], q.shape[1] // k.shape[1]
    seen = torch.arange(k.shape[0], device=q.device)[None] <= torch.arange(cached, cached + n, device=q.device)[:, None]
    o = torch.empty(n, H, v.shape[-1], dtype=q.dtype, device=q.device)
    for h in range(H):
        p = (q[:, h] @ k[:, h // r].t() * scale).masked_fill_(~seen, float("-inf"))
        o[:, h] = torch.softmax(p, -1) @ v[:, h // r]
    return o


def delta_rule(q, k, v, decay, beta, S, cu):
    """`S <- decay S + beta k (v - (decay S)^T k)^T; o = S^T q` for ragged sequences: `q, k [T, H, D]`, `decay [T, H, D or 1]`."""
    q, k = (x * torch.rsqrt(x.square().sum(-1, keepdim=True) + 1e-6) for x in (q, k))
    q = q * q.shape[-1] ** -0.5
    o = torch.empty_like(v)
    n = cu[1:] - cu[:-1]
    for t in range(int(n.max())):
        on = np.nonzero(n > t)[0]
        at, on = torch.from_numpy(cu[:-1][on] + t).cuda(), torch.from_numpy(on).cuda()
        M = S[on] * decay[at].unsqueeze(-1)
        u = (v[at] - torch.einsum("bhd,bhde->bhe", k[at], M)) * beta[at].unsqueeze(-1)
        M = M + k[at].unsqueeze(-1) * u.unsqueeze(-2)
        S[on] = M
        o[at] = torch.einsum("bhd,bhde->bhe", q[at], M)
    return o


def convolve(x, w, window, cu):
    """Causal convolution and SiLU per sequence; `window [B, C, taps - 1]` holds the inputs before, and is moved on."""
    y = torch.empty_like(x)
    taps = w.shape[-1]
    for b in range(len(cu) - 1):
        full = torch.cat([window[b].t(), x[cu[b]:cu[b + 1]]], 0)
        n = int(cu[b + 1] - cu[b])
        y[cu[b]:cu[b + 1]] = sum(full[j:j + n] * w[:, j] for j in range(taps))
        window[b] = full[-(taps - 1):].t()
    return torch.nn.functional.silu(y)


@torch.inference_mode()
def exact(case, seed):
    family, f, B = case["family"], FAMILIES[case["family"]], case["seqs"]
    cached, new = requests(case)
    pages, total = layout(case, seed)
    cu = np.concatenate([[0], np.cumsum(new)])
    T, W = int(cu[-1]), f["width"]
    shape = shapes(family)
    silu = torch.nn.functional.silu

    def w(name):
        x = tensor(family, name, *shape[name], seed).double()
        return x + 1.0 if shape[name][1] == "norm" and family == "qwen3_next" and "linear_attn" not in name else x

    pos = torch.from_numpy(np.concatenate([np.arange(c, c + n) for c, n in zip(cached, new)])).cuda()
    slots = [torch.from_numpy((pages[b][:, None] * PAGE + np.arange(PAGE)).ravel()[:cached[b] + new[b]]).cuda() for b in range(B)]
    slot = torch.cat([slots[b][int(cached[b]):] for b in range(B)])
    x = w("model.embed_tokens.weight")[torch.from_numpy(token_ids(case, seed)).long().cuda()]
    caches, states = [], []
    for i, kind in enumerate(kinds(family)):
        p = f"model.layers.{i}."
        a = p + "self_attn."
        h = rms(x, w(p + "input_layernorm.weight"))
        if kind != "delta":
            cache = torch.empty(cache_shape(family, total), dtype=torch.bfloat16, device="cuda")
            cache = fill_cache(cache, seed, len(caches)).double()
            caches.append(cache[1:])
        if kind == "attention":
            H, K, D = f["heads"], f["kv_heads"], f["dim"]
            q = (h @ w(a + "q_proj.weight").t()).view(T, H, -1)
            gate, q = (q[..., D:], q[..., :D]) if family == "qwen3_next" else (None, q)
            k, v = ((h @ w(a + y + "_proj.weight").t()).view(T, K, D) for y in "kv")
            if a + "q_norm.weight" in shape:
                q, k = rms(q, w(a + "q_norm.weight")), rms(k, w(a + "k_norm.weight"))
            rot = int(D * f.get("rot_share", 1.0))
            q, k = rope(q, pos, f["theta"], rot, False), rope(k, pos, f["theta"], rot, False)
            cache[slot // PAGE, 0, :, slot % PAGE], cache[slot // PAGE, 1, :, slot % PAGE] = k, v
            o = torch.cat([attend(q[cu[b]:cu[b + 1]], cache[slots[b] // PAGE, 0, :, slots[b] % PAGE],
                                  cache[slots[b] // PAGE, 1, :, slots[b] % PAGE], int(cached[b]), D ** -0.5) for b in range(B)])
            o = o if gate is None else o * torch.sigmoid(gate)
            x = x + o.reshape(T, H * D) @ w(a + "o_proj.weight").t()
        elif kind == "mla":
            H, R, nope, rot, vd = f["heads"], f["rank"], f["nope"], f["rot"], f["vdim"]
            if "q_rank" in f:
                q = rms(h @ w(a + "q_a_proj.weight").t(), w(a + "q_a_layernorm.weight")) @ w(a + "q_b_proj.weight").t()
            else:
                q = h @ w(a + "q_proj.weight").t()
            q = q.view(T, H, nope + rot)
            c = h @ w(a + "kv_a_proj_with_mqa.weight").t()
            q_pe, k_pe = q[..., nope:], c[:, None, R:]
            if "theta" in f:
                q_pe, k_pe = rope(q_pe, pos, f["theta"], rot, True), rope(k_pe, pos, f["theta"], rot, True)
            cache.view(-1, R + rot)[slot] = torch.cat([rms(c[:, :R], w(a + "kv_a_layernorm.weight")), k_pe[:, 0]], -1)
            up = w(a + "kv_b_proj.weight").view(H, nope + vd, R)
            q = torch.cat([torch.einsum("thn,hnr->thr", q[..., :nope], up[:, :nope]), q_pe], -1)
            o = []
            for b in range(B):
                seen = cache.view(-1, R + rot)[slots[b]][:, None]
                o.append(attend(q[cu[b]:cu[b + 1]], seen, seen[..., :R], int(cached[b]), (nope + rot) ** -0.5))
            o = torch.einsum("thr,hvr->thv", torch.cat(o), up[:, nope:]).reshape(T, H * vd)
            x = x + o @ w(a + "o_proj.weight").t()
        else:
            H, K, D = f["d_heads"], f["d_kv"], f["d_dim"]
            conv, S = (torch.empty(s, dtype=t, device="cuda") for s, t in zip(state_shapes(family, B), (torch.bfloat16, torch.float32)))
            fill_state(conv, S, seed, len(states) // 2)
            conv, S = conv.double(), S.double()
            fresh = torch.from_numpy(cached == 0).cuda()
            conv[fresh], S[fresh] = 0.0, 0.0
            states += [conv, S]
            if family == "qwen3_next":
                d, r = p + "linear_attn.", H // K
                q, k, v, z = (h @ w(d + "in_proj_qkvz.weight").t()).view(T, K, -1).split([D, D, r * D, r * D], -1)
                beta, dt = (y.reshape(T, H) for y in (h @ w(d + "in_proj_ba.weight").t()).view(T, K, 2 * r).split([r, r], -1))
                taps, out, norm = w(d + "conv1d.weight")[:, 0], w(d + "out_proj.weight"), w(d + "norm.weight")
                decay = torch.exp(-w(d + "A_log").exp() * torch.nn.functional.softplus(dt + w(d + "dt_bias")))[..., None]
                gate = silu(z.reshape(T, H, D))
            else:
                q, k, v = (h @ w(a + y + "_proj.weight").t() for y in "qkv")
                taps = torch.cat([w(a + y + "_conv1d.weight")[:, 0] for y in "qkv"])
                low = lambda y: (h @ w(a + y + "_a_proj.weight").t()) @ w(a + y + "_b_proj.weight").t()
                step = torch.nn.functional.softplus(low("f") + w(a + "dt_bias")).view(T, H, D)
                decay = torch.exp(-w(a + "A_log").exp()[:, None] * step)
                beta, gate = h @ w(a + "b_proj.weight").t(), torch.sigmoid(low("g").view(T, H, D))
                out, norm = w(a + "o_proj.weight"), w(a + "o_norm.weight")
            y = convolve(torch.cat([t.reshape(T, -1) for t in (q, k, v)], -1), taps, conv, cu)
            q, k, v = y.split([K * D, K * D, H * D], -1)
            q, k = (t.reshape(T, K, D).repeat_interleave(H // K, 1) for t in (q, k))
            o = delta_rule(q, k, v.reshape(T, H, D), decay, torch.sigmoid(beta), S, cu)
            x = x + (rms(o, norm) * gate).reshape(T, H * D) @ out.t()
        h = rms(x, w(p + "post_attention_layernorm.weight"))
        m = p + "mlp."
        if "experts" in f:
            score = torch.softmax(h @ w(m + "gate.weight").t(), -1)
            best, ids = score.topk(f["top"], -1)
            best = best / best.sum(-1, keepdim=True)
            up, down = (tensor(family, m + n, *shape[m + n], seed) for n in ("experts.gate_up_proj", "experts.down_proj"))
            y = torch.zeros_like(h)
            for e in range(f["experts"]):
                tok, j = (ids == e).nonzero(as_tuple=True)
                if len(tok):
                    g, u = (h[tok] @ up[e].double().t()).chunk(2, -1)
                    y.index_add_(0, tok, (silu(g) * u) @ down[e].double().t() * best[tok, j][:, None])
            x = x + y
            m += "shared_experts."
        if m + "up_proj.weight" in shape:
            x = x + (silu(h @ w(m + "gate_proj.weight").t()) * (h @ w(m + "up_proj.weight").t())) @ w(m + "down_proj.weight").t()
    last = torch.from_numpy(cu[1:] - 1).cuda()
    logits = rms(x[last], w("model.norm.weight")) @ w("lm_head.weight").t()
    return {"logits": logits, "caches": caches + states}
