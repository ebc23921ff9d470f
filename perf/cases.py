"""Workloads of the engine as a serving program runs them: decode steps, speculative windows, batched decode, prompts, and the
expert block of the mixture-of-experts families at the row counts those calls give it.

Geometries are the repository's own configurations (small hybrid, dense hybrid 27B, the two 512-expert MoE geometries), cut to
a few layers of the same kind: with random weights every further layer amplifies rounding differences, and at eight layers two
correct kernels already differ by 2 % in the logits.  Prompts and fed tokens are random ids: a pass feeds given tokens (as
scoring does) instead of its own picks, so that a near-tie between two of a random model's logits cannot send two runs
different ways.  For the same reason the experts are measured as blocks on given rows: inside a random model a rounding
difference moves the tenth-best of 512 experts for every few tokens.
"""
import math

import torch

from r4dx_b200 import native
from r4dx_b200.config import qwen4_exp_config, qwen_hybrid_27b_config, qwen_hybrid_moe_config, small_hybrid_config
from r4dx_b200.models.batch import BatchModel
from r4dx_b200.models.hybrid import HybridModel
from r4dx_b200.models.moe import MoeBlock
from r4dx_b200.quant.trellis import TrellisWeight, packed_words, random_weight
from r4dx_b200.quant.weights import default_kb_rule, linear_shapes, moe_kb_rule, synthetic_weight_set
from r4dx_b200.runtime.engine import GreedySession

CONFIGS = {"small": small_hybrid_config, "dense": qwen_hybrid_27b_config, "moe": qwen_hybrid_moe_config,
           "streams": qwen4_exp_config}


def listed():
    return [
        # a reply's tokens from a small model at a short context: launches and host calls are what it is made of
        {"name": "decode_small", "path": "decode", "family": "small", "layers": 4, "ctx": 100, "rows": 1, "steps": 16},
        # the headline: one user's reply from the dense model after an 8k prompt
        {"name": "decode_dense_8k", "path": "decode", "family": "dense", "layers": 8, "ctx": 8192, "rows": 1, "steps": 4},
        # a reply deep in a long document (ragged length): the KV cache is a real share of the step
        {"name": "decode_dense_32k", "path": "decode", "family": "dense", "layers": 4, "ctx": 32517, "rows": 1, "steps": 4},
        # speculative decoding, next-token head: windows of one anchor and three drafts
        {"name": "window_dense_4", "path": "window", "family": "dense", "layers": 8, "ctx": 2048, "rows": 4, "steps": 4},
        # speculative decoding, block drafter: windows of one anchor and seven drafts
        {"name": "window_dense_8", "path": "window", "family": "dense", "layers": 4, "ctx": 4099, "rows": 8, "steps": 4},
        # a server with 16 users of the dense model, each with a context of its own
        {"name": "batch_dense_16", "path": "batch", "family": "dense", "layers": 4, "ctx": 512, "rows": 16, "steps": 1},
        # a chat turn's prompt of a few hundred tokens
        {"name": "prompt_dense_333", "path": "prompt", "family": "dense", "layers": 4, "ctx": 333, "rows": 1, "steps": 1},
        # the headline prompt: cold, 8192 tokens in one chunk
        {"name": "prompt_dense_8k", "path": "prompt", "family": "dense", "layers": 8, "ctx": 8192, "rows": 1, "steps": 1},
        # a long document (several chunks, ragged tail): attention over the earlier chunks grows
        {"name": "prompt_dense_30k", "path": "prompt", "family": "dense", "layers": 8, "ctx": 30011, "rows": 1, "steps": 1},
        # the experts of one decoded token of the 512-expert model (a replayed graph, as in its decode step)
        {"name": "experts_1", "path": "experts", "family": "moe", "layers": 4, "ctx": 0, "rows": 1, "steps": 1},
        # the experts of a step of 64 concurrent users
        {"name": "experts_64", "path": "experts", "family": "moe", "layers": 4, "ctx": 0, "rows": 64, "steps": 1},
        # the experts of a prompt chunk
        {"name": "experts_4k", "path": "experts", "family": "moe", "layers": 4, "ctx": 0, "rows": 4096, "steps": 1},
    ]


def draw(rng):
    def spread(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    path = rng.choice(["decode", "decode", "window", "batch", "prompt", "prompt", "experts"])
    case = {"path": path, "family": "dense", "layers": rng.choice([4, 8]), "ctx": 0, "rows": 1, "steps": 1}
    if path == "decode":
        case["family"] = rng.choice(["small", "dense", "dense"])
        case.update(ctx=spread(20, 4000 if case["family"] == "small" else 32000), steps=rng.choice([4, 8]))
    elif path == "window":
        case.update(ctx=spread(20, 12000), rows=rng.randint(2, 8), steps=4)
    elif path == "batch":
        case.update(layers=4, ctx=spread(40, 1000), rows=spread(2, 64))
    elif path == "prompt":
        case["family"] = rng.choice(["small", "dense", "dense"])
        case["ctx"] = spread(12, 8000 if case["family"] == "small" else 24000)
    else:
        case.update(family=rng.choice(["moe", "streams"]), layers=rng.choice([2, 3, 4]), rows=spread(1, 6000))
    return case


def _config(case):
    return CONFIGS[case["family"]](case["layers"])


def _kb_rule(case):
    return moe_kb_rule if case["path"] == "experts" else default_kb_rule


def _tokens(g, cfg, *shape):
    return torch.randint(0, cfg.vocab_size, shape, generator=g, dtype=torch.int32)


def _prepare_experts(case, seed):
    cfg, rows = _config(case), case["rows"]
    H, inner, shared, E = cfg.hidden_size, cfg.moe_intermediate_size, cfg.shared_expert_intermediate_size, cfg.num_experts
    g = torch.Generator(device="cuda").manual_seed(seed)

    def normal(*shape, scale=1.0):
        return (torch.randn(*shape, generator=g, device="cuda") * scale).to(torch.bfloat16)

    def signs(*shape):
        return (torch.randint(0, 2, shape, generator=g, device="cuda") * 2 - 1).to(torch.float16)

    def stack(N, K, kb):
        words = torch.randint(-2**31, 2**31 - 1, (E, packed_words(N, K, kb)), generator=g, device="cuda", dtype=torch.int32)
        suh, svh = signs(E, K), signs(E, N) * 0.02
        return [TrellisWeight(words[e], suh[e], svh[e], N, K, kb) for e in range(E)]

    blocks = []
    for i in range(case["layers"]):
        p = f"text.layers.{i}.moe."
        kb = moe_kb_rule(p + "experts.0.gate_up")
        w = {p + "router": normal(E, H, scale=0.02), p + "shared_gate": normal(1, H, scale=0.02),
             p + "shared.gate_up": random_weight(2 * shared, H, moe_kb_rule(p + "shared.gate_up"), seed=seed + i, device="cuda"),
             p + "shared.down": random_weight(H, shared, moe_kb_rule(p + "shared.down"), seed=seed + i + 64, device="cuda")}
        for name, N, K in (("gate_up", 2 * inner, H), ("down", H, inner)):
            w.update({p + f"experts.{e}.{name}": t for e, t in enumerate(stack(N, K, kb))})
        blocks.append(MoeBlock(cfg, w, i, "cuda", max(rows, 8)))
    s = {"case": case, "blocks": blocks, "h": [normal(rows, H) for _ in blocks], "x": [normal(rows, H) for _ in blocks], "graph": None}
    if rows <= 8:
        _run_blocks(s)                                  # loads the kernels before the capture
        torch.cuda.synchronize()
        s["graph"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(s["graph"]):
            _run_blocks(s)
    return s


def _run_blocks(s):
    for block, h, x in zip(s["blocks"], s["h"], s["x"]):
        block.forward(h, x, s["case"]["rows"], residual=False)


def prepare(case, seed):
    """A loaded model (weights, caches, workspaces, captured decode graphs) with the case's context already in it."""
    native.cuda()
    if case["path"] == "experts":
        return _prepare_experts(case, seed)
    cfg, g = _config(case), torch.Generator().manual_seed(seed)
    w = synthetic_weight_set(cfg, device="cuda", seed=seed % 1000003, kb_rule=_kb_rule(case))
    path, ctx, rows, steps = case["path"], case["ctx"], case["rows"], case["steps"]
    s = {"case": case}
    if path == "batch":
        # every slot has its own prompt; lengths vary by user.  The room past it is for the tokens that passes add.
        m = BatchModel(cfg, w, slots=rows, slot_ctx=ctx + 4096, device="cuda")
        for j in range(rows):
            n = max(1, ctx - int(torch.randint(0, ctx // 4 + 1, (1,), generator=g)))
            m.import_slot(j, _tokens(g, cfg, n).tolist())
        s.update(model=m, slots=list(range(rows)), tokens=_tokens(g, cfg, rows).tolist())
        return s
    max_ctx = ctx + 64
    m = HybridModel(cfg, w, max_ctx=max_ctx, device="cuda")
    m.reserve_prefill(min(ctx, 8192))
    s.update(model=m, prompt=_tokens(g, cfg, ctx))
    if path == "prompt":
        return s
    m.prefill(s["prompt"])
    s["fed"] = _tokens(g, cfg, steps, rows).tolist()
    if path == "decode":
        s["session"] = GreedySession(m)
    else:
        m.enable_graphs((rows,))
    s["checkpoint"] = m.save_checkpoint()
    return s


def _state(m):
    """The recurrent state that a call leaves behind."""
    return [m.gdn_state[i] for i in sorted(m.gdn_state)]


def run(s):
    case = s["case"]
    if case["path"] == "experts":
        if s["graph"] is not None:
            s["graph"].replay()
        else:
            _run_blocks(s)
        return s["x"]
    m = s["model"]
    if case["path"] == "batch":
        if m.pos[0] + 2 > m.slot_ctx:                    # room used up: the users start over at their context length
            for j in s["slots"]:
                m.position_slot(j, case["ctx"])
        m.decode_batch(s["slots"], s["tokens"])
        return {"logits": m.last_logits, "log": [m.log_u[i][:, 0] for i in sorted(m.log_u)]}
    if case["path"] == "prompt":
        m.reset()
        hidden = []                                      # what a drafter or an embedding user takes from a prompt
        m.prefill(s["prompt"], hook=lambda start, count, h: hidden.append(h.clone()))
        return {"logits": m.buf.logits[m.last_row], "hidden": hidden, "state": _state(m)}
    # one more answer from a prompt that is kept: back to its checkpoint, then token by token (or window by window)
    m.restore_checkpoint(s["checkpoint"])
    logits = []
    if case["path"] == "decode":
        s["session"].begin(s["fed"][0][0])
        for (token,) in s["fed"]:
            s["session"].step(token)
            logits.append(m.buf.logits[0].clone())       # what a sampler or a scorer reads
    else:
        for anchor, *drafts in s["fed"]:
            m.verify_window(anchor, drafts)
            logits.append(m.logits_rows(case["rows"]).clone())
    return {"logits": logits, "state": _state(m)}


def work(case):
    """Each weight, cache row and recurrent state that a pass needs, read (and where updated, written) once per model call."""
    cfg, kb = _config(case), _kb_rule(case)
    path, ctx, rows, steps = case["path"], case["ctx"], case["rows"], case["steps"]
    H, V, E, k = cfg.hidden_size, cfg.vocab_size, cfg.num_experts, cfg.num_experts_per_tok
    nbytes = flops = 0.0
    if path == "experts":
        for i in range(case["layers"]):
            p = f"text.layers.{i}.moe."
            expert, shared = 3.0 * H * cfg.moe_intermediate_size, 3.0 * H * cfg.shared_expert_intermediate_size
            touched = E * (1 - (1 - k / E) ** rows)
            nbytes += touched * expert * kb(p + "experts.0.gate_up") / 8 + shared * kb(p + "shared.down") / 8
            nbytes += 2.0 * H * (E + 1) + 4.0 * rows * H
            flops += 2.0 * rows * (k * expert + shared + H * (E + 1))
        return {"bytes": nbytes, "flops": flops}
    n = ctx if path == "prompt" else rows                # rows of one call
    for name, N, K in linear_shapes(cfg):
        nbytes += N * K * kb(name) / 8
        flops += 2.0 * N * K * n
    head_rows = 1 if path == "prompt" else n
    nbytes += V * H * (0.5 + 4 / 64) + head_rows * V * 4
    flops += 2.0 * V * H * head_rows
    attn = sum(cfg.is_attention_layer(i) for i in range(cfg.num_hidden_layers))
    gdn = cfg.num_hidden_layers - attn
    sequences = rows if path == "batch" else 1
    old = 0 if path == "prompt" else ctx * 2 * cfg.kv_dim * sequences
    pairs = n * (n + 1) / 2 if path == "prompt" else n * ctx
    state = 4.0 * cfg.linear_num_value_heads * cfg.linear_key_head_dim ** 2 * sequences
    nbytes += attn * (n * 2 * cfg.kv_dim + old) + gdn * 2 * state + n * (4 * H if path == "prompt" else 2 * H)
    flops += attn * 4.0 * cfg.num_attention_heads * cfg.head_dim * pairs + gdn * 6.0 * n * state / (4 * sequences)
    return {"bytes": nbytes * steps, "flops": flops * steps}


def tolerance(case):
    # bf16 activations between about ten kernels per layer: two of the engine's own kernels for the same products (sums in
    # another order) differ by 1.2 % at four layers and 1.9 % at eight, an expert block by 0.5 %
    return {"rel": 0.02} if case["path"] == "experts" else {"rel": 0.03}
