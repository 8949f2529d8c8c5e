"""The work whose speed is watched: calls a user of this package makes, from the smallest decode
iteration to the largest batches, through the package's public entry points.

A case is a dict of plain values; ``op`` says which entry point it goes through:

* ``iteration``  the attention function of an engine iteration: metadata of the jobs, plan, and one
  ``forward`` per layer (``B200SharedPromptsGenerate``).
* ``layer``      one layer of an iteration that is already planned, KV fill of the new tokens
  included (``AttentionCall.run``): decode, prefill, or both in one batch.
* ``paged``      decode without sharing in one shot (``vllm_paged_attention``).
* ``shared``     KV fill, then decode over a shared prefix in one shot (``vllm_reshape_and_cache``,
  ``flash_paged_attention``).
* ``host``       a decode layer whose inputs and result live in page-locked host memory (``HostStep``).
* ``rotary``     NeoX rotary embedding with the KV fill (``rotary_reshape_and_cache``).
* ``move``       contexts out of the paged caches into plain rows (``move_tokens_from_blocked_*``).
* ``sample``     one token per row of a logits matrix (``sample_top_p``).

Lengths follow from the case alone (``lens`` seeds them), so that a case is always the same amount
of work; contents and the placement of the blocks in the cache follow from the seed of ``prepare``.
"""
import types

import numpy as np
import torch

import parrotserve_b200 as pb
from parrotserve_b200.attn_func import B200SharedPromptsGenerate

BLOCK = 16
DTYPES = {"f16": torch.float16, "bf16": torch.bfloat16, "f32": torch.float32}
DEV = "cuda"


# ---------------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------------
def listed():
    return [
        # A few chat requests over a system prompt, all 32 layers of a 7B model: the smallest iteration,
        # where the host path and launch latencies count.
        dict(name="iteration_4seq_32layers", op="iteration", dtype="f16", layers=32, heads=32, prefix=512, seqs=4,
             suffix_lo=1, suffix_hi=64, fills=0, fill_hi=0, lens=1),
        # The headline decode step (bench.py): 64 sequences of a 7B model over one 4096-token prefix.
        dict(name="decode_7b_64seq", op="layer", dtype="f16", heads=32, groups=1, prefix_lo=4096, prefix_hi=4096, seqs=64,
             skew=0.0, suffix_lo=32, suffix_hi=512, prefills=0, new_lo=0, new_hi=0, lens=2),
        # 13B decode, ragged: 256 sequences spread unevenly over 8 applications with prompts of 1k to 8k.
        dict(name="decode_13b_8groups", op="layer", dtype="f16", heads=40, groups=8, prefix_lo=1024, prefix_hi=8192, seqs=256,
             skew=1.2, suffix_lo=1, suffix_hi=2048, prefills=0, new_lo=0, new_hi=0, lens=3),
        # Continuous batching: 16 prefills and 240 decodes in one batch over a 2048-token prompt.
        dict(name="mixed_16prefill_240decode", op="layer", dtype="f16", heads=32, groups=1, prefix_lo=2048, prefix_hi=2048,
             seqs=240, skew=0.0, suffix_lo=1, suffix_hi=1024, prefills=16, new_lo=256, new_hi=1024, lens=4),
        # One GPU's share (8 of 64 heads) of a box that decodes 2048 sequences over 32 prompts of 16k.
        dict(name="decode_shard_32groups", op="layer", dtype="bf16", heads=8, groups=32, prefix_lo=16384, prefix_hi=16384,
             seqs=2048, skew=0.0, suffix_lo=1, suffix_hi=1024, prefills=0, new_lo=0, new_hi=0, lens=5),
        # Prompts that share nothing: four long prefills.
        dict(name="prefill_4_prompts", op="layer", dtype="bf16", heads=32, groups=0, prefix_lo=0, prefix_hi=0, seqs=0, skew=0.0,
             suffix_lo=0, suffix_hi=0, prefills=4, new_lo=1500, new_hi=3000, lens=6),
        # Plain paged decode with grouped KV heads.
        dict(name="paged_gqa_128seq", op="paged", dtype="f16", heads=32, kv_heads=8, head_size=128, seqs=128, ctx_lo=16, ctx_hi=2048,
             lens=7),
        # The fp32 configuration: 4 sequences over a 512-token prefix.
        dict(name="shared_fp32_4seq", op="shared", dtype="f32", heads=32, prefix=512, seqs=4, suffix_lo=1, suffix_hi=64, lens=8),
        # The headline decode step with its inputs and its result in host memory.
        dict(name="host_7b_64seq", op="host", dtype="f16", heads=32, prefix=4096, seqs=64, suffix_lo=32, suffix_hi=512, lens=9),
        # Rotary embedding and KV fill of a continuous-batching iteration (prefills and decodes).
        dict(name="rotary_fill_10k", op="rotary", dtype="f16", heads=32, prefills=16, new_lo=256, new_hi=1024, seqs=240, lens=10),
        # Cached contexts pulled out of the paged cache into plain rows.
        dict(name="move_8k_tokens", op="move", dtype="f16", heads=32, head_size=128, contexts=16, ctx_lo=128, ctx_hi=1024, lens=11),
        # Sampling after the logits GEMM of a 64-sequence decode step.
        dict(name="sample_64rows", op="sample", dtype="f16", rows=64, vocab=32000, greedy=0.25, lens=12),
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    while True:
        case = _draw(rng)
        w = work(case)
        if w["bytes"] <= 5.5e9 and w["flops"] <= 3.5e11:
            return case


def _draw(rng):
    lens = rng.randrange(1 << 20)
    half = rng.choice(["f16", "bf16"])
    op = rng.choice(["iteration", "decode", "decode", "groups", "mixed", "prefill", "paged", "paged", "shared", "host", "rotary",
                     "move", "sample"])
    if op == "iteration":
        fills = rng.choice([0, 0, 1, 2])
        return dict(op="iteration", dtype=half, layers=rng.choice([12, 24, 32, 40]), heads=rng.choice([12, 32, 40]),
                    prefix=_log_int(rng, 16, 2048), seqs=_log_int(rng, 1, 32), suffix_lo=1, suffix_hi=_log_int(rng, 16, 512),
                    fills=fills, fill_hi=_log_int(rng, 16, 256) if fills else 0, lens=lens)
    if op == "decode":
        prefix = _log_int(rng, 64, 8192)
        return dict(op="layer", dtype=half, heads=rng.choice([4, 8, 16, 32, 40]), groups=1, prefix_lo=prefix, prefix_hi=prefix,
                    seqs=_log_int(rng, 2, 512), skew=0.0, suffix_lo=1, suffix_hi=_log_int(rng, 32, 2048), prefills=0, new_lo=0,
                    new_hi=0, lens=lens)
    if op == "groups":
        prefix = _log_int(rng, 256, 16384)
        return dict(op="layer", dtype=half, heads=rng.choice([8, 16, 32, 40]), groups=_log_int(rng, 2, 32),
                    prefix_lo=max(16, prefix // rng.choice([1, 4, 8])), prefix_hi=prefix, seqs=_log_int(rng, 32, 2048),
                    skew=rng.choice([0.0, 1.2]), suffix_lo=1, suffix_hi=_log_int(rng, 64, 2048), prefills=0, new_lo=0, new_hi=0,
                    lens=lens)
    if op == "mixed":
        prefix = _log_int(rng, 64, 4096)
        new = _log_int(rng, 64, 1024)
        return dict(op="layer", dtype=half, heads=rng.choice([8, 16, 32, 40]), groups=1, prefix_lo=prefix, prefix_hi=prefix,
                    seqs=_log_int(rng, 4, 240), skew=0.0, suffix_lo=1, suffix_hi=_log_int(rng, 64, 1024),
                    prefills=_log_int(rng, 1, 16), new_lo=max(1, new // 4), new_hi=new, lens=lens)
    if op == "prefill":
        new = _log_int(rng, 64, 4096)
        return dict(op="layer", dtype=half, heads=rng.choice([8, 16, 32, 40]), groups=0, prefix_lo=0, prefix_hi=0, seqs=0, skew=0.0,
                    suffix_lo=0, suffix_hi=0, prefills=_log_int(rng, 1, 16), new_lo=max(1, new // 4), new_hi=new, lens=lens)
    if op == "paged":
        heads, kv = rng.choice([(32, 32), (32, 8), (40, 40), (64, 8), (12, 12)])
        return dict(op="paged", dtype=half, heads=heads, kv_heads=kv, head_size=rng.choice([64, 80, 128, 128]),
                    seqs=_log_int(rng, 1, 256), ctx_lo=1, ctx_hi=_log_int(rng, 64, 4096), lens=lens)
    if op == "shared":
        return dict(op="shared", dtype=rng.choice(["f32", half]), heads=rng.choice([12, 32, 40]), prefix=_log_int(rng, 16, 2048),
                    seqs=_log_int(rng, 1, 32), suffix_lo=1, suffix_hi=_log_int(rng, 16, 256), lens=lens)
    if op == "host":
        return dict(op="host", dtype=half, heads=rng.choice([8, 32, 40]), prefix=_log_int(rng, 256, 8192),
                    seqs=_log_int(rng, 4, 128), suffix_lo=1, suffix_hi=_log_int(rng, 32, 512), lens=lens)
    if op == "rotary":
        new = _log_int(rng, 16, 1024)
        return dict(op="rotary", dtype=half, heads=rng.choice([8, 32, 40]), prefills=rng.choice([0, 1, 2, 5, 16]),
                    new_lo=max(1, new // 4), new_hi=new, seqs=_log_int(rng, 1, 256), lens=lens)
    if op == "move":
        ctx = _log_int(rng, 16, 2048)
        return dict(op="move", dtype=rng.choice(["f32", half]), heads=rng.choice([12, 32, 40]), head_size=rng.choice([64, 128]),
                    contexts=_log_int(rng, 1, 16), ctx_lo=max(1, ctx // 4), ctx_hi=ctx, lens=lens)
    return dict(op="sample", dtype=rng.choice(["f32", half]), rows=_log_int(rng, 1, 256),
                vocab=rng.choice([32000, 50272, 32001, 128256]), greedy=rng.choice([0.0, 0.25, 1.0]), lens=lens)


# ---------------------------------------------------------------------------------------------
# lengths of a case
# ---------------------------------------------------------------------------------------------
def _up(n):
    return -(-n // BLOCK)


def _uniform(rng, lo, hi, n):
    return rng.integers(lo, hi + 1, size=n).tolist()


def _layer_lens(c):
    """(prefix length per group, group of each decode row, private length of each decode row, new tokens per prefill)"""
    rng = np.random.default_rng(c["lens"])
    g = c["groups"]
    # a shared context is padded to whole blocks when it is forked
    prefix = [_up(int(p)) * BLOCK for p in np.linspace(c["prefix_lo"], c["prefix_hi"], g)] if g else []
    if g:
        w = np.arange(1, g + 1, dtype=np.float64) ** -c["skew"]
        group = np.sort(rng.choice(g, size=c["seqs"], p=w / w.sum())) if c["skew"] else np.arange(c["seqs"]) * g // max(1, c["seqs"])
        group = group.tolist()
    else:
        group = [-1] * c["seqs"]
    suffix = _uniform(rng, c["suffix_lo"], c["suffix_hi"], c["seqs"])
    new = _uniform(rng, c["new_lo"], c["new_hi"], c["prefills"])
    return prefix, group, suffix, new


def _lens(c):
    rng = np.random.default_rng(c["lens"])
    if c["op"] in ("iteration", "shared", "host"):
        suffix = _uniform(rng, c["suffix_lo"], c["suffix_hi"], c["seqs"])
        fills = _uniform(rng, max(1, c["fill_hi"] // 4), c["fill_hi"], c["fills"]) if c.get("fills") else []
        return _up(c["prefix"]) * BLOCK, suffix, fills
    if c["op"] == "paged":
        return _uniform(rng, c["ctx_lo"], c["ctx_hi"], c["seqs"])
    if c["op"] == "rotary":  # cached tokens before the new ones, and new tokens, of every request
        new = _uniform(rng, c["new_lo"], c["new_hi"], c["prefills"]) + [1] * c["seqs"]
        cached = [0] * c["prefills"] + _uniform(rng, 0, 1023, c["seqs"])
        return cached, new
    return _uniform(rng, c["ctx_lo"], c["ctx_hi"], c["contexts"])  # move


# ---------------------------------------------------------------------------------------------
# bytes and operations of one pass
# ---------------------------------------------------------------------------------------------
def work(case):
    c = case
    esz = 4 if c["dtype"] == "f32" else 2
    op = c["op"]
    if op == "sample":
        return {"bytes": c["rows"] * c["vocab"] * esz + c["rows"] * 8, "flops": 4.0 * c["rows"] * c["vocab"]}
    row = c["heads"] * c.get("head_size", 128) * esz          # a query, output, key or value row
    if op == "move":
        return {"bytes": 4 * sum(_lens(c)) * row, "flops": 0}  # K and V, read and written
    if op == "rotary":
        t = sum(_lens(c)[1])
        return {"bytes": 6 * t * row, "flops": 6.0 * t * row / esz}  # q in place, k and v into the cache
    if op == "paged":
        lens = _lens(c)
        kv = 2 * c["kv_heads"] * c["head_size"] * esz
        return {"bytes": sum(lens) * kv + 2 * len(lens) * row, "flops": 4.0 * sum(lens) * c["heads"] * c["head_size"]}
    if op == "layer":
        prefix, group, suffix, new = _layer_lens(c)
        used = sorted(set(group)) if not new else range(len(prefix))
        keys = sum(prefix[g] for g in used if g >= 0) + sum(suffix) + sum(new)
        shared = prefix[0] if (new and prefix) else 0
        pairs = sum(suffix) + sum(prefix[g] for g in group if g >= 0) + sum(n * shared + n * (n + 1) // 2 for n in new)
        rows, fresh, layers = len(suffix) + sum(new), len(suffix) + sum(new), 1
    else:
        plen, suffix, fills = _lens(c)
        keys = plen + sum(suffix) + sum(fills)
        pairs = sum(suffix) + plen * len(suffix) + sum(n * plen + n * (n + 1) // 2 for n in fills)
        rows = fresh = len(suffix) + sum(fills)
        layers = c.get("layers", 1)
    # every key and value once, queries and outputs, and the fill: the new tokens' keys and values read and written
    return {"bytes": layers * (2 * keys * row + 2 * rows * row + 4 * fresh * row), "flops": layers * 4.0 * pairs * c["heads"] * 128}


def tolerance(case):
    """Four times the largest error seen against the same sums in 64 bits; moved bytes and token ids are exact."""
    if case["op"] in ("move", "sample"):
        return "exact"
    if case["op"] == "rotary":
        return {"rel": 8e-4 if case["dtype"] == "f16" else 6.4e-3}  # one rounding: 2.0e-4, 1.6e-3
    # attention: 2.0e-7, 2.9e-4 and 2.3e-3
    return {"rel": {"f32": 2e-6, "f16": 1.2e-3, "bf16": 1e-2}[case["dtype"]]}


# ---------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------
def _normal(shape, dtype, gen):
    return torch.empty(shape, dtype=dtype, device=DEV).normal_(generator=gen)


def _caches(blocks, heads, head_size, dtype, gen, layers=0):
    x = 16 // torch.empty((), dtype=dtype).element_size()
    lead = (layers, blocks) if layers else (blocks,)
    return (_normal((*lead, heads, head_size // x, BLOCK, x), dtype, gen), _normal((*lead, heads, head_size, BLOCK), dtype, gen))


def _deal(perm, lens):
    """Block ids for contexts of the given lengths, from a permutation of the cache's blocks."""
    out, at = [], 0
    for n in lens:
        out.append(perm[at:at + _up(n)])
        at += _up(n)
    return out


def _table(rows):
    width = max([len(r) for r in rows] + [0])
    t = np.zeros((len(rows), width), dtype=np.int32)
    for i, r in enumerate(rows):
        t[i, :len(r)] = r
    return torch.from_numpy(t).to(DEV)


def _i32(v):
    return torch.tensor(v, dtype=torch.int32, device=DEV)


def _slots(blocks, first, n):
    return [int(blocks[t // BLOCK]) * BLOCK + t % BLOCK for t in range(first, first + n)]


def _pool(lens, seed):
    """Number of blocks of the cache (a tenth of it free) and the order in which they are handed out."""
    blocks = int(sum(_up(n) for n in lens) * 1.1) + 8
    return blocks, np.random.default_rng(seed).permutation(blocks)


def prepare(case, seed):
    c = dict(case)
    gen = torch.Generator(device=DEV).manual_seed(seed)
    return types.SimpleNamespace(op=c["op"], case=c, **PREPARE[c["op"]](c, seed, DTYPES[c["dtype"]], gen))


def _qkv(rows, heads, head_size, dtype, gen):
    """Query, key and value rows as the model makes them: views of one fused projection."""
    fused = _normal((rows, 3 * heads * head_size), dtype, gen)
    return tuple(x.view(rows, heads, head_size) for x in fused.chunk(3, dim=-1))


def _prepare_layer(c, seed, dtype, gen):
    prefix, group, suffix, new = _layer_lens(c)
    blocks, perm = _pool(prefix + new + suffix, seed)
    tabs = _deal(perm, prefix + new + suffix)
    ptab, ntab, stab = tabs[:len(prefix)], tabs[len(prefix):len(prefix) + len(new)], tabs[len(prefix) + len(new):]
    n_new = sum(new)
    rows = n_new + len(suffix)
    kc, vc = _caches(blocks, c["heads"], 128, dtype, gen)
    q, k, v = _qkv(rows, c["heads"], 128, dtype, gen)
    slots = [s for n, t in zip(new, ntab) for s in _slots(t, 0, n)] + [s for n, t in zip(suffix, stab) for s in _slots(t, n - 1, 1)]
    meta = dict(suffix_lens=_i32([0] * n_new + suffix), suffix_tables=_table([[]] * n_new + stab))
    if prefix:
        counts = [0] * len(prefix)
        for g in group:
            counts[g] += 1
        counts[0] += n_new  # prefills come first, and only with a single group
        meta.update(group_row_offsets=_i32(np.cumsum([0] + counts).tolist()), group_prefix_lens=_i32(prefix), group_tables=_table(ptab))
    if new:
        meta.update(seg_row_offsets=_i32(np.cumsum([0] + new).tolist()), seg_kv_lens=_i32(new), seg_tables=_table(ntab))
    call = pb.AttentionCall(num_rows=rows, num_heads=c["heads"], head_size=128, block_size=BLOCK, dtype=dtype, device=q.device,
                            slot_mapping=torch.tensor(slots, dtype=torch.int64, device=DEV), **meta)
    out = torch.empty((rows, c["heads"], 128), dtype=dtype, device=DEV)
    call.plan(q, out, kc, vc)
    return dict(call=call, q=q, k=k, v=v, out=out, kc=kc, vc=vc, ptab=ptab, ntab=ntab, stab=stab, slots=slots)


class _Context:
    """A context of the engine's tree: its own tokens' blocks and slots, and its parent."""

    def __init__(self, parent, blocks, n):
        self.parent_context, self.depth = parent, 0 if parent is None else parent.depth + 1
        self.token_kv_block_ids = [int(blocks[t // BLOCK]) for t in range(n)]
        self.token_kv_slot_ids = _slots(blocks, 0, n)

    def get_context_len(self):
        return len(self.token_kv_slot_ids) + (self.parent_context.get_context_len() if self.parent_context else 0)

    def get_context_block_ids(self):
        return (self.parent_context.get_context_block_ids() if self.parent_context else []) + self.token_kv_block_ids

    def get_context_slot_ids(self):
        return (self.parent_context.get_context_slot_ids() if self.parent_context else []) + self.token_kv_slot_ids


def _prepare_iteration(c, seed, dtype, gen):
    plen, suffix, fills = _lens(c)
    blocks, perm = _pool([plen] + fills + suffix, seed)
    tabs = _deal(perm, [plen] + fills + suffix)
    root = _Context(None, tabs[0], plen)
    jobs = [types.SimpleNamespace(context=_Context(root, t, n), token_ids=list(range(n))) for n, t in zip(fills, tabs[1:])]
    jobs += [types.SimpleNamespace(context=_Context(root, t, n), sampling_config=None) for n, t in zip(suffix, tabs[1 + len(fills):])]
    kc, vc = _caches(blocks, c["heads"], 128, dtype, gen, layers=c["layers"])
    q, k, v = _qkv(sum(fills) + len(suffix), c["heads"], 128, dtype, gen)
    model = [B200SharedPromptsGenerate(i, 128 ** -0.5, c["heads"], 128) for i in range(c["layers"])]
    config = types.SimpleNamespace(block_size=BLOCK, device="cuda:0", dtype=dtype)
    slots = [x for n, t in zip(fills, tabs[1:]) for x in _slots(t, 0, n)]
    slots += [_slots(t, n - 1, 1)[0] for n, t in zip(suffix, tabs[1 + len(fills):])]
    return dict(jobs=jobs, kc=kc, vc=vc, caches=list(zip(kc, vc)), q=q, k=k, v=v, model=model, config=config, ptab=tabs[:1],
                ntab=tabs[1:1 + len(fills)], stab=tabs[1 + len(fills):], slots=slots)


def _prepare_paged(c, seed, dtype, gen):
    lens = _lens(c)
    blocks, perm = _pool(lens, seed)
    kc, vc = _caches(blocks, c["kv_heads"], c["head_size"], dtype, gen)
    share = c["heads"] // c["kv_heads"]
    mapping = None if share == 1 else _i32([h // share for h in range(c["heads"])])
    q = _normal((len(lens), c["heads"], c["head_size"]), dtype, gen)
    return dict(q=q, kc=kc, vc=vc, mapping=mapping, ctx=_i32(lens), tables=_table(_deal(perm, lens)))


def _prepare_shared(c, seed, dtype, gen):
    plen, suffix, _ = _lens(c)
    blocks, perm = _pool([plen] + suffix, seed)
    tabs = _deal(perm, [plen] + suffix)
    kc, vc = _caches(blocks, c["heads"], 128, dtype, gen)
    q, k, v = _qkv(len(suffix), c["heads"], 128, dtype, gen)
    slots = torch.tensor([_slots(t, n - 1, 1)[0] for n, t in zip(suffix, tabs[1:])], dtype=torch.int64, device=DEV)
    return dict(q=q, k=k, v=v, kc=kc, vc=vc, slots=slots, plen=plen, ptab=_i32([int(b) for b in tabs[0]]), ctx=_i32(suffix),
                tables=_table(tabs[1:]), stab=tabs[1:])


def _prepare_host(c, seed, dtype, gen):
    plen, suffix, _ = _lens(c)
    blocks, perm = _pool([plen] + suffix, seed)
    tabs = _deal(perm, [plen] + suffix)
    kc, vc = _caches(blocks, c["heads"], 128, dtype, gen)
    n, tables = len(suffix), _table(tabs[1:])
    step = pb.HostStep(num_rows=n, num_heads=c["heads"], head_size=128, block_size=BLOCK, dtype=dtype, device=kc.device,
                       max_suffix_blocks=tables.shape[1], num_new_tokens=n, group_row_offsets=_i32([0, n]),
                       group_prefix_lens=_i32([plen]), group_tables=_table(tabs[:1]))
    for view in (step.h_query, step.h_key_new, step.h_value_new):
        view.copy_(_normal(view.shape, dtype, gen))
    step.h_slots.copy_(torch.tensor([_slots(t, m - 1, 1)[0] for m, t in zip(suffix, tabs[1:])], dtype=torch.int64))
    step.h_suffix_tables.copy_(tables)
    step.h_suffix_lens.copy_(torch.tensor(suffix, dtype=torch.int32))
    return dict(step=step, kc=kc, vc=vc, ptab=tabs[:1], stab=tabs[1:])


def _prepare_rotary(c, seed, dtype, gen):
    cached, new = _lens(c)
    total = [a + b for a, b in zip(cached, new)]
    blocks, perm = _pool(total, seed)
    tabs = _deal(perm, total)
    kc, vc = _caches(blocks, c["heads"], 128, dtype, gen)
    q, k, v = _qkv(sum(new), c["heads"], 128, dtype, gen)
    slots = [s for a, b, t in zip(cached, new, tabs) for s in _slots(t, a, b)]
    positions = [a + i for a, b in zip(cached, new) for i in range(b)]
    angle = torch.outer(torch.arange(4096, device=DEV, dtype=torch.float32),
                        1.0 / (10000.0 ** (torch.arange(0, 128, 2, device=DEV, dtype=torch.float32) / 128)))
    return dict(q=q, k=k, v=v, kc=kc, vc=vc, slots=torch.tensor(slots, dtype=torch.int64, device=DEV),
                positions=torch.tensor(positions, dtype=torch.int64, device=DEV),
                cos_sin=torch.cat([angle.cos(), angle.sin()], dim=1).to(dtype))


def _prepare_move(c, seed, dtype, gen):
    lens = _lens(c)
    blocks, perm = _pool(lens, seed)
    kc, vc = _caches(blocks, c["heads"], c["head_size"], dtype, gen)
    slots = [s for n, t in zip(lens, _deal(perm, lens)) for s in _slots(t, 0, n)]
    total = len(slots)
    rows = [torch.empty((total, c["heads"], c["head_size"]), dtype=dtype, device=DEV) for _ in range(2)]
    return dict(kc=kc, vc=vc, src=torch.tensor(slots, dtype=torch.int64, device=DEV), dst=torch.arange(total, device=DEV),
                k_rows=rows[0], v_rows=rows[1])


def _prepare_sample(c, seed, dtype, gen):
    # logits of a language model: most of the vocabulary far below a few dozen likely tokens
    logits = torch.empty((c["rows"], c["vocab"]), device=DEV).normal_(0.0, 2.0, generator=gen)
    likely = torch.randint(c["vocab"], (c["rows"], 40), device=DEV, generator=gen)
    logits.scatter_add_(1, likely, torch.empty((c["rows"], 40), device=DEV).uniform_(2.0, 10.0, generator=gen))
    rng = np.random.default_rng(seed)
    plain = rng.random(c["rows"]) < c["greedy"]  # requests that leave both settings at 1.0
    temperature = np.where(plain, 1.0, rng.uniform(0.5, 1.2, c["rows"])).tolist()
    top_p = np.where(plain, 1.0, rng.uniform(0.7, 0.98, c["rows"])).tolist()
    return dict(logits=logits.to(dtype), temperature=temperature, top_p=top_p,
                uniforms=torch.rand(c["rows"], device=DEV, generator=gen))


PREPARE = dict(layer=_prepare_layer, iteration=_prepare_iteration, paged=_prepare_paged, shared=_prepare_shared, host=_prepare_host,
               rotary=_prepare_rotary, move=_prepare_move, sample=_prepare_sample)


# ---------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------
def run(state):
    s = state
    if s.op == "layer":
        s.call.run(s.q, s.out, s.kc, s.vc, key_new=s.k, value_new=s.v)
        return s.out, s.kc, s.vc
    if s.op == "iteration":
        B200SharedPromptsGenerate.kv_cache_getter = staticmethod(s.caches.__getitem__)
        it = types.SimpleNamespace(num_fill_tokens=[], generation_sampling_config=[])
        B200SharedPromptsGenerate.init_iteration_state(it, s.config, s.jobs, s.case["heads"], 128)
        return [layer(s.q, s.k, s.v, it) for layer in s.model], s.kc, s.vc
    if s.op == "paged":
        return pb.vllm_paged_attention(s.q, s.kc, s.vc, s.mapping, s.ctx, s.tables)
    if s.op == "shared":
        pb.vllm_reshape_and_cache(s.k, s.v, s.kc, s.vc, s.slots)
        out = pb.flash_paged_attention(s.q, s.kc, s.vc, None, s.plen, s.ptab, s.ctx, s.tables)
        return out, s.kc, s.vc
    if s.op == "host":
        return s.step.step_graph(s.kc, s.vc), s.kc, s.vc
    if s.op == "rotary":
        pb.rotary_reshape_and_cache(s.positions, s.q, s.k, s.v, s.kc, s.vc, s.slots, s.cos_sin, 128)
        return s.q, s.kc, s.vc
    if s.op == "move":
        pb.move_tokens_from_blocked_k_cache(s.kc, s.k_rows, s.src, s.dst)
        pb.move_tokens_from_blocked_v_cache(s.vc, s.v_rows, s.src, s.dst)
        return s.k_rows, s.v_rows
    return pb.sample_top_p(s.logits, s.temperature, s.top_p, uniforms=s.uniforms)


# ---------------------------------------------------------------------------------------------
# the same in 64 bits, by plain torch
# ---------------------------------------------------------------------------------------------
def _rows_of(kc, vc, blocks, n):
    """Keys and values of a context's first n tokens, [n, heads, head_size] in 64 bits."""
    ids = torch.as_tensor([int(b) for b in blocks[:_up(n)]], dtype=torch.int64, device=DEV)
    k, v = kc[ids], vc[ids]
    k = k.permute(0, 3, 1, 2, 4).reshape(len(ids) * BLOCK, kc.shape[1], -1)
    v = v.permute(0, 3, 1, 2).reshape(len(ids) * BLOCK, vc.shape[1], -1)
    return k[:n].double(), v[:n].double()


def _fill(kc, vc, k, v, slots):
    s = torch.as_tensor(slots, dtype=torch.int64, device=DEV)
    rows = k.shape[0]
    kc[s // BLOCK, :, :, s % BLOCK, :] = k.reshape(rows, kc.shape[1], kc.shape[2], kc.shape[4]).to(kc.dtype)
    vc[s // BLOCK, :, :, s % BLOCK] = v.reshape(rows, vc.shape[1], vc.shape[2]).to(vc.dtype)


def _attend(q, parts, out):
    """Rows q [n, heads, d] over the keys and values of all parts; a part is (k, v, tokens each row sees or None)."""
    scale = q.shape[2] ** -0.5
    for lo in range(0, q.shape[1], 8):
        h = slice(lo, lo + 8)
        scores = []
        for k, _, seen in parts:
            x = torch.einsum("nhd,thd->hnt", q[:, h].double(), k[:, h]) * scale
            if seen is not None:
                x.masked_fill_(torch.arange(k.shape[0], device=DEV)[None, None, :] >= seen[None, :, None], float("-inf"))
            scores.append(x)
        p = torch.softmax(torch.cat(scores, dim=2), dim=2)
        out[:, h] = torch.einsum("hnt,thd->nhd", p, torch.cat([v[:, h] for _, v, _ in parts]))


def _exact_rows(q, kc, vc, prefix, ptab, group, suffix, stab, new, ntab):
    """A batch: the prefills' rows first (under the first prefix, where there is one), then one row per sequence."""
    out = torch.zeros(q.shape, dtype=torch.float64, device=DEV)
    shared = [_rows_of(kc, vc, t, n) for t, n in zip(ptab, prefix)]
    at = 0
    for n, t in zip(new, ntab):
        own = (*_rows_of(kc, vc, t, n), torch.arange(1, n + 1, device=DEV))
        _attend(q[at:at + n], ([(*shared[0], None)] if shared else []) + [own], out[at:at + n])
        at += n
    for g, n, t in zip(group, suffix, stab):
        _attend(q[at:at + 1], ([(*shared[g], None)] if g >= 0 else []) + [(*_rows_of(kc, vc, t, n), None)], out[at:at + 1])
        at += 1
    return out


def exact(case, seed):
    """What ``run`` returns, in 64 bits; None for moved bytes (the caches of an attention call) and token ids."""
    c = case
    if c["op"] in ("move", "sample"):
        return None
    s = prepare(case, seed)
    if c["op"] == "rotary":
        half = s.cos_sin.shape[1] // 2
        cos, sin = (x[:, None, :].double() for x in s.cos_sin[s.positions].split(half, dim=1))

        def turn(x):
            a, b = x[..., :half].double(), x[..., half:].double()
            return torch.cat([a * cos - b * sin, b * cos + a * sin], dim=-1)

        kc = s.kc.double()
        _fill(kc, s.vc, turn(s.k), s.v, s.slots)
        return turn(s.q), kc, s.vc
    if c["op"] == "paged":
        share = c["heads"] // c["kv_heads"]
        out = torch.zeros(s.q.shape, dtype=torch.float64, device=DEV)
        for i, (n, t) in enumerate(zip(_lens(c), s.tables.tolist())):
            k, v = (x.repeat_interleave(share, dim=1) for x in _rows_of(s.kc, s.vc, t, n))
            _attend(s.q[i:i + 1], [(k, v, None)], out[i:i + 1])
        return out
    if c["op"] == "layer":
        prefix, group, suffix, new = _layer_lens(c)
        _fill(s.kc, s.vc, s.k, s.v, s.slots)
        return _exact_rows(s.q, s.kc, s.vc, prefix, s.ptab, group, suffix, s.stab, new, s.ntab), None, None
    plen, suffix, fills = _lens(c)
    group = [0] * len(suffix)
    if c["op"] == "iteration":
        outs = []
        for kc, vc in s.caches:
            _fill(kc, vc, s.k, s.v, s.slots)
            outs.append(_exact_rows(s.q, kc, vc, [plen], s.ptab, group, suffix, s.stab, fills, s.ntab).flatten(1))
        return outs, None, None
    if c["op"] == "shared":
        _fill(s.kc, s.vc, s.k, s.v, s.slots)
        return _exact_rows(s.q, s.kc, s.vc, [plen], [s.ptab.tolist()], group, suffix, s.stab, [], []), None, None
    h = s.step
    _fill(s.kc, s.vc, h.h_key_new.to(DEV), h.h_value_new.to(DEV), h.h_slots.to(DEV))
    return _exact_rows(h.h_query.to(DEV), s.kc, s.vc, [plen], s.ptab, group, suffix, s.stab, [], []), None, None
