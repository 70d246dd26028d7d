"""Workloads of the compressed-KV path as a program that serves with this package calls them.

Every case names a ``path`` (which public entry points one pass goes through) and its sizes.  The paths and
what they stand for in use:

  mg_encode    one frame's K or V written by the Matrix-Game cache (``mg_codec.encode_tensor``: online C-means,
               projection, INT4).  The smallest write there is; one per layer, tensor and frame.
  lb_encode    K and V of one LingBot chunk committed (``lingbot_codec.encode_pair``).
  append       a history written chunk by chunk against given centres (``codec.encode_append`` into a
               ``CompressedHistory`` that starts over), K and V: the prefill of a rollout.
  decode       the window of a rolling cache rebuilt to K and V rows (``lingbot_codec.decode_segments``):
               the form for callers that keep their own attention.
  read         ``attention.codec_attention`` over one layer's history, with or without the rotation of the
               rebuilt keys by the tokens' positions.
  fast         ``attention.hybrid_attention``: protected frames at full width, the rest through low-width
               readers on most heads.
  lb_turn      one turn of a LingBot rollout (``lingbot_attention.codec_cache_attention``): the committing call
               of a chunk, then the first denoising call of the next one, over a sink + recent window.
  lb_fast      one denoising call of LingBot's mixed-width step (``lingbot_attention.attend``).
  roundtrip    history written and attended with fp32 operators and rows.

Rows are a uniformly drawn centre plus 0.3 N(0,1), operators N(0, 1/width), queries N(0,1), as everywhere in
this package's tests and benchmark.  A frame is 1,560 tokens (30 x 52) unless the case says otherwise.
"""
from __future__ import annotations

import math

import torch

from nanokv_b200 import lingbot_attention, lingbot_codec, mg_codec
from nanokv_b200.attention import Reader, RopeTable, codec_attention, hybrid_attention
from nanokv_b200.cache import CompressedHistory
from nanokv_b200.codec import GROUP32_FP16, Operator, QuantSpec, encode_append

FRAME, WIDTH = 1560, 52
HEAD_DIM = 128
NOISE = 0.3
# (heads, rank) of the configurations this package is built and tested for; heads of 128
SHAPES = ((12, 192), (16, 256), (16, 512), (24, 384), (40, 640))


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the smallest write: one 880-token frame of one tensor of one Matrix-Game layer
        dict(name="mg_encode_frame", path="mg_encode", heads=24, rank=384, tokens=880, clusters=64),
        # a three-frame LingBot chunk, K and V, as the rollout commits it
        dict(name="lb_encode_chunk", path="lb_encode", heads=40, rank=640, tokens=4680, clusters=64),
        # sixteen frames written one by one: many small calls, one scale per token
        dict(name="append_frames", path="append", heads=24, rank=384, tokens=24960, chunk=1560, clusters=256,
             group32=False),
        # eight frames in one call, 512 centres (16-bit ids), 32-wide groups with fp16 scales
        dict(name="append_group32", path="append", heads=40, rank=640, tokens=12480, chunk=12480, clusters=512,
             group32=True),
        # eighteen frames of the rolling window rebuilt for a caller with its own attention
        dict(name="decode_window", path="decode", heads=40, rank=640, tokens=28080, chunk=4680, clusters=64),
        # the smallest read: a short history and few queries, where launches and latency count
        dict(name="read_short", path="read", heads=12, rank=192, tokens=2048, queries=256, clusters=16, rope=False),
        # an ordinary read: sixteen frames, three frames of queries
        dict(name="read_16_frames", path="read", heads=24, rank=384, tokens=24960, queries=4680, clusters=256,
             rope=False),
        # the largest read: sixty-four frames of a 40-head layer
        dict(name="read_64_frames", path="read", heads=40, rank=640, tokens=99840, queries=4680, clusters=512,
             rope=False),
        # a ragged history with keys rotated inside the read, one frame of queries
        dict(name="read_rope_ragged", path="read", heads=40, rank=640, tokens=26917, queries=1560, clusters=256,
             rope=True),
        # mixed widths: 32 frames, the last two at full width, 18 of 24 heads read 32 wide
        dict(name="fast_32_frames", path="fast", heads=24, rank=384, tokens=49920, queries=4680, clusters=256,
             low_heads=18, low_width=32),
        # one rollout turn over an 18-frame window with a 6-frame sink
        dict(name="lb_turn", path="lb_turn", heads=40, rank=640, tokens=28080, chunk=4680, clusters=64),
        # fp32 operators: the exact-arithmetic configuration
        dict(name="roundtrip_f32", path="roundtrip", heads=12, rank=192, tokens=2048, queries=256, clusters=16),
    ]


def _log_uniform(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    path = rng.choice(("mg_encode", "lb_encode", "append", "decode", "read", "read", "fast", "lb_turn", "lb_fast",
                       "roundtrip"))
    heads, rank = rng.choice(SHAPES)
    case = dict(path=path, heads=heads, rank=rank)
    if path == "mg_encode":
        case.update(tokens=_log_uniform(rng, 256, 8000), clusters=64)
    elif path == "lb_encode":
        case.update(tokens=_log_uniform(rng, 500, 9360), clusters=rng.choice((64, 64, 128, 256)))
    elif path == "append":
        chunk = _log_uniform(rng, 400, 12480)
        case.update(tokens=chunk * rng.randint(1, max(1, 24960 // chunk)), chunk=chunk,
                    clusters=rng.choice((64, 256, 512)), group32=rng.random() < 0.5)
    elif path == "decode":
        chunk = _log_uniform(rng, 400, 4680)
        case.update(tokens=chunk * rng.randint(1, max(1, 28080 // chunk)), chunk=chunk, clusters=64)
    elif path == "read":
        case.update(tokens=_log_uniform(rng, 500, 60000), queries=_log_uniform(rng, 64, 4680),
                    clusters=rng.choice((16, 64, 256, 512)), rope=rng.random() < 0.4)
    elif path == "fast":
        case.update(tokens=FRAME * rng.randint(4, 32), queries=_log_uniform(rng, 256, 4680), clusters=256,
                    low_heads=heads * 3 // 4, low_width=rng.choice((32, 64)))
    elif path in ("lb_turn", "lb_fast"):
        chunk = FRAME * rng.randint(1, 3)
        case.update(tokens=chunk * rng.randint(4, 6), chunk=chunk, clusters=64)
    else:
        case.update(heads=12, rank=192, tokens=_log_uniform(rng, 300, 4096), queries=_log_uniform(rng, 32, 512),
                    clusters=16)
    return case


# ------------------------------------------------------------------ inputs
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _centers(case, gen):
    return torch.randn(case["clusters"], case["heads"] * HEAD_DIM, generator=gen, device="cuda")


def _rows(count, centers, gen, dtype=torch.bfloat16):
    pick = torch.randint(centers.shape[0], (count,), generator=gen, device="cuda")
    rows = torch.randn(count, centers.shape[1], generator=gen, device="cuda").mul_(NOISE)
    return rows.add_(centers.index_select(0, pick)).to(dtype)


def _weights(case, gen, dtype=torch.bfloat16):
    joint, rank = case["heads"] * HEAD_DIM, case["rank"]
    return dict(mean=0.1 * torch.randn(joint, generator=gen, device="cuda"),
                encoder=(torch.randn(rank, joint, generator=gen, device="cuda") / math.sqrt(joint)).to(dtype),
                decoder=(torch.randn(joint, rank, generator=gen, device="cuda") / math.sqrt(rank)).to(dtype))


def _queries(count, heads, gen, dtype=torch.bfloat16):
    return torch.randn(count, heads, HEAD_DIM, generator=gen, device="cuda").to(dtype)


def _history(case, tokens, centers, rows_dtype, op, gen, chunk=FRAME):
    """A shared-table history of one tensor, written frame by frame."""
    hist = CompressedHistory(joint=case["heads"] * HEAD_DIM, rank=case["rank"], capacity=tokens,
                             max_segments=-(-tokens // chunk), centers_per_segment=case["clusters"],
                             shared_centers=True)
    hist.centers.copy_(centers.to(torch.bfloat16))
    for start in range(0, tokens, 8 * chunk):
        rows = _rows(min(8 * chunk, tokens - start), centers, gen, rows_dtype)
        for first in range(0, rows.shape[0], chunk):
            encode_append(hist, rows[first:first + chunk], op, QuantSpec(), centers="resident")
    return hist


def _freqs(rows=1024):
    """complex128 [rows, 64]: temporal, vertical and horizontal bands side by side."""
    def band(dim):
        angles = torch.outer(torch.arange(rows),
                             1.0 / torch.pow(10000.0, torch.arange(0, dim, 2).to(torch.float64).div(dim)))
        return torch.polar(torch.ones_like(angles), angles)
    d = HEAD_DIM
    return torch.cat([band(d - 4 * (d // 6)), band(2 * (d // 6)), band(2 * (d // 6))], dim=1)


def _reader(case, gen, low_heads, low_width):
    """Reader payload: the first heads read ``low_width`` wide, the others at full width."""
    heads, rank = case["heads"], case["rank"]
    groups = []
    for ids, width in ((range(low_heads), low_width), (range(low_heads, heads), HEAD_DIM)):
        count = len(ids)
        indices = torch.arange(width).expand(count, width).contiguous()
        select = torch.zeros(count, HEAD_DIM, width).scatter_(1, indices[:, None, :], 1.0)
        read = [torch.randn(count, width, rank, generator=gen, device="cuda") / math.sqrt(rank) for _ in range(2)]
        groups.append(dict(heads=torch.tensor(list(ids)), indices=indices,
                           q_reduce=select * math.sqrt(HEAD_DIM / width), k_read=read[0], v_read=read[1],
                           k_affine=select.clone(), v_affine=select.clone(),
                           lift=select.transpose(1, 2).contiguous()))
    return dict(heads=heads, native_dim=HEAD_DIM, rank=rank, groups=groups)


def _lingbot_cache(case, layer, centers, gen):
    """Per-layer codec cache of a rollout that has committed ``tokens`` tokens in chunks."""
    heads = case["heads"]
    for target in "kv":
        lingbot_codec.register_operator(target, layer, **_weights(case, gen))
    cache = {}
    lingbot_attention.configure_cache(cache, layer=layer, sp_rank=0, options={
        "codec_rank": case["rank"], "codec_clusters": case["clusters"], "codec_iters": 2,
        "codec_basis_root_k": "registered", "codec_basis_root_v": "registered"})
    for start in range(0, case["tokens"], case["chunk"]):
        key, value = (_rows(case["chunk"], centers, gen).view(1, -1, heads, HEAD_DIM) for _ in range(2))
        cache["codec_commit_start"] = start
        cache["codec_segments"].append(lingbot_codec.encode_pair(key, value, cache=cache))
        cache["codec_committed_end"] = start + case["chunk"]
    return cache


def _window(case):
    """The rollout's policy: six sink frames, as much window as is committed."""
    return dict(capacity=case["tokens"], sink_tokens=min(6 * FRAME, case["tokens"] // 2),
                max_attention_size=case["tokens"])


def prepare(case, seed):
    gen = _generator(seed)
    path, heads = case["path"], case["heads"]
    layer = int(seed) % 1000003      # operators are registered per layer: a layer of this state's own
    state = dict(case=case, layer=layer)
    centers = _centers(case, gen)
    if path == "mg_encode":
        mg_codec.register_operator("k", layer, **_weights(case, gen))
        state["rows"] = _rows(case["tokens"], centers, gen)[None]
    elif path == "lb_encode":
        for target in "kv":
            lingbot_codec.register_operator(target, layer, **_weights(case, gen))
        state["key"], state["value"] = (_rows(case["tokens"], centers, gen).view(1, -1, heads, HEAD_DIM)
                                        for _ in range(2))
        state["cache"] = {"codec_layer": layer, "codec_rank": case["rank"], "codec_clusters": case["clusters"],
                          "codec_iters": 2, "codec_commit_start": 0, "codec_basis_root_k": "registered",
                          "codec_basis_root_v": "registered"}
    elif path == "append":
        quant = GROUP32_FP16 if case["group32"] else QuantSpec()
        state["quant"], state["centers"] = quant, centers.to(torch.bfloat16)
        for name in "kv":
            state["op_" + name] = Operator(**_weights(case, gen))
            state["rows_" + name] = _rows(case["tokens"], centers, gen)
            state["hist_" + name] = CompressedHistory(
                joint=heads * HEAD_DIM, rank=case["rank"], capacity=case["tokens"], group=quant.group,
                max_segments=case["tokens"] // case["chunk"], centers_per_segment=case["clusters"],
                scale_dtype=quant.scale_dtype)
    elif path == "decode":
        state["segments"] = _lingbot_cache(case, layer, centers, gen)["codec_segments"]
    elif path == "read":
        for name in "kv":
            state["op_" + name] = Operator(**_weights(case, gen))
            state["hist_" + name] = _history(case, case["tokens"], centers, torch.bfloat16, state["op_" + name], gen)
        state["q"] = _queries(case["queries"], heads, gen)
        state["rope"] = {}
        if case["rope"]:
            state["rope"] = dict(rope=RopeTable(_freqs(), frame_seqlen=FRAME, width=WIDTH),
                                 positions=torch.arange(case["tokens"], dtype=torch.int32, device="cuda"))
    elif path == "fast":
        protected = 2 * FRAME
        for name in "kv":
            op = state["op_" + name] = Operator(**_weights(case, gen))
            state["old_" + name] = _history(case, case["tokens"] - protected, centers, torch.bfloat16, op, gen)
            state["new_" + name] = _history(case, protected, centers, torch.bfloat16, op, gen)
        state["reader"] = Reader(_reader(case, gen, case["low_heads"], case["low_width"]), dtype=torch.bfloat16)
        state["q"] = _queries(case["queries"], heads, gen)
    elif path in ("lb_turn", "lb_fast"):
        state["cache"] = _lingbot_cache(case, layer, centers, gen)
        state["table"] = RopeTable(_freqs(), frame_seqlen=FRAME, width=WIDTH)
        count, start = case["chunk"], case["tokens"]
        state["steps"] = []
        for turn in range(2 if path == "lb_turn" else 1):
            q = _queries(count, heads, gen)
            now = torch.arange(start + turn * count, start + (turn + 1) * count, dtype=torch.int32, device="cuda")
            state["steps"].append(dict(
                q_pre=q[None], q=state["table"].rotate(q, now)[None], start=start + turn * count,
                key=_rows(count, centers, gen).view(1, -1, heads, HEAD_DIM),
                value=_rows(count, centers, gen).view(1, -1, heads, HEAD_DIM)))
        if path == "lb_fast":
            lingbot_attention.register_reader(layer, _reader(case, gen, heads * 3 // 4, 64),
                                              policy={"recent_native_frames": 2, "sink_native_frames": 1})
            state["freqs"], state["grid"] = _freqs(), torch.tensor([[64, FRAME // WIDTH, WIDTH]])
    else:
        for name in "kv":
            state["op_" + name] = Operator(**_weights(case, gen, torch.float32))
            state["rows_" + name] = _rows(case["tokens"], centers, gen, torch.float32)
            state["hist_" + name] = CompressedHistory(joint=heads * HEAD_DIM, rank=case["rank"],
                                                      capacity=case["tokens"], max_segments=1,
                                                      centers_per_segment=case["clusters"])
        state["centers"] = centers.to(torch.bfloat16)
        state["q"] = _queries(case["queries"], heads, gen, torch.float32)
    return state


# ------------------------------------------------------------------ one pass
def _written(hist):
    return [hist.codes, hist.scales, hist.ids]


def run(state):
    case = state["case"]
    path = case["path"]
    if path == "mg_encode":
        payload = mg_codec.encode_tensor("k", state["layer"], state["rows"])
        return [payload[name] for name in ("packed_codes", "scale", "centers", "ids")]
    if path == "lb_encode":
        pair = lingbot_codec.encode_pair(state["key"], state["value"], cache=state["cache"])
        return [pair[target][name] for target in "kv"
                for name in ("latent_packed", "latent_scale", "centers", "ids")]
    if path == "append":
        hist_k, hist_v = state["hist_k"], state["hist_v"]
        hist_k.retain([])                  # the rollout starts over
        hist_v.retain([])
        for first in range(0, case["tokens"], case["chunk"]):
            part = slice(first, first + case["chunk"])
            encode_append(hist_k, state["rows_k"][part], state["op_k"], state["quant"], centers=state["centers"])
            encode_append(hist_v, state["rows_v"][part], state["op_v"], state["quant"], centers=state["centers"])
        return _written(hist_k) + _written(hist_v)
    if path == "decode":
        return lingbot_codec.decode_segments(state["segments"], dtype=torch.bfloat16, device="cuda")
    if path == "read":
        return codec_attention(state["q"], state["hist_k"], state["hist_v"], state["op_k"], state["op_v"],
                               **state["rope"])
    if path == "fast":
        native = dict(k=state["new_k"], v=state["new_v"], op_k=state["op_k"], op_v=state["op_v"])
        low = dict(k=state["old_k"], v=state["old_v"], k_mean=state["op_k"].mean, v_mean=state["op_v"].mean)
        return hybrid_attention(state["q"], state["q"], [native], [low], state["reader"])
    if path == "lb_turn":
        # the rollout's cache as it stands at the start of the turn; the committing call appends to it
        cache = dict(state["cache"], codec_segments=list(state["cache"]["codec_segments"]))
        results = []
        for step, commit in zip(state["steps"], (True, False)):
            cache["codec_commit"] = commit
            results += lingbot_attention.codec_cache_attention(
                cache, step["q"], step["key"], step["value"], current_start=step["start"], rope=state["table"],
                **_window(case))
        return results
    if path == "lb_fast":
        step = state["steps"][0]
        return lingbot_attention.attend(
            step["q_pre"], step["q"], step["key"], step["value"], state["cache"], current_start=step["start"],
            grid_sizes=state["grid"], freqs=state["freqs"], frame_seqlen=FRAME, **_window(case))
    for name in "kv":
        state["hist_" + name].retain([])
        encode_append(state["hist_" + name], state["rows_" + name], state["op_" + name], QuantSpec(),
                      centers=state["centers"])
    out, lse = codec_attention(state["q"], state["hist_k"], state["hist_v"], state["op_k"], state["op_v"])
    return [out, lse] + _written(state["hist_k"]) + _written(state["hist_v"])


# ------------------------------------------------------------------ what a pass cannot do without
def _encode_work(tokens, case, size=2, iters=0):
    """One tensor: rows, operator and centres read, codes and scales written; the assignment (once per C-means
    iteration) and the projection.  ``iters`` 0: given centres."""
    joint, rank, clusters = case["heads"] * HEAD_DIM, case["rank"], case["clusters"]
    scales = 2 * rank // 32 if case.get("group32") else 2
    data = tokens * (joint * size + rank // 2 + scales + (1 if clusters <= 256 else 2))
    fixed = rank * joint * size + joint * 4 + clusters * joint * 2
    return data + fixed, 2.0 * tokens * joint * (clusters * max(iters, 1) + rank)


def _read_work(tokens, queries, case, heads=None, width=HEAD_DIM, size=2, codec=True):
    """Rebuild and attend ``tokens`` at ``width`` on ``heads`` heads: packed history, operators and queries
    in, (O, lse) out."""
    heads = case["heads"] if heads is None else heads
    rank, joint = case["rank"], heads * width
    data = 2.0 * queries * joint * size + queries * heads * 4
    flops = 4.0 * tokens * queries * joint
    if codec:
        data += 2.0 * (tokens * (rank // 2 + 3) + joint * rank * size + case["clusters"] * joint * 2)
        flops += 4.0 * tokens * rank * joint
    else:
        data += 2.0 * tokens * joint * size
    return data, flops


def work(case):
    path, heads = case["path"], case["heads"]
    joint, tokens = heads * HEAD_DIM, case["tokens"]
    if path == "mg_encode":
        parts = [_encode_work(tokens, case, iters=2)]
    elif path == "lb_encode":
        parts = [_encode_work(tokens, case, iters=2)] * 2
    elif path == "append":
        parts = [_encode_work(tokens, case)] * 2
    elif path == "decode":
        segments = tokens // case["chunk"]
        parts = [(tokens * (joint * 2 + case["rank"] // 2 + 3) + joint * case["rank"] * 2
                  + segments * case["clusters"] * joint * 2, 2.0 * tokens * joint * case["rank"])] * 2
    elif path == "read":
        parts = [_read_work(tokens, case["queries"], case)]
    elif path == "fast":
        low, rest = case["low_heads"], heads - case["low_heads"]
        parts = [_read_work(2 * FRAME, case["queries"], case),
                 _read_work(tokens - 2 * FRAME, case["queries"], case, low, case["low_width"]),
                 _read_work(tokens - 2 * FRAME, case["queries"], case, rest)]
    elif path == "lb_turn":
        # each call sees ``tokens`` keys: the window's and its own chunk's
        count = case["chunk"]
        parts = [_read_work(tokens - count, count, case), _read_work(count, count, case, codec=False)] * 2
        parts += [_encode_work(count, case, iters=2)] * 2
    elif path == "lb_fast":
        count = case["chunk"]
        protected = min(3 * FRAME, tokens - count)
        low, rest = heads * 3 // 4, heads - heads * 3 // 4
        parts = [_read_work(protected, count, case), _read_work(count, count, case, codec=False),
                 _read_work(tokens - count - protected, count, case, low, 64),
                 _read_work(tokens - count - protected, count, case, rest)]
    else:
        parts = [_encode_work(tokens, case, 4)] * 2 + [_read_work(tokens, case["queries"], case, size=4)]
    return dict(bytes=sum(p[0] for p in parts), flops=sum(p[1] for p in parts))


def tolerance(case):
    """About four times what the same pass gives with its sums in another order (the CUDA-core kernels, or float64)."""
    path = case["path"]
    if path in ("mg_encode", "lb_encode"):
        # C-means: two start rows may come from one true cluster, so a distance can tie to its last bit; one label
        # that flips moves its centre, and with it the codes of that centre's tokens (seen: 1.3e-2 of the codes,
        # 2.3e-2 on the scales, 1560 tokens); without a flip 7e-5 and 2e-4
        return {"rel": 3e-2, "max": 0.5, "differ": 1e-2}
    if path == "append":
        # a coefficient moves by its last bits: a code by one step at a rounding boundary (seen: 6e-5 of the
        # codes), a scale by one step of its own type (2e-4 in norm)
        return {"rel": 8e-4, "max": 2e-2, "differ": 3e-4}
    if path == "decode":
        return {"rel": 2e-3, "max": 2e-2}      # the last bf16 rounding of a row value
    if path == "roundtrip":
        # O 2e-5 against float64; one scale of the stored bf16 ones may move by one step (1.6e-4 in norm)
        return {"rel": 6e-4, "max": 1e-2, "differ": 2e-5}
    return {"rel": 1e-2, "max": 8e-2}          # softmax weights in bf16 (seen: 2.5e-3, largest 2e-2)
