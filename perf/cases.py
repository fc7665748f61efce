"""What this library's users have it do, as cases that can be timed and checked.

Two kinds of case are whole calls: `step` is a decode step of a Qwen3 model (its launches replayed from a CUDA graph, as generation
does), `prompts` is `Engine.step` over the prompts of a batch.  The others are the parts that the library's other designs are made of,
each with its projections and in both directions: a further portion of a prompt (several rows per sequence) or one token per sequence
(`rows` == `sequences`).  A pass whose launches the engine would replay from a graph (one token each, or a bfloat16 pass of at most
1,024 rows) is replayed from one here too; a longer one is launched call by call.

  masked   grouped-query attention of Rovurax (chunks), Barorax (chunks, rotation, unit-norm queries and keys, one more term in the
           denominator) and Tarudra (window, rotation, biases, one more term)
  latent   latent attention of Rovurax (gate per head, sink) and Tarudra (query latents, window, gate per value)
  experts  routed feed-forward of Tenetar (squared-ReLU experts in groups, identity experts, shared expert) and Retuvik (gated experts)
  wkv      Retuvik's matrix-state recurrence;  ssm  Barorax's selective scan;  gated  Ravapel's gated recurrence;  delta  Tarudra's
           gated delta rule: each goes on from a state

Sizes are the library's own benchmark sizes: layers of a 1.7B and of an 8B model, and of the 0.6B one."""
import math
import random

import numpy as np
import torch

DEVICE = "cuda:0"
EPS = 1e-6
PAGE = 64
SIZES = {      # width, feed-forward, query heads, key/value heads
    "0.6b": (1024, 3072, 16, 8),
    "1.7b": (2048, 6144, 16, 8),
    "8b": (4096, 12288, 32, 8),
}
PARTS = ("masked", "latent", "experts", "wkv", "ssm", "gated", "delta")
RECURRENT = ("wkv", "ssm", "gated", "delta")
GRAPH_ROWS = 1024


def listed():
    return [
        # generation with a batch of 8 at the benchmark's mean context: the headline workload, four layers of it
        dict(name="step 8b batch 8", kind="step", size="8b", dtype="bfloat16", sequences=8, rows=8, context=3072, layers=4),
        # one user, short context, small model: the smallest call, where launches and latency count
        dict(name="step 1.7b batch 1", kind="step", size="1.7b", dtype="bfloat16", sequences=1, rows=1, context=300, layers=2),
        # a batch of prompts of unequal lengths arriving together
        dict(name="prompts 1.7b ragged", kind="prompts", size="1.7b", dtype="bfloat16", sequences=16, rows=9456, context=0, layers=2),
        # the 32-bit path (exact replay of traces): a prompt of ordinary length
        dict(name="prompts 1.7b 32-bit", kind="prompts", size="1.7b", dtype="float32", sequences=2, rows=700, context=0, layers=1),
        # long prompts through windowed attention with biases and rotation
        dict(name="masked prompt 8b", kind="masked", size="8b", dtype="bfloat16", sequences=2, rows=8192, context=0, style="tarudra",
             head_dim=128, v_dim=128, span=2048),
        # a full batch decoding through chunked attention
        dict(name="masked decode 8b batch 64", kind="masked", size="8b", dtype="bfloat16", sequences=64, rows=64, context=3072, style="barorax",
             head_dim=128, v_dim=128, span=1024),
        # one prompt through latent attention
        dict(name="latent prompt 8b", kind="latent", size="8b", dtype="bfloat16", sequences=1, rows=2048, context=0, style="rovurax",
             head_dim=128, v_dim=128, rank=256, rot=64, span=0),
        # routed experts over the rows of a prompt
        dict(name="experts prompt 1.7b", kind="experts", size="1.7b", dtype="bfloat16", sequences=1, rows=2048, context=0, style="retuvik",
             experts=16, top=4, ff=1024),
        # the recurrences over a portion of one prompt, over several short ones, and decoding a full batch
        dict(name="wkv prompt 1.7b", kind="wkv", size="1.7b", dtype="bfloat16", sequences=1, rows=2048, context=64, head_dim=64),
        dict(name="ssm prompt 1.7b", kind="ssm", size="1.7b", dtype="bfloat16", sequences=1, rows=2048, context=64, states=16),
        dict(name="gated decode 1.7b batch 64", kind="gated", size="1.7b", dtype="bfloat16", sequences=64, rows=64, context=512, head_dim=128, v_dim=128),
        dict(name="delta prompts 1.7b", kind="delta", size="1.7b", dtype="bfloat16", sequences=4, rows=2011, context=64, head_dim=128, v_dim=128),
    ]


def _log(rng, lo, hi):
    """A whole number from lo to hi, spread over its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))))


def _cost(case):
    w = work(case)
    return max(w["bytes"], w["flops"] / (50 if case["dtype"] == "bfloat16" else 5))


def draw(rng):
    most = max(_cost(c) for c in listed())
    while True:
        kind = rng.choice(("step", "prompts") + PARTS)
        c = dict(kind=kind, size=rng.choice(sorted(SIZES)), dtype="float32" if rng.random() < 0.15 else "bfloat16")
        one = kind == "step" or (kind != "prompts" and rng.random() < 0.5)       # one token per sequence
        wide = c["dtype"] == "bfloat16"
        if one:
            c["sequences"] = c["rows"] = _log(rng, 1, 64 if wide else 8)
            c["context"] = _log(rng, 16, 8192 if wide else 1024)
        else:
            c["rows"] = _log(rng, 12, 8192 if wide else 600)
            c["sequences"] = _log(rng, 1, min(16, c["rows"] // 8 or 1))
            c["context"] = _log(rng, 1, 512) if kind in RECURRENT else 0
        if kind in ("step", "prompts"):
            c["layers"] = rng.randint(1, 4)
        elif kind == "masked":
            c["style"] = rng.choice(("rovurax", "barorax", "tarudra"))
            c["head_dim"], c["v_dim"], c["span"] = rng.choice((64, 96, 128, 128)), rng.choice((64, 128, 128)), rng.choice((0, 333, 1024, 2048))
        elif kind == "latent":
            c["style"] = rng.choice(("rovurax", "tarudra"))
            c["head_dim"], c["v_dim"], c["rank"], c["rot"] = rng.choice((64, 128)), rng.choice((64, 128)), rng.choice((128, 256)), rng.choice((32, 64))
            c["span"] = rng.choice((0, 777, 1024)) if c["style"] == "tarudra" else 0
        elif kind == "experts":
            c["style"] = rng.choice(("tenetar", "retuvik"))
            c["experts"], c["top"], c["ff"] = rng.choice((8, 16, 32)), rng.randint(1, 4), 256 * rng.randint(2, 8)
        elif kind == "ssm":
            c["states"] = rng.choice((8, 16, 16, 32))
        elif kind == "wkv":
            c["head_dim"] = 64
        else:
            c["head_dim"], c["v_dim"] = rng.choice((64, 128)), rng.choice((64, 128))
        if _cost(c) <= most:
            return c


# ------------------------------------------------------------------------------------------ what a case holds
def _lengths(case):
    """Rows of every sequence: unequal shares of `rows`, the same for the same case."""
    n, rows = case["sequences"], case["rows"]
    if rows == n:
        return [1] * n
    r = random.Random("%d rows in %d" % (rows, n))
    share = [r.uniform(0.2, 1.8) for _ in range(n)]
    out = [max(1, int(rows * s / sum(share))) for s in share]
    out[max(range(n), key=lambda i: out[i])] += rows - sum(out)
    return out


def _starts(case):
    """The position at which every sequence's rows start: between half of `context` and all of it."""
    n, ctx = case["sequences"], case["context"]
    r = random.Random("%d sequences at %d" % (n, ctx))
    return [ctx - r.randrange(ctx // 2 + 1) if n > 1 else ctx for _ in range(n)]


def _vocab(case):
    return 16384


def _heads(case):
    w, _, h, g = SIZES[case["size"]]
    if case["kind"] == "wkv":
        return w // case["head_dim"], 0
    if case["kind"] == "gated":
        return w // case["v_dim"], 0
    if case["kind"] == "delta":
        return w // case["v_dim"], w // case["v_dim"] // 2
    return h, g


def _shapes(case):
    """Checkpoint tensors: name -> (shape, how it is made).  m: a matrix; n: norm weights near 1; s: small numbers."""
    w, ff, h, g = SIZES[case["size"]]
    k = case["kind"]
    if k in ("step", "prompts"):
        out = {"model.embed_tokens.weight": ((_vocab(case), w), "m"), "lm_head.weight": ((_vocab(case), w), "m"), "model.norm.weight": ((w,), "n")}
        for i in range(case["layers"]):
            p = "model.layers.%d." % i
            out.update({p + "self_attn.q_proj.weight": ((h * 128, w), "m"), p + "self_attn.k_proj.weight": ((g * 128, w), "m"),
                        p + "self_attn.v_proj.weight": ((g * 128, w), "m"), p + "self_attn.o_proj.weight": ((w, h * 128), "m"),
                        p + "self_attn.q_norm.weight": ((128,), "n"), p + "self_attn.k_norm.weight": ((128,), "n"),
                        p + "mlp.gate_proj.weight": ((ff, w), "m"), p + "mlp.up_proj.weight": ((ff, w), "m"), p + "mlp.down_proj.weight": ((w, ff), "m"),
                        p + "input_layernorm.weight": ((w,), "n"), p + "post_attention_layernorm.weight": ((w,), "n")})
        return out
    heads, groups = _heads(case)
    d, v = case.get("head_dim", 0), case.get("v_dim", 0)
    if k == "masked":
        out = {"q": ((heads * d, w), "m"), "k": ((groups * d, w), "m"), "v": ((groups * v, w), "m"), "o": ((w, heads * v), "m")}
        if case["style"] == "tarudra":
            out.update({"q_bias": ((heads * d,), "s"), "k_bias": ((groups * d,), "s"), "v_bias": ((groups * v,), "s"), "o_bias": ((w,), "s")})
        return out
    if k == "latent":
        r, rot, q_rank = case["rank"], case["rot"], w // 4 if case["style"] == "tarudra" else 0
        out = {"dq": ((q_rank, w), "m"), "dq_norm": ((q_rank,), "n")} if q_rank else {}
        out.update({"q": ((heads * (d + rot), q_rank or w), "m"), "dkv": ((r + rot, w), "m"), "dkv_norm": ((r,), "n"), "uk": ((heads * d, r), "m"),
                    "uv": ((heads * v, r), "m"), "o": ((w, heads * v), "m"), "gate": ((heads * v if q_rank else heads, w), "m")})
        if not q_rank:
            out["sink"] = ((heads,), "s")
        return out
    if k == "experts":
        e, f = case["experts"], case["ff"]
        t = case["style"] == "tenetar"
        out = {"router": ((e + 2 if t else e, w), "m"), "correction": ((e + 2 if t else e,), "s")}
        for i in range(e):
            out.update({"e%d.up" % i: ((f, w), "m"), "e%d.down" % i: ((w, f), "m")})
            if not t:
                out["e%d.gate" % i] = ((f, w), "m")
        if t:
            out.update({"shared.up": ((f, w), "m"), "shared.down": ((w, f), "m"), "shared.gate": ((1, w), "m")})
        return out
    if k == "wkv":
        hn = heads * d
        out = {"mu." + s: ((w,), "u") for s in "rkvgw"}
        out.update({s: ((hn, w), "m") for s in "rkvg"})
        out.update({"w1": ((64, w), "m"), "w2": ((hn, 64), "m"), "w0": ((hn,), "d"), "u": ((heads, d), "s"), "norm": ((hn,), "n"), "o": ((w, hn), "m")})
        return out
    if k == "ssm":
        i, s, r = 2 * w, case["states"], w // 16
        return {"in": ((2 * i, w), "m"), "conv": ((i, 4), "c"), "conv_bias": ((i,), "s"), "x": ((r + 2 * s, i), "m"), "dt": ((i, r), "m"),
                "dt_bias": ((i,), "b"), "A_log": ((i, s), "a"), "D": ((i,), "n"), "o": ((w, i), "m")}
    if k == "gated":
        return {"q": ((heads * d, w), "m"), "f": ((heads * d, w), "m"), "f_bias": ((heads * d,), "s"), "lower": ((heads * d,), "u"),
                "v": ((heads * v, w), "m"), "norm": ((v,), "n"), "o": ((w, heads * v), "m")}
    rows = {"q": groups * d, "k": groups * d, "v": heads * v}
    out = {s: ((n, w), "m") for s, n in rows.items()}
    out.update({s + "_conv": ((n, 4), "c") for s, n in rows.items()})
    out.update({"a": ((heads, w), "m"), "b": ((heads, w), "m"), "A_log": ((heads,), "s"), "dt_bias": ((heads,), "b"), "norm": ((v,), "n"),
                "g": ((heads * v, w), "m"), "o": ((w, heads * v), "m")})
    return out


def _tensor(shape, how, dtype, gen):
    t = torch.empty(shape, dtype=torch.float32 if how != "m" else dtype, device=DEVICE)
    if how == "m":                                   # outputs of unit size for inputs of unit size
        return t.normal_(0.0, shape[-1] ** -0.5, generator=gen)
    if how == "n":
        return t.normal_(1.0, 0.1, generator=gen)
    if how == "u":                                   # blends and lower bounds
        return t.uniform_(0.05, 0.95, generator=gen)
    if how == "d":                                   # decay exponents: from quickly forgetting to long memory
        return t.uniform_(-6.0, 0.0, generator=gen)
    if how == "b":                                   # step sizes after softplus from about 0.001 to 0.1
        return t.uniform_(-7.0, -2.2, generator=gen)
    if how == "a":                                   # decay rates 1 .. states per channel
        return t.copy_(torch.log(torch.arange(1, shape[1] + 1, device=DEVICE, dtype=torch.float32)).expand(shape)).add_(
            torch.empty_like(t).normal_(0.0, 0.1, generator=gen))
    if how == "c":                                   # four taps
        return t.normal_(0.0, 0.5, generator=gen)
    return t.normal_(0.0, 0.5, generator=gen)


def _state_floats(case):
    w, _, _, _ = SIZES[case["size"]]
    heads, groups = _heads(case)
    k, d, v = case["kind"], case.get("head_dim", 0), case.get("v_dim", 0)
    if k == "wkv":
        return heads * d * d, w
    if k == "ssm":
        return 2 * w * case["states"], 3 * 2 * w
    if k == "gated":
        return heads * v * d, 0
    return heads * v * d, 4 * (2 * groups * d + heads * v)


def _inputs(case, seed):
    """Everything that is drawn: tensors by name, the rows, and what the sequences' cache or state holds."""
    gen = torch.Generator(device=DEVICE)
    gen.manual_seed(seed)
    dt = getattr(torch, case["dtype"])
    t = {n: _tensor(s, how, dt, gen) for n, (s, how) in _shapes(case).items()}
    w, _, h, g = SIZES[case["size"]]
    got = {"tensors": t, "past": [], "state": None}
    normal = lambda *shape: torch.empty(shape, dtype=dt, device=DEVICE).normal_(generator=gen)
    if case["kind"] in ("step", "prompts"):
        got["tokens"] = torch.randint(0, _vocab(case), (case["rows"],), generator=gen, device=DEVICE, dtype=torch.int64)
    else:
        got["x"] = normal(case["rows"], w)
    if case["kind"] in RECURRENT:
        a, b = _state_floats(case)
        got["state"] = torch.empty((case["sequences"], a + b), device=DEVICE).normal_(0.0, 0.3, generator=gen)
    elif case["kind"] != "experts":
        for s in _starts(case):                       # keys (and values) of the positions before the rows, per layer
            if s == 0:
                got["past"].append(None)
            elif case["kind"] == "step":
                got["past"].append([(normal(s, g, 128), normal(s, g, 128)) for _ in range(case["layers"])])
            elif case["kind"] == "masked":
                got["past"].append([(normal(s, g, case["head_dim"]), normal(s, g, case["v_dim"]))])
            else:
                got["past"].append([(normal(s, 1, case["rank"] + case["rot"]), None)])
    return got


# ------------------------------------------------------------------------------------------ the library's parts
def _part_spec(case):
    """(kind of part, its parameters, its position encoding's kind and parameters or None)"""
    w, ff, h, g = SIZES[case["size"]]
    heads, groups = _heads(case)
    k, names = case["kind"], {n: n for n in _shapes(case)}
    d, v = case.get("head_dim", 0), case.get("v_dim", 0)
    if k == "masked":
        p = dict(hidden_size=w, q_heads=heads, kv_heads=groups, head_dim=d, v_dim=v, scale=d ** -0.5, ring=False, names=names)
        if case["style"] == "tarudra":
            p.update(window=case["span"] or None, position="rot", sink_zero=True, bias=True)
            return "masked_attention", p, ("yarn_rope", dict(rotary_dim=d, theta=1000000.0))
        if case["style"] == "barorax":
            p.update(chunk=case["span"] or None, position="rot", sink_zero=True, qk_unit_eps=EPS, scale=8.0 / d)
            return "masked_attention", p, ("yarn_rope", dict(rotary_dim=d, theta=10000.0))
        p.update(chunk=case["span"] or None)
        return "masked_attention", p, None
    if k == "latent":
        p = dict(hidden_size=w, heads=heads, head_dim=d, rot_dim=case["rot"], v_dim=v, kv_rank=case["rank"], scale=(d + case["rot"]) ** -0.5,
                 norm_eps=EPS, position="rot", gate=True, names=names)
        if case["style"] == "tarudra":
            p.update(q_rank=w // 4, window=case["span"] or None, gate_wide=True)
            return "latent_attention", p, ("yarn_rope", dict(rotary_dim=case["rot"], theta=1000000.0, layout="half"))
        p.update(sink=True)
        return "latent_attention", p, ("yarn_rope", dict(rotary_dim=case["rot"], theta=1000000.0))
    if k == "experts":
        p = dict(hidden_size=w, experts=case["experts"], top=case["top"], expert_size=case["ff"])
        n = dict(router="router", correction="correction", up="e{e}.up", down="e{e}.down")
        if case["style"] == "tenetar":
            n.update(shared_up="shared.up", shared_down="shared.down", shared_gate="shared.gate")
            p.update(identity=2, groups=2, keep_groups=1, shared_size=case["ff"], shared_gate=True, names=n)
        else:
            n.update(gate="e{e}.gate")
            p.update(activation="swiglu", choice="logits", names=n)
        return "routed_experts", p, None
    if k == "wkv":
        names["mu"] = "mu.{s}"
        return "matrix_state_recurrence", dict(hidden_size=w, heads=heads, head_dim=d, decay_rank=64, eps=EPS, names=names), None
    if k == "ssm":
        return "selective_scan", dict(hidden_size=w, inner=2 * w, state=case["states"], conv=4, dt_rank=w // 16, names=names), None
    if k == "gated":
        return "channel_gated_recurrence", dict(hidden_size=w, heads=heads, head_dim=d, v_dim=v, eps=EPS, names=names), None
    return "gated_delta_rule", dict(hidden_size=w, heads=heads, kv_heads=groups, head_dim=d, v_dim=v, taps=4, eps=EPS, names=names), None


def _qwen3(case):
    from x0ne_engine_b200 import Qwen3Config
    w, ff, h, g = SIZES[case["size"]]
    return Qwen3Config(hidden_size=w, intermediate_size=ff, num_hidden_layers=case["layers"], num_attention_heads=h, num_key_value_heads=g,
                       head_dim=128, vocab_size=_vocab(case), max_position_embeddings=16384, rms_norm_eps=EPS, rope_theta=1000000.0,
                       tie_word_embeddings=False, dtype=case["dtype"]).to_spec()


def _fill(cache, slots, past):
    """Puts the sequences' past keys and values into their pages: keys of every kv head, then values."""
    for entry, group in ((e, g) for g in cache.groups for e in g.entries):
        pages = group.storage[group.entries.index(entry)].view(group.n_pages, -1)
        for slot, kv in zip(slots, past):
            if kv is None:
                continue
            k, v = kv[entry]
            n = -(-k.shape[0] // PAGE)
            at = torch.from_numpy(group.table_host[slot, :n].astype(np.int64)).to(DEVICE)
            flat = []
            for rows in (k, v):
                if rows is not None:
                    whole = torch.zeros((n * PAGE,) + tuple(rows.shape[1:]), dtype=rows.dtype, device=DEVICE)
                    whole[:rows.shape[0]] = rows
                    flat.append(whole.view(n, PAGE, rows.shape[1], rows.shape[2]).transpose(1, 2).reshape(n, -1))
            pages[at] = torch.cat(flat, dim=1)


def _context(case, cache, slots, dtype, tokens=None):
    """The tables of one pass over every sequence's rows, as the engine makes them."""
    from x0ne_engine_b200.csrc import ops
    from x0ne_engine_b200.engine.engine import StepContext
    from x0ne_engine_b200.engine.workspace import Workspace
    lens, starts = _lengths(case), _starts(case)
    first = np.concatenate([[0], np.cumsum(lens)])
    tile = ops.PREFILL_TILE_ROWS if dtype == torch.bfloat16 else 64
    tiles = [(s, int(first[s]) + r) for s, n in enumerate(lens) for r in range(0, n, tile)]
    dev = lambda v: torch.tensor(v, dtype=torch.int32, device=DEVICE)
    ws = Workspace(case["rows"], torch.device(DEVICE))
    ws.max_want = case["rows"]
    return StepContext(
        n_rows=case["rows"], tokens=dev([0] * case["rows"]) if tokens is None else tokens.to(torch.int32),
        row_slot=dev([slots[s] for s, n in enumerate(lens) for _ in range(n)]), row_pos=dev([starts[s] + i for s, n in enumerate(lens) for i in range(n)]),
        dtype=dtype, ws=ws, cache=cache, decode=max(lens) == 1, n_seqs=len(lens), max_seq_rows=max(lens),
        max_context=max(s + n for s, n in zip(starts, lens)), seq_first_row=dev(list(first)), seq_slot=dev(slots), seq_pos0=dev(starts), n_tiles=len(tiles),
        tile_seq=dev([t[0] for t in tiles]), tile_row0=dev([t[1] for t in tiles]),
        sm_count=torch.cuda.get_device_properties(DEVICE).multi_processor_count)


def _replayed(call, states):
    """The call as a CUDA graph; what its first run changes in `states` is put back."""
    saved = [s.clone() for s in states]
    call()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        call()
    for s, b in zip(states, saved):
        s.copy_(b)
    return graph


def prepare(case, seed):
    """What a program holds before the call: weights bound to the part or model, the cache or state of its sequences, the pass's tables,
    and the captured launches where the engine would replay them."""
    from x0ne_engine_b200.cache import SequenceCache
    from x0ne_engine_b200.config.spec import PartSpec
    from x0ne_engine_b200.engine.engine import Engine
    from x0ne_engine_b200.engine.model import CausalLM
    from x0ne_engine_b200.parts import FEED_FORWARDS, MIXERS, POSITIONS, BuildEnv
    dt, device = getattr(torch, case["dtype"]), torch.device(DEVICE)
    got = _inputs(case, seed)
    lens, starts = _lengths(case), _starts(case)
    longest = -(-max(s + n for s, n in zip(starts, lens)) // PAGE) * PAGE
    room = sum(-(-(s + n) // PAGE) * PAGE for s, n in zip(starts, lens))
    if case["kind"] == "prompts":
        engine = Engine(_qwen3(case), got["tensors"], dt, DEVICE, max_tokens=room, max_seq_len=longest, max_step_tokens=case["rows"], max_slots=case["sequences"])
        return {"engine": engine, "prompts": [p.tolist() for p in got["tokens"].cpu().split(lens)]}
    if case["kind"] == "step":
        spec = _qwen3(case)
        model = CausalLM(spec, dt, device, max_positions=longest)
        model.bind(got["tensors"])
        needs, reads = model.cache_needs(), [None] * case["layers"]
    else:
        kind, params, position = _part_spec(case)
        params = PartSpec(kind, params)
        env = BuildEnv(dtype=dt, device=device, max_positions=longest)
        if position is not None:
            env.positions["rot"] = POSITIONS.get(position[0])(PartSpec(*position), env)
        part = (FEED_FORWARDS if case["kind"] == "experts" else MIXERS).get(kind)(params, env)
        part.bind(got["tensors"])
        needs, reads = [part.cache_needs(params) if case["kind"] != "experts" else []], [None]
    cache = SequenceCache(needs, reads, room, longest, dt, device, max_slots=case["sequences"])
    slots = [cache.acquire(s + n) for s, n in zip(starts, lens)]
    states = []
    if case["kind"] in RECURRENT:
        state = cache.state(0)
        states = [state]
        order = torch.tensor(slots, device=DEVICE)
        if case["kind"] == "delta" or case["kind"] == "gated":       # (rows padded to 16 bytes)
            assert state.shape[1] == got["state"].shape[1]
        state[order] = got["state"]
    if got["past"]:
        _fill(cache, slots, got["past"])
    ctx = _context(case, cache, slots, dt, got.get("tokens"))
    n = case["rows"]
    if case["kind"] == "step":
        logits = torch.empty((n, spec.vocab_size), dtype=torch.float32, device=DEVICE)
        rows = torch.arange(n, dtype=torch.int32, device=DEVICE)
        call = lambda: model.forward(ctx, rows, n, logits)
        result = {"logits": logits}
    else:
        call = (lambda: part.forward(ctx, got["x"], n)) if case["kind"] == "experts" else (lambda: part.forward(ctx, 0, got["x"], n))
        result = None
    state = {"ctx": ctx, "cache": cache, "result": result, "states": states, "call": call, "graph": None, "rows": n, "order": slots}
    if ctx.decode or (dt == torch.bfloat16 and n <= GRAPH_ROWS):
        def kept():
            state["out"] = call()
        state["graph"] = _replayed(kept, states)
        state["result"] = result or {"out": state["out"][:n]}
    if states and slots != sorted(slots):
        raise RuntimeError("the cache hands out slots in order")
    return state


def run(state):
    if "engine" in state:
        engine = state["engine"]
        slots = [engine.new_sequence(len(p)) for p in state["prompts"]]
        logits = engine.step(slots, state["prompts"])
        for s in slots:
            engine.free_sequence(s)
        return {"logits": logits}
    if state["graph"] is not None:
        state["graph"].replay()
        out = state["result"]
    else:
        got = state["call"]()
        out = state["result"] or {"out": got[:state["rows"]]}
    return dict(out, state=state["states"][0]) if state["states"] else out


# ------------------------------------------------------------------------------------------ what a pass cannot do without
def _seen(case):
    """(query, key) pairs that attention scores, and keys that it has to read."""
    span = case.get("span", 0)
    chunked = case["kind"] == "masked" and case["style"] != "tarudra"
    pairs = keys = 0
    for s, n in zip(_starts(case), _lengths(case)):
        pos = np.arange(s, s + n, dtype=np.int64)
        lo = np.zeros_like(pos) if not span else pos - pos % span if chunked else np.maximum(0, pos - span + 1)
        pairs += int((pos - lo + 1).sum())
        keys += int(pos[-1] - lo[0] + 1)
    return pairs, keys


def work(case):
    w, ff, h, g = SIZES[case["size"]]
    k, n, b = case["kind"], case["rows"], 2 if case["dtype"] == "bfloat16" else 4
    shapes = {name: s for name, (s, how) in _shapes(case).items()}
    size = lambda s: int(np.prod(s))
    matrices = {name: size(s) for name, s in shapes.items() if len(s) == 2 and not name.endswith("conv") and name not in ("A_log", "u")}
    if k in ("step", "prompts"):
        wanted = case["sequences"]
        pairs, keys = _seen(case)
        head, layers = _vocab(case) * w, sum(v for name, v in matrices.items() if "layers" in name)
        flops = 2 * n * layers + 2 * wanted * head + 4 * pairs * h * 128 * case["layers"]
        return {"bytes": b * (layers + head + n * w + 2 * keys * g * 128 * case["layers"]) + 4 * wanted * _vocab(case), "flops": flops}
    heads, groups = _heads(case)
    d, v = case.get("head_dim", 0), case.get("v_dim", 0)
    io = 2 * b * n * w
    if k == "experts":
        pairs = n * case["top"]
        hit = case["experts"] * (1 - (1 - case["top"] / case["experts"]) ** n)
        per = (3 if case["style"] == "retuvik" else 2) * case["ff"] * w
        shared = 2 * case["ff"] * w if case["style"] == "tenetar" else 0
        return {"bytes": io + b * (hit * per + shared + matrices["router"]), "flops": 2 * pairs * per + 2 * n * (shared + matrices["router"])}
    weights = sum(matrices.values())
    if k == "masked":
        pairs, keys = _seen(case)
        return {"bytes": io + b * (weights + keys * groups * (d + v)), "flops": 2 * n * weights + 2 * pairs * heads * (d + v)}
    if k == "latent":
        pairs, keys = _seen(case)
        row = case["rank"] + case["rot"]
        return {"bytes": io + b * (weights + keys * row), "flops": 2 * n * weights + 2 * pairs * heads * (row + case["rank"])}
    state = sum(_state_floats(case))
    per = {"wkv": 6 * heads * d * d, "ssm": 7 * 2 * w * case.get("states", 0), "gated": 5 * heads * d * v, "delta": 7 * heads * d * v}[k]
    return {"bytes": io + b * weights + 8 * case["sequences"] * state, "flops": 2 * n * weights + n * per}


def tolerance(case):
    """Of the largest differences seen between a pass and 64-bit results, about four times."""
    if case["dtype"] == "float32":
        return {"rel": 2e-5}
    return {"rel": 0.03 if case["kind"] in ("step", "prompts") else 0.02}


# ------------------------------------------------------------------------------------------ the same in 64 bits
def _rms(x):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS)


def _rotate(x, pos, dims, theta, half):
    """x [rows, heads, d]: the first `dims` values of every head turn by position x frequency."""
    f = theta ** (-2.0 * torch.arange(dims // 2, dtype=torch.float64, device=DEVICE) / dims)
    ang = pos.to(torch.float64)[:, None] * f
    c, s = torch.cos(ang)[:, None], torch.sin(ang)[:, None]
    a, b = (slice(0, dims // 2), slice(dims // 2, dims)) if half else (slice(0, dims, 2), slice(1, dims, 2))
    out = x.clone()
    out[..., a], out[..., b] = x[..., a] * c - x[..., b] * s, x[..., b] * c + x[..., a] * s
    return out


def _attend(q, k, v, pos, scale, window=0, chunk=0, sink=None):
    """q [rows, H, d] at positions `pos`, k [keys, G, d] and v [keys, G, e] of positions 0 ..: softmax attention head by head."""
    rep = q.shape[1] // k.shape[1]
    out = torch.empty((q.shape[0], q.shape[1], v.shape[2]), dtype=q.dtype, device=DEVICE)
    at = torch.arange(k.shape[0], device=DEVICE)
    for a in range(0, q.shape[0], 4096):
        p = pos[a:a + 4096, None]
        unseen = at > p
        if window:
            unseen = unseen | (at <= p - window)
        if chunk:
            unseen = unseen | (at < p - p % chunk)
        for i in range(q.shape[1]):
            s = (q[a:a + 4096, i] @ k[:, i // rep].T * scale).masked_fill_(unseen, -math.inf)
            top = s.amax(-1, keepdim=True)
            if sink is not None:
                top = torch.maximum(top, sink[i])
            s = s.sub_(top).exp_()
            total = s.sum(-1, keepdim=True)
            if sink is not None:
                total = total + torch.exp(sink[i] - top)
            out[a:a + 4096, i] = s @ v[:, i // rep] / total
    return out


def _exact_qwen3(case, got):
    w, ff, h, g = SIZES[case["size"]]
    t = {n: v.double() for n, v in got["tensors"].items()}
    lens, starts = _lengths(case), _starts(case)
    first = np.concatenate([[0], np.cumsum(lens)])
    pos = torch.cat([torch.arange(s, s + n, device=DEVICE) for s, n in zip(starts, lens)])
    x = t["model.embed_tokens.weight"][got["tokens"]]
    for i in range(case["layers"]):
        p = "model.layers.%d." % i
        y = _rms(x) * t[p + "input_layernorm.weight"]
        q, k, v = ((y @ t[p + "self_attn.%s_proj.weight" % s].T).view(len(y), -1, 128) for s in "qkv")
        q, k = (_rotate(_rms(u) * t[p + "self_attn.%s_norm.weight" % s], pos, 128, 1000000.0, True) for u, s in ((q, "q"), (k, "k")))
        att = torch.empty((len(y), h * 128), dtype=torch.float64, device=DEVICE)
        for j in range(len(lens)):
            a, b = first[j], first[j + 1]
            ks, vs = k[a:b], v[a:b]
            if got["past"][j] is not None:
                ks, vs = (torch.cat([o.double(), u]) for o, u in zip(got["past"][j][i], (ks, vs)))
            att[a:b] = _attend(q[a:b], ks, vs, pos[a:b], 128 ** -0.5).flatten(1)
        x = x + att @ t[p + "self_attn.o_proj.weight"].T
        y = _rms(x) * t[p + "post_attention_layernorm.weight"]
        x = x + (torch.nn.functional.silu(y @ t[p + "mlp.gate_proj.weight"].T) * (y @ t[p + "mlp.up_proj.weight"].T)) @ t[p + "mlp.down_proj.weight"].T
    last = x[torch.from_numpy(first[1:] - 1).to(DEVICE)]
    return {"logits": _rms(last) * t["model.norm.weight"] @ t["lm_head.weight"].T}


def _exact_masked(case, t, x, got, pos, cuts):
    heads, groups = _heads(case)
    d, v, style = case["head_dim"], case["v_dim"], case["style"]
    bias = lambda s: t[s + "_bias"] if style == "tarudra" else 0.0
    q, k, val = ((x @ t[s].T + bias(s)).view(len(x), -1, n) for s, n in (("q", d), ("k", d), ("v", v)))
    if style != "rovurax":
        q, k = (_rotate(u, pos, d, 1000000.0 if style == "tarudra" else 10000.0, False) for u in (q, k))
    if style == "barorax":
        q, k = _rms(q), _rms(k)
    sink = None if style == "rovurax" else torch.zeros(heads, dtype=torch.float64, device=DEVICE)
    out = torch.empty((len(x), heads * v), dtype=torch.float64, device=DEVICE)
    for j, (a, b) in enumerate(cuts):
        ks, vs = k[a:b], val[a:b]
        if got["past"][j] is not None:
            ks, vs = (torch.cat([o.double(), u]) for o, u in zip(got["past"][j][0], (ks, vs)))
        out[a:b] = _attend(q[a:b], ks, vs, pos[a:b], 8.0 / d if style == "barorax" else d ** -0.5, case["span"] if style == "tarudra" else 0,
                           case["span"] if style != "tarudra" else 0, sink).flatten(1)
    return {"out": out @ t["o"].T + bias("o")}


def _exact_latent(case, t, x, got, pos, cuts):
    heads, _ = _heads(case)
    d, v, r, rot, wide = case["head_dim"], case["v_dim"], case["rank"], case["rot"], case["style"] == "tarudra"
    q = _rms(x @ t["dq"].T) * t["dq_norm"] if wide else x
    q = (q @ t["q"].T).view(len(x), heads, d + rot)
    q_rot = _rotate(q[..., d:], pos, rot, 1000000.0, wide)
    down = x @ t["dkv"].T
    rows = torch.cat([_rms(down[:, :r]) * t["dkv_norm"], _rotate(down[:, None, r:], pos, rot, 1000000.0, wide)[:, 0]], dim=1)
    q = torch.cat([torch.einsum("nhd,hdr->nhr", q[..., :d], t["uk"].view(heads, d, r)), q_rot], dim=2)
    out = torch.empty((len(x), heads, r), dtype=torch.float64, device=DEVICE)
    for j, (a, b) in enumerate(cuts):
        all_rows = rows[a:b] if got["past"][j] is None else torch.cat([got["past"][j][0][0][:, 0].double(), rows[a:b]])
        out[a:b] = _attend(q[a:b], all_rows[:, None], all_rows[:, None, :r], pos[a:b], (d + rot) ** -0.5, case["span"], 0, None if wide else t["sink"])
    out = torch.einsum("nhr,hvr->nhv", out, t["uv"].view(heads, v, r))
    gate = torch.sigmoid(x @ t["gate"].T)
    return {"out": (out * (gate.view(len(x), heads, v) if wide else gate[..., None])).flatten(1) @ t["o"].T}


def _exact_experts(case, t, x):
    e, top = case["experts"], case["top"]
    z = x @ t["router"].T
    if case["style"] == "tenetar":
        score = torch.softmax(z, -1)
        pick = score + t["correction"]
        halves = pick.view(len(x), 2, -1)
        keep = halves.amax(-1).argmax(-1)
        pick = halves.masked_fill(torch.arange(2, device=DEVICE)[None, :, None] != keep[:, None, None], -math.inf).flatten(1)
        chosen = pick.topk(top, dim=-1).indices
        weight = score.gather(1, chosen)
    else:
        value, chosen = (z + t["correction"]).topk(top, dim=-1)
        weight = torch.softmax(value, -1)
    out = torch.zeros_like(x)
    for i in range(e):
        row, slot = (chosen == i).nonzero(as_tuple=True)
        u = x[row]
        if case["style"] == "tenetar":
            y = torch.relu(u @ t["e%d.up" % i].T) ** 2
        else:
            y = torch.nn.functional.silu(u @ t["e%d.gate" % i].T) * (u @ t["e%d.up" % i].T)
        out.index_add_(0, row, y @ t["e%d.down" % i].T * weight[row, slot][:, None])
    if case["style"] == "tenetar":
        out += x * (weight * (chosen >= e)).sum(-1, keepdim=True)
        out += torch.sigmoid(x @ t["shared.gate"].T) * (torch.relu(x @ t["shared.up"].T) ** 2 @ t["shared.down"].T)
    return {"out": out}


def _walk(cuts, step):
    """Calls step(sequences, rows) for the first token of every sequence, then the second of those that have one, and so on."""
    for i in range(max(b - a for a, b in cuts)):
        live = [j for j, (a, b) in enumerate(cuts) if a + i < b]
        step(slice(None) if len(live) == len(cuts) else torch.tensor(live, device=DEVICE), torch.tensor([cuts[j][0] + i for j in live], device=DEVICE))


def _conv(x, taps, before, cuts):
    """Causal convolution of every channel, then silu; before[j]: the rows ahead of sequence j's first, oldest first."""
    out = torch.empty_like(x)
    for j, (a, b) in enumerate(cuts):
        ext = torch.cat([before[j], x[a:b]])
        out[a:b] = sum(ext[i:i + b - a] * taps[:, i] for i in range(taps.shape[1]))
    return out


def _exact_wkv(case, t, x, state, cuts):
    heads, d = _heads(case)[0], case["head_dim"]
    n = heads * d * d
    before = torch.empty_like(x)
    for j, (a, b) in enumerate(cuts):
        before[a], before[a + 1:b] = state[j, n:], x[a:b - 1]
    mix = {s: x + (before - x) * t["mu." + s] for s in "rkvgw"}
    r, k, v = ((mix[s] @ t[s].T).view(len(x), heads, d) for s in "rkv")
    w = torch.exp(-torch.exp(torch.tanh(mix["w"] @ t["w1"].T) @ t["w2"].T + t["w0"])).view(len(x), heads, d)
    S, out = state[:, :n].view(-1, heads, d, d).clone(), torch.empty_like(v)

    def step(live, at):
        kv = k[at][..., None] * v[at][:, :, None]
        out[at] = (r[at][:, :, None] @ (S[live] + t["u"][..., None] * kv))[:, :, 0]
        S[live] = S[live] * w[at][..., None] + kv

    _walk(cuts, step)
    o = _rms(out).flatten(1) * t["norm"] * torch.nn.functional.silu(mix["g"] @ t["g"].T)
    return {"out": o @ t["o"].T, "state": torch.cat([S.flatten(1), torch.stack([x[b - 1] for _, b in cuts])], dim=1)}


def _exact_ssm(case, t, x, state, cuts):
    i, s = 2 * x.shape[1], case["states"]
    r = x.shape[1] // 16
    u, z = (x @ t["in"].T).split(i, dim=1)
    before = state[:, i * s:].view(-1, 3, i)
    kept = torch.stack([torch.cat([before[j], u[a:b]])[-3:] for j, (a, b) in enumerate(cuts)])
    u = torch.nn.functional.silu(_conv(u, t["conv"], before, cuts) + t["conv_bias"])
    low, B, C = (u @ t["x"].T).split([r, s, s], dim=1)
    dt = torch.nn.functional.softplus(low @ t["dt"].T + t["dt_bias"])
    A, S, y = -torch.exp(t["A_log"]), state[:, :i * s].view(-1, i, s).clone(), torch.empty_like(u)

    def step(live, at):
        S[live] = S[live] * torch.exp(dt[at][..., None] * A) + (dt[at] * u[at])[..., None] * B[at][:, None]
        y[at] = (S[live] @ C[at][..., None])[..., 0]

    _walk(cuts, step)
    y = (y + t["D"] * u) * torch.nn.functional.silu(z)
    return {"out": y @ t["o"].T, "state": torch.cat([S.flatten(1), kept.flatten(1)], dim=1)}


def _exact_gated(case, t, x, state, cuts):
    heads, d, v = _heads(case)[0], case["head_dim"], case["v_dim"]
    q = torch.nn.functional.silu(x @ t["q"].T).view(-1, heads, d)
    z = x @ t["f"].T + t["f_bias"]
    k = ((1 - t["lower"]) * torch.sigmoid(-z)).view(-1, heads, d)
    val = (x @ t["v"].T).view(-1, heads, v)
    S, out = state.view(-1, heads, v, d).clone(), torch.empty_like(val)

    def step(live, at):
        S[live] = S[live] * (1 - k[at])[:, :, None] + val[at][..., None] * k[at][:, :, None]
        out[at] = (S[live] @ q[at][..., None])[..., 0]

    _walk(cuts, step)
    return {"out": (_rms(out) * t["norm"]).flatten(1) @ t["o"].T, "state": S.flatten(1)}


def _exact_delta(case, t, x, state, cuts):
    (heads, groups), d, v = _heads(case), case["head_dim"], case["v_dim"]
    n = heads * v * d
    raw = torch.cat([x @ t[s].T for s in "qkv"], dim=1)
    starts, ring = _starts(case), state[:, n:].view(len(cuts), 4, -1).clone()
    before = torch.stack([torch.stack([ring[j, (p - i) % 4] * (p >= i) for i in (3, 2, 1)]) for j, p in enumerate(starts)])
    for j, (a, b) in enumerate(cuts):
        for i in range(max(a, b - 4), b):
            ring[j, (starts[j] + i - a) % 4] = raw[i]
    y = torch.nn.functional.silu(_conv(raw, torch.cat([t[s + "_conv"] for s in "qkv"]), before, cuts))
    q, k, val = (u.view(len(x), -1, m) for u, m in zip(y.split([groups * d, groups * d, heads * v], dim=1), (d, d, v)))
    q, k = (u / torch.sqrt((u * u).sum(-1, keepdim=True) + 1e-6) for u in (q, k))
    q, k = (u.repeat_interleave(heads // groups, dim=1) for u in (q * d ** -0.5, k))
    beta = torch.sigmoid(x @ t["b"].T)
    g = torch.exp(-torch.exp(t["A_log"]) * torch.nn.functional.softplus(x @ t["a"].T + t["dt_bias"]))
    S, out = state[:, :n].view(-1, heads, v, d).clone(), torch.empty_like(val)

    def step(live, at):
        now = S[live] * g[at][..., None, None]
        u = beta[at][..., None] * (val[at] - (now @ k[at][..., None])[..., 0])
        S[live] = now + u[..., None] * k[at][:, :, None]
        out[at] = (S[live] @ q[at][..., None])[..., 0]

    _walk(cuts, step)
    o = (_rms(out) * t["norm"]).flatten(1) * torch.nn.functional.silu(x @ t["g"].T)
    whole = torch.cat([S.flatten(1), ring.flatten(1)], dim=1)
    return {"out": o @ t["o"].T, "state": whole}


def exact(case, seed):
    got = _inputs(case, seed)
    if case["kind"] in ("step", "prompts"):
        return _exact_qwen3(case, got)
    t, x = {n: v.double() for n, v in got["tensors"].items()}, got["x"].double()
    if case["kind"] == "experts":
        return _exact_experts(case, t, x)
    lens, starts = _lengths(case), _starts(case)
    first = np.concatenate([[0], np.cumsum(lens)]).tolist()
    cuts = list(zip(first[:-1], first[1:]))
    if case["kind"] in RECURRENT:
        return {"wkv": _exact_wkv, "ssm": _exact_ssm, "gated": _exact_gated, "delta": _exact_delta}[case["kind"]](case, t, x, got["state"].double(), cuts)
    pos = torch.cat([torch.arange(s, s + n, device=DEVICE) for s, n in zip(starts, lens)])
    return (_exact_masked if case["kind"] == "masked" else _exact_latent)(case, t, x, got, pos, cuts)
