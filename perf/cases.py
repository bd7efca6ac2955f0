"""The calls that a user of this package makes, at the sizes at which they are made: decode steps through the packed
cache (call by call and inside a captured graph), the operators, the bulk encoders and the prefill attention.

Data.  Keys are N(0,1) times a lognormal(0,1) scale per RoPE block with two blocks eight times larger (the rotary
embedding turns each block's pair of equal-scale Gaussians within itself, so it is left out: the distribution is the
same), values and queries N(0,1), all fp16.  The scales and the quantiser tables calibrated on them stand for the
model: they are the same for every seed, each layer and KV head has its own, and a program calibrates them once.
Keys, values, queries and rotary angles come from the seed."""
import math

import torch

from blockgtq_b200 import BlockGTQKVManager, BlockGTQProductionCache, fused_blockgtq_decode_attention
from blockgtq_b200 import fused_blockgtq_prefill_attention
from blockgtq_b200.layer import encode, prefill_attention, rotate_q_bulk
from blockgtq_b200.quantizer import (BlockGTQQuantizer, build_batched_encode_args, compress_k_mixed_batched,
                                     compress_k_packed_batched, compress_v_nibble4_batched, compress_v_packed_batched)

HD = 128
DEV = "cuda:0"


# -- the cases ----------------------------------------------------------------------------------------------------

def _step(name, mode, layers, batch, n_q, n_kv, ctx, k_bits, v_bits, sink=0, window=0):
    return dict(name=name, kind="step", mode=mode, layers=layers, batch=batch, n_q=n_q, n_kv=n_kv, ctx=ctx,
                k_bits=k_bits, v_bits=v_bits, sink=sink, window=window)


def listed():
    return [
        # the first tokens of a chat: one short sequence, every layer called from Python; launches and host time
        _step("step_b1_t500", "call", 4, 1, 32, 8, 500, 3.0, 3),
        # one very long sequence on one GPU, called layer by layer
        _step("step_b1_t131072_k2v2", "call", 2, 1, 32, 8, 131072, 2.0, 2),
        # a serving engine's step (all layers in one captured graph): few KV heads, wide query groups, long context
        _step("graph_b8_t32768_k3v3", "graph", 4, 8, 16, 2, 32768, 3.0, 3),
        # the same for a large batch with the fp16 sink and recent window
        _step("graph_b32_t16384_k2v2_win128", "graph", 2, 32, 32, 8, 16384, 2.0, 2, 4, 128),
        # the production cache (nibble/raw keys, nibble values), rotary embedding applied by the step, a length just
        # past a multiple of every tile and a query group that is no power of two
        _step("production_b4_t4099", "production", 3, 4, 24, 8, 4099, 4.0, 3),
        # one rank's share of a sequence that is cut across GPUs: attention over a token range, fp32 output and LSE
        dict(name="attend_chunk_t16384", kind="attend", batch=1, n_q=32, n_kv=8, ctx=20000, lo=3616, hi=20000,
             k_bits=2.0, v_bits=2),
        # the decode operator as a program of the reference calls it: per KV head
        dict(name="op_decode_b2_t2047", kind="op", batch=2, gqa=4, heads=2, ctx=2047, k_bits=3.0, v_bits=3),
        # prompts taken over from a model's fp16 cache: a short one in a few layers, a large batch in one
        dict(name="encode_b1_t777", kind="encode", layers=4, batch=1, n_kv=8, n_q=32, tokens=777, k_bits=3.0, v_bits=3),
        dict(name="encode_b4_t32768", kind="encode", layers=1, batch=4, n_kv=8, n_q=32, tokens=32768, k_bits=3.0, v_bits=3),
        # the batched encode operators in the production cache's layout
        dict(name="compress_mixed_t4500", kind="compress", mixed=True, n_kv=8, rows=4500, k_bits=3.0, v_bits=3),
        # layer-major prefill of one layer: encode the prompt's keys and values, rotate its queries, attend
        dict(name="prefill_t16384", kind="prefill", entry="layer", batch=1, n_q=32, n_kv=8, queries=16384, cached=0,
             k_bits=3.0, v_bits=3),
        # a further piece of a conversation prefilled behind a cached context, wide query groups, ragged sizes
        dict(name="prefill_q700_t9100", kind="prefill", entry="layer", batch=1, n_q=16, n_kv=2, queries=700, cached=8400,
             k_bits=3.0, v_bits=3),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["step", "attend", "op", "encode", "compress", "prefill"], [42, 8, 8, 16, 8, 18])[0]
    k_bits, v_bits = rng.choice([2.0, 2.5, 3.0, 3.5, 4.0]), rng.choice([2, 3, 3, 4])
    n_kv = rng.choice([1, 2, 4, 8, 8])
    gqa = rng.choice([1, 2, 3, 4, 4, 5, 6, 7, 8])
    if kind == "step":
        mode = rng.choice(["call", "call", "graph", "graph", "production"])
        layers = rng.randint(2, 4)
        batch = _log(rng, 1, 32)
        # no more packed bytes in a pass than the largest listed step reads
        ctx = _log(rng, 64, min(131072, 32 * 16384 * 8 * 2 / (batch * n_kv * layers * (2 if k_bits > 2.5 else 1))))
        sink, window = (4, 128) if mode != "production" and rng.random() < 0.3 else (0, 0)
        return dict(kind="step", mode=mode, layers=layers, batch=batch, n_q=gqa * n_kv, n_kv=n_kv, ctx=ctx, k_bits=k_bits,
                    v_bits=v_bits, sink=sink, window=window)
    if kind == "attend":
        ctx = _log(rng, 500, 65536)
        lo = rng.randint(0, ctx // 4)
        return dict(kind="attend", batch=_log(rng, 1, 8), n_q=gqa * n_kv, n_kv=n_kv, ctx=ctx, lo=lo, hi=ctx - rng.randint(0, ctx // 8),
                    k_bits=k_bits, v_bits=v_bits)
    if kind == "op":
        return dict(kind="op", batch=_log(rng, 1, 8), gqa=gqa, heads=rng.randint(1, 4), ctx=_log(rng, 200, 32768), k_bits=k_bits,
                    v_bits=v_bits)
    if kind == "encode":
        batch = _log(rng, 1, 8)
        layers = rng.randint(1, 4)
        tokens = _log(rng, 17, 4 * 32768 / (batch * layers))
        return dict(kind="encode", layers=layers, batch=batch, n_kv=n_kv, n_q=gqa * n_kv, tokens=tokens, k_bits=k_bits, v_bits=v_bits)
    if kind == "compress":
        return dict(kind="compress", mixed=rng.random() < 0.5, n_kv=n_kv, rows=_log(rng, 30, 65536), k_bits=k_bits, v_bits=v_bits)
    entry = rng.choice(["layer", "layer", "operator"])
    if entry == "operator":
        n_kv = 1
    queries = _log(rng, 48, 16384)
    cached = 0 if rng.random() < 0.5 else _log(rng, 500, 32768)
    batch = rng.choice([1, 1, 2])
    # no more query-key pairs than the largest listed prefill
    most = 32 * 16384 * 16384 / 2
    while batch * gqa * n_kv * queries * (cached + queries / 2) > most:
        queries = queries * 2 // 3
    return dict(kind="prefill", entry=entry, batch=batch, n_q=gqa * n_kv, n_kv=n_kv, queries=queries, cached=cached, k_bits=k_bits,
                v_bits=v_bits)


# -- the model: block scales and calibrated tables, made once per configuration -------------------------------------

_models = {}


def _model(layers, n_kv, k_bits, v_bits):
    """Per layer: block scales (n_kv, 128) and the calibrated quantisers of its KV heads."""
    key = (layers, n_kv, k_bits, v_bits)
    if key not in _models:
        gen = torch.Generator().manual_seed(20 + n_kv)
        out = []
        for _ in range(layers):
            scales, quants = [], []
            for h in range(n_kv):
                s = torch.exp(torch.randn(HD // 2, generator=gen))
                s[torch.randperm(HD // 2, generator=gen)[:2]] *= 8
                s = torch.cat([s, s])
                qz = BlockGTQQuantizer(HD, avg_bits=k_bits, device=torch.device(DEV))
                qz.calibrate(torch.randn(512, HD, generator=gen), torch.randn(1024, HD, generator=gen) * s)
                qz.init_v_quantizer(v_bits=v_bits, seed=42 + h)
                scales.append(s)
                quants.append(qz)
            out.append((torch.stack(scales).to(DEV), quants))
        _models[key] = out
    return _models[key]


def _randn(gen, *shape):
    return torch.randn(*shape, generator=gen, device=DEV, dtype=torch.float16)


def _keys(gen, scales, batch, n_tok):
    return _randn(gen, batch, scales.shape[0], n_tok, HD) * scales.to(torch.float16)[None, :, None, :]


def _heads(gen, batch, heads, scales=None):
    """(batch, heads, 1, 128) as a projection's output gives it: the heads of a token side by side."""
    x = _randn(gen, batch, 1, heads, HD)
    if scales is not None:
        x = x * scales.to(torch.float16)[None, None]
    return x.transpose(1, 2)


def _k_bytes(qz, mixed=False):
    pm = qz.pack_meta
    return pm["nopack_start"] // 2 + pm["nopack_len"] if mixed else pm["total_packed_bytes"]


def _token_bytes(quants, v_bits, mixed=False):
    """Packed bytes of one token over the KV heads: keys, one fp16 norm per width group, values, one fp16 norm."""
    return sum(_k_bytes(q, mixed) + 2 * q._n_groups + (64 if mixed else 16 * v_bits) + 2 for q in quants)


# -- prepare ----------------------------------------------------------------------------------------------------

def prepare(case, seed):
    gen = torch.Generator(device=DEV).manual_seed(seed)
    return {"step": _prepare_step, "attend": _prepare_attend, "op": _prepare_op, "encode": _prepare_encode,
            "compress": _prepare_compress, "prefill": _prepare_prefill}[case["kind"]](case, gen)


def _manager(case, model, max_len):
    mgr = BlockGTQKVManager(len(model), case["n_q"], case["n_kv"], HD, max_seq_len=max_len, batch_size=case["batch"],
                            k_avg_bits=case["k_bits"], v_bits=case["v_bits"], device=DEV, n_sink=case.get("sink", 0),
                            recent_window=case.get("window", 0))
    for li, (_, quants) in enumerate(model):
        mgr.set_quantizers(li, quants)
    return mgr


class _Prompt:
    """A model's fp16 cache, a layer's keys and values made when they are asked for."""

    def __init__(self, gen, model, batch, n_tok):
        self.gen, self.model, self.batch, self.n_tok = gen, model, batch, n_tok

    def __getitem__(self, li):
        scales = self.model[li][0]
        return (_keys(self.gen, scales, self.batch, self.n_tok),
                _randn(self.gen, self.batch, scales.shape[0], self.n_tok, HD))


class _Pairs:
    """The same for a sequence of (k, v) pairs of which each layer's is read twice."""

    def __init__(self, prompt):
        self.prompt, self.li, self.kv = prompt, None, None

    def __getitem__(self, li):
        if self.li != li:
            self.li, self.kv = li, self.prompt[li]
        return self.kv


def _prepare_step(case, gen):
    L, B, n_q, n_kv, T = case["layers"], case["batch"], case["n_q"], case["n_kv"], case["ctx"]
    model = _model(L, n_kv, case["k_bits"], case["v_bits"])
    prompt = _Pairs(_Prompt(gen, model, B, T))
    rope = None
    if case["mode"] == "production":
        quants = [q for _, q in model]
        obj = BlockGTQProductionCache(quants, [build_batched_encode_args(q, device=DEV) for q in quants],
                                      [[q.build_kernel_args() for q in row] for row in quants], L, n_kv, n_q, HD, T + 16,
                                      v_bits=case["v_bits"], device=DEV, batch_size=B)
        for li in range(L):
            k, v = prompt[li]
            obj._encode_batched(li, k, v, 0)
        obj.seq_len = T
        mgr, packed = obj._mgr, (obj.k_packed, obj.k_norms, obj.v_packed, obj.v_norms)
        ang = torch.rand(B, 1, HD // 2, generator=gen, device=DEV) * 2 * math.pi
        ang = torch.cat([ang, ang], dim=-1)
        rope = (ang.cos().half(), ang.sin().half())
    else:
        obj = mgr = _manager(case, model, T + 16)
        mgr.init_from_cache(prompt)
        packed = (mgr._k_packed, mgr._k_norms, mgr._v_packed, mgr._v_norms)
    # the row that the step appends to the packed cache (with an fp16 window: the token that leaves the window), and
    # the fp16 row of the new token
    row = T if not case["window"] else T - case["sink"] - case["window"]
    state = [t[li][:, :, row] for li in range(L) for t in packed if row >= 0]
    if case["window"]:
        slot = T if T < case["sink"] else case["sink"] + (T - case["sink"]) % (case["window"] + 1)
        state += [b[li][:, :, slot] for li in range(L) for b in (mgr._k_buf, mgr._v_buf)]
    qkv = [(_heads(gen, B, n_q), _heads(gen, B, n_kv, model[li][0]), _heads(gen, B, n_kv)) for li in range(L)]
    graph = None
    if case["mode"] == "graph":
        for li, parts in enumerate(qkv):
            for dst, src in zip(mgr.static_inputs(li), parts):
                dst.copy_(src)
            mgr.layer_step(li)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            for li in range(L):
                mgr.layer_step(li)
        state.append(mgr.static_outputs())
    return dict(kind="step", mode=case["mode"], obj=obj, mgr=mgr, qkv=qkv, rope=rope, graph=graph, state=state)


def _prepare_attend(case, gen):
    model = _model(1, case["n_kv"], case["k_bits"], case["v_bits"])
    mgr = _manager(case, model, case["ctx"])
    mgr.init_from_cache(_Pairs(_Prompt(gen, model, case["batch"], case["ctx"])))
    return dict(kind="attend", mgr=mgr, q=_heads(gen, case["batch"], case["n_q"]), rng=(case["lo"], case["hi"]))


def _prepare_op(case, gen):
    B, T, gqa = case["batch"], case["ctx"], case["gqa"]
    (scales, quants), = _model(1, 4, case["k_bits"], case["v_bits"])
    q = _randn(gen, B, case["heads"] * gqa, 1, HD)
    calls = []
    for h in range(case["heads"]):
        qz = quants[h]
        ka = qz.build_kernel_args()
        kp, kn, _ = qz.compress_packed(_keys(gen, scales[h:h + 1], B, T))
        vp, vn = qz.compress_v_packed(_randn(gen, B, 1, T, HD))
        calls.append((qz.rotate_q_for_packed_kernel(q[:, h * gqa:(h + 1) * gqa]), kp, kn.half(), ka["codebook_flat"],
                      ka["lut_offset"], ka["norm_group"], ka["segments_b"], vp, vn, qz.v_lut, qz._v_rot))
    return dict(kind="op", calls=calls, v_bits=case["v_bits"])


def _prepare_encode(case, gen):
    model = _model(case["layers"], case["n_kv"], case["k_bits"], case["v_bits"])
    mgr = _manager(case, model, case["tokens"] + 16)
    prompt = _Prompt(gen, model, case["batch"], case["tokens"])
    mgr.static_qkv()                            # the cache exists before the first prompt arrives
    return dict(kind="encode", mgr=mgr, kv=[prompt[li] for li in range(case["layers"])], n=case["tokens"])


def _prepare_compress(case, gen):
    (scales, quants), = _model(1, case["n_kv"], case["k_bits"], case["v_bits"])
    return dict(kind="compress", mixed=case["mixed"], args=build_batched_encode_args(quants, device=DEV),
                k=_keys(gen, scales, 1, case["rows"])[0], v=_randn(gen, case["n_kv"], case["rows"], HD))


def _prepare_prefill(case, gen):
    B, n_q, n_kv, S, C = case["batch"], case["n_q"], case["n_kv"], case["queries"], case["cached"]
    T = C + S
    model = _model(1, max(n_kv, 2) if case["entry"] == "operator" else n_kv, case["k_bits"], case["v_bits"])
    scales, quants = model[0]
    q = _randn(gen, B, S, n_q, HD).transpose(1, 2)
    if case["entry"] == "operator":             # one KV head, its cache encoded by the single-head operators
        qz = quants[1]
        ka = qz.build_kernel_args()
        kp, kn, _ = qz.compress_packed(_keys(gen, scales[1:2], B, T))
        vp, vn = qz.compress_v_packed(_randn(gen, B, 1, T, HD))
        call = (qz.rotate_q_for_packed_kernel(q.contiguous()), kp, kn.half(), ka["codebook_flat"], ka["lut_offset"],
                ka["norm_group"], ka["segments_b"], vp, vn, qz.v_lut, qz._v_rot)
        return dict(kind="prefill", entry="operator", call=call, v_bits=case["v_bits"], offset=C)
    mgr = _manager(case, model, T)
    k, v = _Prompt(gen, model, B, T)[0]
    mgr.init_from_cache([(k, v)])
    return dict(kind="prefill", entry="layer", mgr=mgr, layer=mgr._layers[0], q=q, k=k[:, :, C:], v=v[:, :, C:], n=T, offset=C,
                cache=(mgr._k_packed[0], mgr._k_norms[0], mgr._v_packed[0], mgr._v_norms[0]))


# -- run ----------------------------------------------------------------------------------------------------------

def run(s):
    kind = s["kind"]
    if kind == "step":
        # The step of one position, over and over: a program calls increment_seq_len once behind all its layers.
        if s["graph"] is not None:
            s["graph"].replay()
            return s["state"]
        if s["rope"] is not None:
            outs = [s["obj"].encode_and_attend(li, q, k, v, rope=s["rope"]) for li, (q, k, v) in enumerate(s["qkv"])]
        else:
            outs = [s["obj"].append_and_attend(li, q, k, v) for li, (q, k, v) in enumerate(s["qkv"])]
        return outs + s["state"]
    if kind == "attend":
        return s["mgr"].attend(0, s["q"], token_range=s["rng"], want_partial=True)
    if kind == "op":
        return [fused_blockgtq_decode_attention(q, kp, kn, cb, lo, ng, segs, vp, vn, lut, v_bits=s["v_bits"], v_rotation=rot,
                                                return_lse=True)
                for q, kp, kn, cb, lo, ng, segs, vp, vn, lut, rot in s["calls"]]
    if kind == "encode":
        m, n = s["mgr"], s["n"]
        m.init_from_cache(s["kv"])
        return [t[:, :, :, :n] for t in (m._k_packed, m._k_norms, m._v_packed, m._v_norms)]
    if kind == "compress":
        if s["mixed"]:
            return compress_k_mixed_batched(s["k"], s["args"]) + compress_v_nibble4_batched(s["v"], s["args"])
        return compress_k_packed_batched(s["k"], s["args"]) + compress_v_packed_batched(s["v"], s["args"])
    if s["entry"] == "operator":
        q, kp, kn, cb, lo, ng, segs, vp, vn, lut, rot = s["call"]
        return fused_blockgtq_prefill_attention(q, kp, kn, cb, lo, ng, segs, vp, vn, lut, v_bits=s["v_bits"], v_rotation=rot,
                                                q_pos_offset=s["offset"])
    lt, cache = s["layer"], s["cache"]
    encode(lt, s["k"], s["v"], s["offset"], *cache, flags=s["mgr"]._enc_flags)
    return prefill_attention(lt, rotate_q_bulk(lt, s["q"]), *cache, s["n"], q_pos_offset=s["offset"], v_rot=lt.v_rot)


# -- what a pass cannot do without ----------------------------------------------------------------------------------

def work(case):
    kind, v_bits = case["kind"], case["v_bits"]
    if kind == "step":
        B, T, n_q, n_kv = case["batch"], case["ctx"], case["n_q"], case["n_kv"]
        model = _model(case["layers"], n_kv, case["k_bits"], v_bits)
        packed, fp16 = T + 1, 0
        if case["window"]:
            packed = max(0, T - case["sink"] - case["window"])
            fp16 = T + 1 - packed
        nbytes = sum(B * packed * _token_bytes(q, v_bits, case["mode"] == "production") for _, q in model)
        nbytes += case["layers"] * B * HD * 2 * (2 * fp16 * n_kv + 2 * n_q + 2 * n_kv)      # fp16 region; q, out, k, v
        return {"bytes": nbytes, "flops": case["layers"] * 4.0 * B * n_q * HD * (T + 1)}
    if kind == "attend":
        B, n_q, n = case["batch"], case["n_q"], case["hi"] - case["lo"]
        (_, quants), = _model(1, case["n_kv"], case["k_bits"], v_bits)
        return {"bytes": B * n * _token_bytes(quants, v_bits) + B * n_q * (HD * 8 + 4), "flops": 4.0 * B * n_q * HD * n}
    if kind == "op":
        B, T = case["batch"], case["ctx"]
        (_, quants), = _model(1, 4, case["k_bits"], v_bits)
        rows = B * case["gqa"] * case["heads"]
        return {"bytes": B * T * _token_bytes(quants[:case["heads"]], v_bits) + rows * (HD * 4 + 4), "flops": 4.0 * rows * HD * T}
    if kind in ("encode", "compress"):
        layers, rows = (case["layers"], case["batch"] * case["tokens"]) if kind == "encode" else (1, case["rows"])
        model = _model(layers, case["n_kv"], case["k_bits"], v_bits)
        per = sum(_token_bytes(q, v_bits, case.get("mixed", False)) for _, q in model)
        if kind == "compress":
            per += sum(2 * q._n_groups for q in model[0][1])                                # fp32 key norms
        return {"bytes": rows * (layers * case["n_kv"] * HD * 4 + per), "flops": rows * layers * case["n_kv"] * 4.0 * HD * HD}
    B, n_q, n_kv, S, C = case["batch"], case["n_q"], case["n_kv"], case["queries"], case["cached"]
    operator = case["entry"] == "operator"
    model = _model(1, 2 if operator else n_kv, case["k_bits"], v_bits)
    quants = model[0][1][1:2] if operator else model[0][1]
    nbytes = B * n_q * S * HD * 4 + B * (C + S) * _token_bytes(quants, v_bits)
    flops = 4.0 * B * n_q * HD * (S * C + S * (S + 1) / 2) + B * n_q * S * 2.0 * HD * HD
    if not operator:
        nbytes += B * S * n_kv * HD * 4
        flops += B * S * (n_kv * 4.0 + n_q * 2.0) * HD * HD
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """Attention: fp16 queries, probabilities and outputs, sums in fp32.  Encoded bytes: a coordinate within the
    rounding of a bin's edge may take either code."""
    if case["kind"] in ("encode", "compress"):
        return {"rel": 1e-3, "differ": 1e-3}
    return {"rel": 2e-3, "max": 2e-2, "differ": 1e-3}
