"""Decodes whose clusters merge their shares in the launch, against the split form with its merge launch.

Both round p * norm to fp16 relative to running maxima that other groups of tokens give: each weight may differ by 2^-11 of itself
on either side, so a row by 2^-10 of its largest value; the log-sum-exp sums fp32 weights."""
import random

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _manager(batch, n_kv, gqa, cap, gen, **kw):
    from blockgtq_b200 import BlockGTQKVManager
    from helpers import HD, synth_head
    mgr = BlockGTQKVManager(1, n_kv * gqa, n_kv, HD, max_seq_len=cap, batch_size=batch, device=DEV, **kw)
    cal = [synth_head(gen, 256, gqa) for _ in range(n_kv)]
    mgr.calibrate(0, torch.stack([c[0] for c in cal]).float(), torch.stack([c[1] for c in cal]).float())
    return mgr


def _rand(gen, *shape):
    return torch.randn(*shape, generator=gen).half().to(DEV)


# clusters of 8, 4 and 2; query groups of one, an odd number and eight; both cache layouts
@pytest.mark.parametrize("batch,n_kv,gqa,cap,k_bits,v_bits,mixed,c", [
    (1, 2, 4, 2100, 3.0, 3, False, 8), (2, 7, 1, 1100, 2.0, 2, False, 8), (1, 8, 7, 510, 4.0, 4, False, 4), (4, 8, 3, 1030, 3.0, 1, False, 4),
    (9, 8, 8, 300, 2.5, 3, False, 2), (1, 4, 5, 90, 3.5, 2, False, 2), (3, 8, 2, 1500, 4.0, 3, True, 4)])
def test_merged_in_the_launch(batch, n_kv, gqa, cap, k_bits, v_bits, mixed, c):
    from blockgtq_b200 import _lib
    from blockgtq_b200.layer import attend, merges
    gen = torch.Generator().manual_seed(cap)
    mgr = _manager(batch, n_kv, gqa, cap, gen, k_avg_bits=k_bits, v_bits=v_bits, k_mixed=mixed, v_nibble=mixed)
    mgr.init_from_cache([tuple(_rand(gen, batch, n_kv, cap, 128) for _ in range(2))])
    assert mgr._cluster_flags >> _lib.DEC_CLUSTER_SHIFT == c
    lt, cache = mgr._layers[0], (mgr._k_packed[0], mgr._k_norms[0], mgr._v_packed[0], mgr._v_norms[0])
    plain, flags = mgr._dec_flags, mgr._dec_flags | mgr._cluster_flags
    assert merges(lt, flags | _lib.DEC_PROGRAMMATIC) and not merges(lt, plain | _lib.DEC_PROGRAMMATIC)
    q = _rand(gen, batch, n_kv * gqa, 128)
    odd = torch.empty(lt.v_rot.numel() + 1, device=DEV)[1:].view_as(lt.v_rot).copy_(lt.v_rot)       # off its 16-byte boundary
    top = float((mgr._v_norms[0].float().max() * max(t.centroids.abs().max() for t in lt.v_tables)).item())
    tile = 256 * c
    for lo, hi, rot in ((0, 0, lt.v_rot), (0, 1, lt.v_rot), (0, 15, None), (0, 16, odd), (0, 17, lt.v_rot), (16, 16 * c + 1, lt.v_rot),
                        (0, min(cap, tile), None), (0, min(cap, tile + 1), odd), (64, cap, lt.v_rot), (0, cap, lt.v_rot)):
        args = dict(rotate=True, v_rot=rot, want_f32=True, want_lse=True, status=mgr._status)
        out, o32, lse = attend(lt, q, *cache, lo, hi, flags=flags, **args)
        want, w32, wlse = attend(lt, q, *cache, lo, hi, flags=plain, **args)
        assert torch.equal(out, o32.half()), (lo, hi)
        norm = 1.0 if rot is None else 128 ** 0.5           # a rotation may gather a row's whole difference in one dim
        assert (o32 - w32).abs().max().item() <= 2.0 ** -10 * top * norm, (lo, hi)
        if lo == hi:
            assert not o32.any() and torch.equal(lse, wlse) and torch.isinf(lse).all()
        else:
            assert (lse - wlse).abs().max().item() <= 1e-5 * max(1.0, wlse.abs().max().item()), (lo, hi)
    mgr.check_status()


@pytest.mark.parametrize("batch,n_kv,gqa,start,cap,sink,window", [
    (1, 8, 4, 0, 40, 0, 0), (2, 2, 8, 254, 600, 0, 0), (4, 8, 3, 1020, 1030, 0, 0), (1, 8, 4, 3, 40, 2, 4), (2, 4, 4, 700, 720, 4, 128), (9, 8, 1, 260, 300, 0, 9)])
def test_layer_steps(batch, n_kv, gqa, start, cap, sink, window):
    """A layer's steps call by call and replayed, with and without fp16 regions (a packed region that is still empty among them):
    the same cache bytes as the split form, rows within the bound."""
    gen = torch.Generator().manual_seed(start)
    from blockgtq_b200 import BlockGTQKVManager
    regions = dict(n_sink=sink, recent_window=window)
    a = _manager(batch, n_kv, gqa, cap, gen, **regions)
    b = BlockGTQKVManager(1, n_kv * gqa, n_kv, 128, max_seq_len=cap, batch_size=batch, device=DEV, **regions)
    b.set_quantizers(0, a.quantizers[0])
    for m in (a, b):
        m._ensure_storage()
    assert a._cluster_flags
    b._cluster_flags = 0
    if start:
        kv = tuple(_rand(gen, batch, n_kv, start, 128) for _ in range(2))
        for m in (a, b):
            m.init_from_cache([kv])
    graph = None
    for step in range(6):
        q, k, v = (_rand(gen, batch, n, 1, 128) for n in (n_kv * gqa, n_kv, n_kv))
        want = b.append_and_attend(0, q, k, v).float()
        if step < 3:
            got = a.append_and_attend(0, q, k, v).float()
        else:
            for dst, src in zip(a.static_inputs(0), (q, k, v)):
                dst.copy_(src)
            if graph is None:
                a._sync_pos()
                graph = torch.cuda.CUDAGraph()
                with torch.cuda.graph(graph):
                    a.layer_step(0)
            graph.replay()
            got = a.static_outputs()[0].unsqueeze(2).float()
        for m in (a, b):
            m.increment_seq_len()
        # (an fp16 region's values are at most as large as their norm, which the packed rows' is within a factor of)
        top = max(float(a._v_norms[0].float().max() * max(t.centroids.abs().max() for t in a._layers[0].v_tables)), 2.0) * 128 ** 0.5
        assert (got - want).abs().max().item() <= 2.0 ** -10 * top + 2.0 ** -11 * want.abs().max().item()
        for x, y in zip((a._k_packed, a._k_norms, a._v_packed, a._v_norms, a._k_buf, a._v_buf), (b._k_packed, b._k_norms, b._v_packed, b._v_norms, b._k_buf, b._v_buf)):
            assert x is y is None or torch.equal(x, y)
    # several calls' worth of attention over what is there, with the regions' partial
    out, o32, lse = a.attend(0, q, want_partial=True)
    want, w32, wlse = b.attend(0, q, want_partial=True)
    assert (o32 - w32).abs().max().item() <= 2.0 ** -10 * top and (lse - wlse).abs().max().item() <= 1e-5 * max(1.0, wlse.abs().max().item())
    a.check_status()


def test_rows_too_wide_for_the_merging_form():
    """Packed rows padded until the stages no longer fit beside the shares: the call is left to the split form."""
    from blockgtq_b200 import fused_blockgtq_decode_attention
    from blockgtq_b200.quantizer import BlockGTQQuantizer
    from helpers import HD, synth_head
    gen = torch.Generator().manual_seed(5)
    qz = BlockGTQQuantizer(HD, avg_bits=4.0, device=torch.device(DEV))
    qc, kc = synth_head(gen, 256, 4)
    qz.calibrate(qc.float(), kc.float())
    qz.init_v_quantizer(v_bits=4, seed=42)
    ka, T = qz.build_kernel_args(), 700
    kp, kn, _ = qz.compress_packed(_rand(gen, 1, 1, T, HD))
    vp, vn = qz.compress_v_packed(_rand(gen, 1, 1, T, HD))
    q = qz.rotate_q_for_packed_kernel(_rand(gen, 1, 4, 1, HD))
    kw = torch.zeros(1, 1, T + 8, 160, dtype=torch.uint8, device=DEV)[:, :, :T, :kp.shape[3]]
    kw.copy_(kp)

    def call(k):
        return fused_blockgtq_decode_attention(q, k, kn.half(), ka["codebook_flat"], ka["lut_offset"], ka["norm_group"], ka["segments_b"],
                                               vp, vn, qz.v_lut, v_bits=4, v_rotation=qz._v_rot, return_lse=True)
    (a, al), (b, bl) = call(kp), call(kw)
    top = float(vn.float().max() * qz.v_lut.float().abs().max()) * HD ** 0.5
    assert (a.float() - b.float()).abs().max().item() <= 2.0 ** -10 * top + 2.0 ** -11 * b.float().abs().max().item()
    assert (al - bl).abs().max().item() <= 1e-5 * max(1.0, bl.abs().max().item())


def test_numbers_of_splits_that_are_refused():
    """The merging form has no splits, and takes no number of them that the split form does not take."""
    from blockgtq_b200 import _lib
    from blockgtq_b200.layer import attend, merges
    gen = torch.Generator().manual_seed(4)
    mgr = _manager(1, 2, 4, 300, gen)
    mgr.init_from_cache([tuple(_rand(gen, 1, 2, 300, 128) for _ in range(2))])
    lt, cache = mgr._layers[0], (mgr._k_packed[0], mgr._k_norms[0], mgr._v_packed[0], mgr._v_norms[0])
    flags = mgr._dec_flags | mgr._cluster_flags
    assert merges(lt, flags | _lib.DEC_PROGRAMMATIC)
    q = _rand(gen, 1, 8, 128)
    for n in (0, -1, (1 << 31) - 1):
        with pytest.raises(RuntimeError):
            attend(lt, q, *cache, 0, 300, rotate=False, n_splits=n, flags=flags)
    with pytest.raises(OverflowError):
        attend(lt, q, *cache, 0, 300, rotate=False, n_splits=1 << 31, flags=flags)
    assert torch.equal(*(attend(lt, q, *cache, 0, 300, rotate=False, n_splits=n, flags=flags)[0] for n in (1, 33)))


@pytest.mark.parametrize("batch,n_kv,gqa,cap,c", [(1, 2, 4, 2100, 8), (1, 8, 7, 510, 4), (9, 8, 8, 300, 2)])
def test_scores_that_are_no_numbers(batch, n_kv, gqa, cap, c):
    """A share with such a score counts as empty, and no other one: what is left is the attention over the other shares' tokens.
    Values that are infinite, and rows without any share left, come out as from the split form."""
    from blockgtq_b200.layer import attend
    gen = torch.Generator().manual_seed(cap + 1)
    mgr = _manager(batch, n_kv, gqa, cap, gen)
    mgr.init_from_cache([tuple(_rand(gen, batch, n_kv, cap, 128) for _ in range(2))])
    lt, cache = mgr._layers[0], (mgr._k_packed[0], mgr._k_norms[0], mgr._v_packed[0], mgr._v_norms[0])
    plain, flags = mgr._dec_flags, mgr._dec_flags | mgr._cluster_flags
    q = _rand(gen, batch, n_kv * gqa, 128)
    top = float((mgr._v_norms[0].float().max() * max(t.centroids.abs().max() for t in lt.v_tables)).item())

    def run(fl, lo=0, hi=cap, **kw):
        return attend(lt, q, *cache, lo, hi, flags=fl, **dict(dict(rotate=True, want_f32=True, want_lse=True), **kw))

    tiles, share = (cap + 15) // 16, c // 2
    lo, hi = 16 * (tiles * share // c), min(cap, 16 * (tiles * (share + 1) // c))
    norms, kept = cache[1], cache[1].clone()
    norms[:, :, lo + 1] = float("nan")
    _, got, lse = run(flags)
    (_, a, la), (_, b, lb) = run(plain, 0, lo), run(plain, hi, cap)
    want_lse = torch.logaddexp(la, lb)
    want = a * (la - want_lse).exp()[..., None] + b * (lb - want_lse).exp()[..., None]
    assert (got - want).abs().max().item() <= 2.0 ** -10 * top and (lse - want_lse).abs().max().item() <= 1e-5 * max(1.0, lse.abs().max().item())
    norms.copy_(kept)
    for head in range(n_kv):            # one head without a usable share, the others untouched
        norms[:, head] = float("nan")
        (_, got, lse), (_, want, want_lse) = run(flags, v_rot=lt.v_rot), run(plain, v_rot=lt.v_rot)
        rows = slice(head * gqa, (head + 1) * gqa)
        assert not got[:, rows].any() and not want[:, rows].any() and torch.isneginf(lse[:, rows]).all() and torch.isneginf(want_lse[:, rows]).all()
        assert (got - want).abs().max().item() <= 2.0 ** -10 * top * 128 ** 0.5
        norms.copy_(kept)
    cache[3][:, :, 0] = float("inf")    # (of a token that no share leaves out)
    for rot in (None, lt.v_rot):
        (_, got, lse), (_, want, want_lse) = run(flags, v_rot=rot), run(plain, v_rot=rot)
        assert not got.isfinite().any() and not want.isfinite().any()
        assert (lse - want_lse).abs().max().item() <= 1e-5 * max(1.0, lse.abs().max().item())


def test_the_other_partial_beside_an_empty_range():
    """Partials of any kind, infinities and NaN among them, with no packed tokens: the same rows as from the split form."""
    from blockgtq_b200.layer import attend
    gen = torch.Generator().manual_seed(3)
    mgr = _manager(2, 2, 4, 600, gen)
    mgr.init_from_cache([tuple(_rand(gen, 2, 2, 600, 128) for _ in range(2))])
    lt, cache = mgr._layers[0], (mgr._k_packed[0], mgr._k_norms[0], mgr._v_packed[0], mgr._v_norms[0])
    q, other = _rand(gen, 2, 8, 128), torch.randn(2, 8, 128, generator=gen).to(DEV)
    inf, nan = float("inf"), float("nan")
    lse = torch.tensor([[0.0, 3.5, -200.0, 90.0, -inf, inf, nan, 1.0]] * 2, device=DEV)
    other[0, 7, 5], other[1, 7, 6], other[1, 4, 3] = nan, inf, nan
    for hi in (0, 40):
        got, want = (attend(lt, q, *cache, 0, hi, rotate=True, v_rot=lt.v_rot, buf_o=other, buf_lse=lse, want_f32=True, want_lse=True,
                            flags=mgr._dec_flags | f) for f in (mgr._cluster_flags, 0))
        for g, w in zip(got, want):
            assert torch.equal(g.isnan(), w.isnan()) and torch.equal(g.isinf(), w.isinf())
            if hi == 0:
                assert torch.equal(g.nan_to_num(), w.nan_to_num())


@pytest.mark.parametrize("batch,n_kv,gqa,v_bits,cap", [(1, 8, 8, 3, 3200), (2, 4, 4, 4, 3900)])
def test_attention_past_the_steps_limit(batch, n_kv, gqa, v_bits, cap):
    """A capacity past which captured layers take the split form and attentions, called one by one, still merge: the same rows."""
    from blockgtq_b200 import _lib
    from blockgtq_b200.layer import attend
    gen = torch.Generator().manual_seed(8)
    mgr = _manager(batch, n_kv, gqa, cap, gen, v_bits=v_bits)
    n = cap - 7
    mgr.init_from_cache([tuple(_rand(gen, batch, n_kv, n, 128) for _ in range(2))])
    assert not mgr._cluster_flags and mgr._attend_flags >> _lib.DEC_CLUSTER_SHIFT == 8
    q = _rand(gen, batch, n_kv * gqa, 128)
    lt, cache = mgr._layers[0], (mgr._k_packed[0], mgr._k_norms[0], mgr._v_packed[0], mgr._v_norms[0])
    top = float((mgr._v_norms[0].float().max() * max(t.centroids.abs().max() for t in lt.v_tables)).item())
    for lo, hi in ((0, n), (5, 1700), (40, 40)):
        out, o32, lse = mgr.attend(0, q, token_range=(lo, hi), want_partial=True)
        _, want, want_lse = attend(lt, q, *cache, lo, hi, rotate=True, v_rot=lt.v_rot, want_f32=True, want_lse=True, flags=mgr._dec_flags)
        if hi > lo:
            assert (lse - want_lse).abs().max().item() <= 1e-5 * max(1.0, want_lse.abs().max().item())
        else:
            assert torch.equal(lse, want_lse)
        assert (o32 - want).abs().max().item() <= 2.0 ** -10 * top * 128 ** 0.5
        assert torch.equal(out, o32.half())


def _regions(mgr, n_tok):
    """Sink and packed tokens of a step's attention (a token that leaves the window is packed behind it)."""
    from oracle import bgtq_oracle as O
    return O.three_region_plan(n_tok - 1, mgr.n_sink, mgr.recent_window)[:2] if mgr._buffered else (0, n_tok)


def _step_reference(mgr, q, ks, vs, b, hq, n_tok):
    """A query head's attention in 64 bits over the dequantised packed rows and the fp16 rows: weights and values of all tokens in
    order (packed values in V's rotated space), and V's rotation."""
    import numpy as np
    from helpers import oracle_meta
    from oracle import bgtq_oracle as O
    n_sink, n_packed = _regions(mgr, n_tok)
    h = hq // (mgr.n_q // mgr.n_kv)
    qz = mgr.quantizers[0][h]
    meta = oracle_meta(qz._tables, qz._v_tables)
    q64, k, v = (x.cpu().numpy().astype(np.float64) for x in (q[b, hq, 0], ks[b, h, :n_tok], vs[b, h, :n_tok]))
    lo, hi = n_sink, n_sink + n_packed
    row = lambda t: t[0, b, h, :n_packed].cpu().numpy()
    s = k @ q64
    s[lo:hi] = O.dequant_k(row(mgr._k_packed)[:, :qz._total_packed_bytes], row(mgr._k_norms), meta) @ \
        O.rotate_q(q[b, hq].cpu().numpy(), meta)[0].astype(np.float64)
    v[lo:hi] = O.dequant_v(row(mgr._v_packed), row(mgr._v_norms), meta, f16_product=False)
    return s * mgr.scale, v, slice(lo, hi), meta["v_rot"].astype(np.float64)


def _attend_reference(s, v, packed, rot):
    """Output, and the size of what rounds: each packed weight to fp16 relative to two running maxima, 2^-10 of itself, which the
    rotation may gather in one dim."""
    import numpy as np
    w = np.exp(s - s.max())
    w /= w.sum()
    p = w[packed] @ v[packed]
    rest = np.concatenate([w[:packed.start], w[packed.stop:]]) @ np.concatenate([v[:packed.start], v[packed.stop:]])
    return p @ rot + rest, np.linalg.norm(w[packed] @ np.abs(v[packed]))


@pytest.mark.parametrize("batch,n_kv,gqa,start,cap,sink,window", [
    (1, 8, 4, 0, 40, 0, 0), (2, 2, 8, 254, 600, 0, 0), (4, 8, 3, 1020, 1030, 0, 0), (1, 8, 4, 3, 40, 2, 4), (2, 4, 4, 700, 720, 4, 128), (9, 8, 1, 260, 300, 0, 9)])
def test_layer_steps_weigh_single_rows(batch, n_kv, gqa, start, cap, sink, window):
    """Queries that single rows decide: the one just appended, the first and last of a CTA's share, the oldest, one of the fp16 window,
    and two such rows against each other.  Without the row, or with its weight a few percent off, the output is off by many
    times the bound; the reference says so itself."""
    import numpy as np
    from blockgtq_b200 import _lib
    gen = torch.Generator().manual_seed(start + 1)
    mgr = _manager(batch, n_kv, gqa, cap, gen, n_sink=sink, recent_window=window)
    mgr._ensure_storage()
    c = mgr._cluster_flags >> _lib.DEC_CLUSTER_SHIFT
    assert c
    ks, vs = (torch.randn(batch, n_kv, cap, 128, generator=gen).half() for _ in range(2))
    if start:
        mgr.init_from_cache([(ks[:, :, :start].to(DEV), vs[:, :, :start].to(DEV))])
    graph, single, shared, rng = None, 0, 0, random.Random(start)
    for step in range(6):
        n_tok = start + step + 1
        packed0, n_packed = _regions(mgr, n_tok)
        tiles = (n_packed + 15) // 16
        cuts = [16 * (tiles * r // c) for r in range(1, c)]
        rows = [n_tok - 1] + ([packed0 + n_packed - 1, packed0] if n_packed else []) + ([n_tok - window, n_tok - window // 2 - 1] if window else [])
        rows += [packed0 + t for cut in cuts for t in (cut - 1, cut) if 0 <= t < n_packed]
        rows = sorted(set(rows))
        q = torch.empty(batch, n_kv * gqa, 1, 128, dtype=torch.float16)
        decisive = {}
        for b in range(batch):
            for hq in range(n_kv * gqa):
                pick = rng.sample(rows, min(len(rows), rng.randint(1, 2)))
                decisive[b, hq] = pick
                q[b, hq, 0] = sum(14.0 * 128 ** 0.5 * ks[b, hq // gqa, t].float() / ks[b, hq // gqa, t].float().square().sum() for t in pick).half()
        args = [q.to(DEV)] + [x[:, :, n_tok - 1:n_tok].to(DEV) for x in (ks, vs)]
        if step < 3:
            got = mgr.append_and_attend(0, *args)
        else:
            for dst, src in zip(mgr.static_inputs(0), args):
                dst.copy_(src)
            if graph is None:
                mgr._sync_pos()
                graph = torch.cuda.CUDAGraph()
                with torch.cuda.graph(graph):
                    mgr.layer_step(0)
            graph.replay()
            got = mgr.static_outputs()[0].unsqueeze(2)
        mgr.increment_seq_len()
        mgr.check_status()
        got = got.double().cpu().numpy()
        for i, ((b, hq), pick) in enumerate(decisive.items()):
            if len(decisive) > 40 and (i + step) % (len(decisive) // 40):
                continue
            s, v, packed, rot = _step_reference(mgr, args[0], ks, vs, b, hq, n_tok)
            want, size = _attend_reference(s, v, packed, rot)
            # (2^-10 again: a score is off by as much where the library rounds an element of the rotated query the other way)
            bound = 2.0 ** -9 * size + 2.0 ** -10 * np.abs(want).max()
            assert np.abs(got[b, hq, 0] - want).max() <= bound, (step, b, hq, pick)
            if n_tok > 1:
                def off(row, by):
                    moved = s.copy()
                    moved[row] += by
                    return np.abs(_attend_reference(moved, v, packed, rot)[0] - want).max() / bound
                single += sum(off(t, -np.inf) > 10 for t in pick)
                shared += len(pick) == 2 and off(pick[0], 0.1) > 2
    assert single >= 20 and shared >= 5
