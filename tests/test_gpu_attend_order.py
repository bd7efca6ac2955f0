"""An attention enqueued right behind the encode that writes its rows reads the new rows, however busy the stream is:
the launches may start while the encode still runs, and only the rows that they may read by then are read."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _manager(layers, batch, n_kv, gqa, cap, **kw):
    from blockgtq_b200 import BlockGTQKVManager
    from helpers import HD, synth_head
    gen = torch.Generator().manual_seed(n_kv)
    mgr = BlockGTQKVManager(layers, n_kv * gqa, n_kv, HD, max_seq_len=cap, batch_size=batch, device=DEV, **kw)
    cal = [synth_head(gen, 256, gqa) for _ in range(n_kv)]
    for li in range(layers):
        mgr.calibrate(li, torch.stack([c[0] for c in cal]).float(), torch.stack([c[1] for c in cal]).float())
    return mgr


def _kv(gen, batch, n_kv, n):
    from helpers import HD
    return tuple(torch.randn(batch, n_kv, n, HD, generator=gen, device=DEV).half() for _ in range(2))


class _Busy:
    """Ordinary work that keeps the stream occupied while the host enqueues what follows."""

    def __init__(self):
        self.a = torch.randn(4096, 4096, device=DEV).half()
        self.out = torch.empty_like(self.a)

    def __call__(self):
        for _ in range(3):
            torch.mm(self.a, self.a, out=self.out)


# rows of the bulk encode (batch x tokens) from its smallest to several waves of tiles; few heads leave SMs free for the
# launches behind it, and with the queries already in the packed basis the decode is the launch right behind the encode
@pytest.mark.parametrize("batch,n_kv,T,baked,window", [(1, 1, 128, False, 0), (1, 8, 800, False, 0), (2, 2, 400, False, 0),
                                                       (1, 1, 800, True, 0), (1, 8, 128, True, 0), (1, 2, 700, False, 64),
                                                       (1, 4, 6000, True, 0)])
def test_attend_behind_a_bulk_encode(batch, n_kv, T, baked, window):
    from helpers import HD
    gqa = 4
    mgr = _manager(1, batch, n_kv, gqa, T + 8, n_sink=4 if window else 0, recent_window=window)
    for qz in mgr.quantizers[0]:
        qz._q_perm_baked = baked
    gen = torch.Generator(device=DEV).manual_seed(T)
    prompts = [_kv(gen, batch, n_kv, T) for _ in range(2)]
    q = torch.randn(batch, n_kv * gqa, 1, HD, generator=gen, device=DEV).half()
    want = []
    for kv in prompts:
        mgr.init_from_cache([kv])
        torch.cuda.synchronize()
        want.append([t.clone() for t in mgr.attend(0, q, want_partial=True)])
        torch.cuda.synchronize()
    assert not torch.equal(want[0][0], want[1][0])
    busy = _Busy()
    got = []
    for i in range(60):
        busy()
        mgr.init_from_cache([prompts[i & 1]])
        got.append(mgr.attend(0, q, want_partial=True))
    torch.cuda.synchronize()
    for i, r in enumerate(got):
        assert all(torch.equal(a, b) for a, b in zip(r, want[i & 1])), i
    mgr.check_status()


@pytest.mark.parametrize("batch,n_kv,t,S", [(1, 1, 0, 128), (1, 2, 600, 130), (2, 8, 37, 64), (1, 4, 3000, 800)])
def test_append_and_attend_of_several_tokens(batch, n_kv, t, S):
    from helpers import HD
    gqa = 2
    mgr = _manager(1, batch, n_kv, gqa, t + S + 8)
    gen = torch.Generator(device=DEV).manual_seed(t + S)
    if t:
        mgr.init_from_cache([_kv(gen, batch, n_kv, t)])
    pieces = [_kv(gen, batch, n_kv, S) for _ in range(2)]
    q = torch.randn(batch, n_kv * gqa, 1, HD, generator=gen, device=DEV).half()
    want = []
    for k, v in pieces:
        mgr._append_tokens(0, k, v, t)
        torch.cuda.synchronize()
        want.append(mgr.attend(0, q, t + S)[0].unsqueeze(2))
        torch.cuda.synchronize()
    assert not torch.equal(want[0], want[1])
    busy = _Busy()
    got = []
    for i in range(60):
        busy()
        got.append(mgr.append_and_attend(0, q, *pieces[i & 1]))
    torch.cuda.synchronize()
    for i, r in enumerate(got):
        assert torch.equal(r, want[i & 1]), i
    mgr.check_status()


@pytest.mark.parametrize("batch,n_kv,T", [(1, 1, 128), (1, 8, 800), (2, 2, 3000)])
def test_layer_step_behind_a_bulk_encode(batch, n_kv, T):
    """The step's decode reads the older rows and the position before its own dependency wait; the rows may come from an
    encode right in front of the step, the position from the kernel that advanced it."""
    from helpers import HD
    gqa = 4
    mgr = _manager(1, batch, n_kv, gqa, T + 64)
    mgr._ensure_storage()
    gen = torch.Generator(device=DEV).manual_seed(T + 1)
    prompts = [_kv(gen, batch, n_kv, T) for _ in range(2)]
    steps = [(torch.randn(batch, n_kv * gqa, 1, HD, generator=gen, device=DEV).half(),) + _kv(gen, batch, n_kv, 1) for _ in range(4)]

    def run(i, sync):
        mgr.seq_len = T
        mgr._sync_pos()                 # nothing but the encode's launch is left between it and the first step
        mgr._encode_kv(0, *prompts[i], 0, T)
        out = []
        for s in steps:
            sync()
            out.append(mgr.append_and_attend(0, *s).clone())
            sync()
            mgr.increment_seq_len()
        return out

    want = [run(i, torch.cuda.synchronize) for i in range(2)]
    assert not torch.equal(want[0][0], want[1][0])
    busy = _Busy()
    got = []
    for i in range(40):
        busy()
        got.append(run(i & 1, lambda: None))
    torch.cuda.synchronize()
    for i, r in enumerate(got):
        assert all(torch.equal(a, b) for a, b in zip(r, want[i & 1])), i
    mgr.check_status()


def test_operator_with_a_rotation_made_for_the_call():
    """The operator's V rotation may be a tensor that the call itself converts: the merge reads it as converted, not as its
    memory was a moment before."""
    from blockgtq_b200 import fused_blockgtq_decode_attention
    from blockgtq_b200.quantizer import BlockGTQQuantizer
    from helpers import HD, synth_head
    gen = torch.Generator().manual_seed(6)
    qz = BlockGTQQuantizer(HD, avg_bits=3.0, device=torch.device(DEV))
    qs, ks = synth_head(gen, 256, 2)
    qz.calibrate(qs.float(), ks.float())
    qz.init_v_quantizer(v_bits=3, seed=42)
    ka = qz.build_kernel_args()
    kp, kn, _ = qz.compress_packed(torch.randn(1, 1, 700, HD, generator=gen).half().to(DEV))
    vp, vn = qz.compress_v_packed(torch.randn(1, 1, 700, HD, generator=gen).half().to(DEV))
    q = torch.randn(1, 2, 1, HD, generator=gen).half().to(DEV)
    rots = [torch.linalg.qr(torch.randn(HD, HD, generator=gen))[0].half().to(DEV) for _ in range(2)]
    kn = kn.half()

    def run(rot):
        return fused_blockgtq_decode_attention(q, kp, kn, ka["codebook_flat"], ka["lut_offset"], ka["norm_group"], ka["segments_b"],
                                               vp, vn, qz.v_lut, v_bits=3, v_rotation=rot)

    want = []
    for r in rots:
        r32 = r.float()
        torch.cuda.synchronize()
        want.append(run(r32).clone())
        torch.cuda.synchronize()
    busy = _Busy()
    got = []
    for i in range(60):
        busy()
        got.append(run(rots[i & 1]))
        got.append(run(rots[1 - (i & 1)]))
    torch.cuda.synchronize()
    for i in range(60):
        assert torch.equal(got[2 * i], want[i & 1]) and torch.equal(got[2 * i + 1], want[1 - (i & 1)]), i


def test_a_preparation_with_nothing_to_do_keeps_the_order():
    """A step preparation that skips both sides and has no queries still ends behind the work in front of it."""
    from blockgtq_b200 import _lib
    from blockgtq_b200.layer import LayerTables, decode, encode, step_prepare
    from helpers import HD, tables_for
    n_kv, T = 2, 2000
    tabs = [tables_for("a3_1to8", h) for h in range(n_kv)]
    lt = LayerTables([t[0] for t in tabs], [t[1] for t in tabs], DEV)
    gen = torch.Generator(device=DEV).manual_seed(9)
    cache = (torch.zeros(1, n_kv, T + 8, lt.max_tpb, dtype=torch.uint8, device=DEV), torch.zeros(1, n_kv, T + 8, lt.max_ng, dtype=torch.float16, device=DEV),
             torch.zeros(1, n_kv, T + 8, lt.vpb, dtype=torch.uint8, device=DEV), torch.zeros(1, n_kv, T + 8, dtype=torch.float16, device=DEV))
    prompts = [_kv(gen, 1, n_kv, T) for _ in range(2)]
    one = _kv(gen, 1, n_kv, 1)
    q = torch.randn(1, 2 * n_kv, HD, generator=gen, device=DEV).half()
    n_splits = 8

    def run(i, sync):
        encode(lt, *prompts[i], 0, *cache)
        sync()
        step_prepare(lt, None, *one, T, *cache, flags=_lib.ENC_SKIP_K | _lib.ENC_SKIP_V | _lib.ENC_PROGRAMMATIC)
        sync()
        part_o = torch.zeros(1, 2 * n_kv, n_splits, HD, device=DEV) if sync is torch.cuda.synchronize else parts.pop()
        part_lse = torch.empty(1, 2 * n_kv, n_splits, device=DEV)
        return decode(lt, q, *cache, 0, T, n_splits=n_splits, flags=_lib.DEC_PROGRAMMATIC, part_o=part_o, part_lse=part_lse)

    want = [run(i, torch.cuda.synchronize) for i in range(2)]
    assert not torch.equal(want[0][1], want[1][1])
    parts = [torch.zeros(1, 2 * n_kv, n_splits, HD, device=DEV) for _ in range(60)]        # (nothing ordinary is enqueued in between)
    busy = _Busy()
    got = []
    for i in range(60):
        busy()
        got.append(run(i & 1, lambda: None))
    torch.cuda.synchronize()
    for i, (o, lse) in enumerate(got):
        assert torch.equal(o, want[i & 1][0]) and torch.equal(lse, want[i & 1][1]), i
