"""The step's append takes four batch entries of a head per CTA when there are many rows: the same bytes as row by row."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("B,gqa,mixed,ring,rope", [(16, 4, False, False, False), (20, 3, True, False, True), (32, 1, False, True, False),
                                                   (40, 8, True, False, False)])
def test_grouped_append_matches_single_rows(B, gqa, mixed, ring, rope):
    from blockgtq_b200 import _lib
    from blockgtq_b200.layer import LayerTables, step_prepare
    from helpers import HD, tables_for
    n_kv = 8
    tabs = [tables_for("a3_1to8", h % 2) for h in range(n_kv)]
    lt = LayerTables([t[0] for t in tabs], [t[1] for t in tabs], DEV)
    gen = torch.Generator(device=DEV).manual_seed(B)
    q, k, v = (torch.randn(B, n, 1, HD, generator=gen, device=DEV).half() for n in (n_kv * gqa, n_kv, n_kv))
    cs, sn = (torch.randn(B, HD, generator=gen, device=DEV).half() for _ in range(2))
    flags = _lib.ENC_K_MIXED | _lib.ENC_V_NIBBLE if mixed else 0
    kb, vb, cap, win, sink = (lt.max_mixed_bytes if mixed else lt.max_tpb), (HD // 2 if mixed else lt.vpb), 12, 4, 2
    pos = torch.tensor([9], dtype=torch.int32, device=DEV)
    bufs = [torch.randn(B, n_kv, sink + win + 1, HD, generator=gen, device=DEV).half() for _ in range(2)]

    def run(sl):
        n = sl.stop - sl.start
        out = [torch.zeros(n, n_kv, cap, kb, dtype=torch.uint8, device=DEV), torch.zeros(n, n_kv, cap, lt.max_ng, dtype=torch.float16, device=DEV),
               torch.zeros(n, n_kv, cap, vb, dtype=torch.uint8, device=DEV), torch.zeros(n, n_kv, cap, dtype=torch.float16, device=DEV)]
        b = [t[sl].clone() for t in bufs]
        r = step_prepare(lt, q[sl], k[sl], v[sl], 0, *out, flags=flags, pos_dev=pos, rope=(cs[sl], sn[sl]) if rope else None,
                         ring=(b[0], b[1], sink, win) if ring else None)
        return [r] + out + b

    whole, parts = run(slice(0, B)), [run(slice(i, i + 1)) for i in range(B)]
    for i, t in enumerate(whole):
        assert torch.equal(t, torch.cat([p[i] for p in parts])), i
