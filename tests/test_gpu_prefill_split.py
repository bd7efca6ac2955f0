"""Prefill attention where its launch takes another form: the cache cut among several CTAs, query groups that do not
divide a block of rows, the last row block and tile ragged or exactly full, no causal limit; and the bulk rotation at
the edges of its row tiles.  Oracle: the mma.sync kernel (held to the float64 oracle elsewhere) and an fp32 product."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _layer(n_kv):
    from blockgtq_b200.layer import LayerTables
    from helpers import tables_for
    tabs = [tables_for("a3_1to8", h % 2) for h in range(n_kv)]
    return LayerTables([t[0] for t in tabs], [t[1] for t in tabs], DEV)


@pytest.mark.parametrize("n_kv,gqa,S_q,offset,causal", [(1, 7, 40, 5000, True), (2, 5, 257, 0, True), (1, 1, 256, 128, True),
                                                        (1, 1, 1, 4095, True), (2, 4, 64, 3000, False), (1, 8, 33, 0, True)])
def test_prefill_launch_forms(n_kv, gqa, S_q, offset, causal):
    from blockgtq_b200 import _lib
    from blockgtq_b200.layer import encode, prefill_attention, rotate_q_bulk
    from helpers import HD
    lt = _layer(n_kv)
    gen = torch.Generator(device=DEV).manual_seed(7 * S_q + offset)
    B, T = 2, offset + S_q
    q, k, v = (torch.randn(B, n, s, HD, generator=gen, device=DEV).half() for n, s in ((n_kv * gqa, S_q), (n_kv, T), (n_kv, T)))
    kp = torch.zeros(B, n_kv, T, lt.max_tpb, dtype=torch.uint8, device=DEV)
    kn = torch.zeros(B, n_kv, T, lt.max_ng, dtype=torch.float16, device=DEV)
    vp = torch.zeros(B, n_kv, T, lt.vpb, dtype=torch.uint8, device=DEV)
    vn = torch.zeros(B, n_kv, T, dtype=torch.float16, device=DEV)
    encode(lt, k, v, 0, kp, kn, vp, vn)
    q_rot = rotate_q_bulk(lt, q)
    for rot in (lt.v_rot, None):
        args = dict(q_pos_offset=offset, causal=causal, v_rot=rot)
        a = prefill_attention(lt, q_rot, kp, kn, vp, vn, T, **args)
        b = prefill_attention(lt, q_rot, kp, kn, vp, vn, T, flags=_lib.PF_NO_TCGEN05, **args)
        assert torch.isfinite(a.float()).all()
        assert ((a.float() - b.float()).abs() <= 1e-3 + b.float().abs() * 2.0 ** -10).all()
    assert _lib.lib().bgtq_prefill_tcgen05_status() == 0


@pytest.mark.parametrize("n_kv,gqa,S", [(1, 1, 1), (2, 3, 127), (1, 4, 32), (2, 2, 129), (1, 8, 300)])
def test_bulk_rotation(n_kv, gqa, S):
    from blockgtq_b200.layer import rotate_q_bulk
    from helpers import HD
    lt = _layer(n_kv)
    gen = torch.Generator(device=DEV).manual_seed(S)
    q = torch.randn(2, S, n_kv * gqa, HD, generator=gen, device=DEV).half().transpose(1, 2)
    want = rotate_q_bulk(lt, q.float()).float()         # fp32 queries: gather + fp32 product
    got = rotate_q_bulk(lt, q).float()
    assert got.shape == want.shape
    assert ((got - want).abs() <= 1e-5 + want.abs() * 2.0 ** -10).all()
