"""The bulk encoder at the edges of its 128-row tiles: every row of a launch has the bytes it has in a launch of other
rows around it, on contiguous and strided inputs, padded cache rows and both layouts."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("case,B,T,t0,pad", [("a3_1to8", 1, 128, 0, 0), ("a2_1to8", 1, 129, 3, 1), ("a4_rt1", 9, 16, 1, 0),
                                              ("a3_1to6", 2, 391, 0, 3), ("u3", 1, 4000, 5, 0)])
@pytest.mark.parametrize("mixed", [False, True])
def test_rows_do_not_depend_on_their_tile(case, B, T, t0, pad, mixed):
    from blockgtq_b200 import _lib
    from blockgtq_b200.layer import LayerTables, encode
    from helpers import HD, tables_for
    tabs = [tables_for(case, h) for h in range(2)]
    lt = LayerTables([t[0] for t in tabs], [t[1] for t in tabs], DEV)
    gen = torch.Generator(device=DEV).manual_seed(T)
    k, v = (torch.randn(B, T, 2, HD, generator=gen, device=DEV).half().transpose(1, 2) * s for s in (3.0, 1.0))
    k[0, 0, T // 2] = 0
    flags = _lib.ENC_K_MIXED | _lib.ENC_V_NIBBLE if mixed else 0
    kb, vb = (lt.max_mixed_bytes, HD // 2) if mixed else (lt.max_tpb, lt.vpb)

    def run(k, v, t0, flags):
        n, t = k.shape[0], t0 + k.shape[2]
        out = [torch.full((n, 2, t + 2, w), 9, dtype=torch.uint8, device=DEV) for w in (kb + pad, vb + pad)]
        out += [torch.full((n, 2, t + 2, lt.max_ng), 9.0, dtype=torch.float16, device=DEV), torch.full((n, 2, t + 2), 9.0, dtype=torch.float16, device=DEV)]
        encode(lt, k, v, t0, out[0], out[2], out[1], out[3], flags=flags)
        return out

    whole = run(k, v, t0, flags)
    assert all((x[:, :, :t0] == 9).all() and (x[:, :, t0 + T:] == 9).all() for x in whole)
    assert (whole[0][:, :, t0:t0 + T, kb:] == 0).all() and (whole[1][:, :, :, vb:] == 9).all()
    # the same rows, 7 rows later in their tiles and with contiguous input
    k2, v2 = (torch.cat([x[:, :, -7:], x], dim=2).contiguous() for x in (k, v))
    shifted = run(k2, v2, 0, flags)
    for a, b in zip(whole, shifted):
        assert torch.equal(a[:, :, t0:t0 + T], b[:, :, 7:7 + T])
    # the warp-MMA encoder computes the same codes but for coordinates on a bin's edge
    other = run(k, v, t0, flags | _lib.ENC_NO_TCGEN05)
    for a, b in zip(whole[:2], other[:2]):
        assert (a != b).float().mean().item() < 2e-3
    for a, b in zip(whole[2:], other[2:]):
        assert ((a.float() - b.float()).abs() <= 2e-3 * b.float().abs()).float().mean().item() > 0.999
    assert _lib.lib().bgtq_encode_tcgen05_status() == 0


@pytest.mark.parametrize("case", ["a3_1to8", "u3"])
@pytest.mark.parametrize("mixed", [False, True])
def test_one_tile_per_cta_and_more(case, mixed):
    """The build for launches whose CTAs have one tile each gives the bytes of the one for more tiles."""
    from blockgtq_b200 import _lib
    from blockgtq_b200.layer import LayerTables, encode
    from helpers import HD, tables_for
    tabs = [tables_for(case, h) for h in range(2)]
    lt = LayerTables([t[0] for t in tabs], [t[1] for t in tabs], DEV)
    tiles = torch.cuda.get_device_properties(0).multi_processor_count // 4      # x 2 heads x (K, V): the most with one per CTA
    n = 128 * tiles + 1
    gen = torch.Generator(device=DEV).manual_seed(1)
    k, v = (torch.randn(1, 2, n, HD, generator=gen, device=DEV).half() * s for s in (3.0, 1.0))
    flags = _lib.ENC_K_MIXED | _lib.ENC_V_NIBBLE if mixed else 0
    kb, vb = (lt.max_mixed_bytes, HD // 2) if mixed else (lt.max_tpb, lt.vpb)

    def run(parts):
        out = [torch.zeros(1, 2, n, w, dtype=torch.uint8, device=DEV) for w in (kb, vb)]
        out += [torch.zeros(1, 2, n, lt.max_ng, dtype=torch.float16, device=DEV), torch.zeros(1, 2, n, dtype=torch.float16, device=DEV)]
        for lo, hi in parts:
            encode(lt, k[:, :, lo:hi], v[:, :, lo:hi], lo, out[0], out[2], out[1], out[3], flags=flags)
        return out

    for a, b in zip(run([(0, n)]), run([(0, n - 1), (n - 200, n)])):
        assert torch.equal(a, b)
    assert _lib.lib().bgtq_encode_tcgen05_status() == 0


@pytest.mark.parametrize("n", [129, 130 * 148])
@pytest.mark.parametrize("mixed", [False, True])
def test_any_order_of_dims(n, mixed):
    """Heads whose packed order does not keep RoPE pairs side by side take the bulk encoder's other way into packed order: the
    same bytes as the reference's order gives for inputs whose dims are exchanged accordingly."""
    import copy
    from blockgtq_b200 import _lib
    from blockgtq_b200.layer import LayerTables, encode
    from helpers import HD, tables_for
    kt, vt = tables_for("a3_1to8", 0)
    gen = torch.Generator().manual_seed(n)
    order = torch.randperm(HD, generator=gen)
    other = copy.copy(kt)
    other.head_perm = order[kt.head_perm]
    k, v = (torch.randn(1, 1, n, HD, generator=gen).half().to(DEV) for _ in range(2))
    k2 = torch.empty_like(k)
    k2[..., order.to(DEV)] = k
    flags = _lib.ENC_K_MIXED | _lib.ENC_V_NIBBLE if mixed else 0

    def run(table, keys):
        lt = LayerTables([table], [vt], DEV)
        kb, vb = (lt.max_mixed_bytes, HD // 2) if mixed else (lt.max_tpb, lt.vpb)
        out = [torch.zeros(1, 1, n, w, dtype=torch.uint8, device=DEV) for w in (kb, vb)]
        out += [torch.zeros(1, 1, n, lt.max_ng, dtype=torch.float16, device=DEV), torch.zeros(1, 1, n, dtype=torch.float16, device=DEV)]
        encode(lt, keys, v, 0, out[0], out[2], out[1], out[3], flags=flags)
        return out

    for a, b in zip(run(kt, k), run(other, k2)):
        assert torch.equal(a, b)
    assert _lib.lib().bgtq_encode_tcgen05_status() == 0
