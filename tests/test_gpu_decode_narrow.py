"""Rows too wide for the 32-token warp tile: the kernel specialised for 16-token tiles gives the general kernel's bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("T", [1, 15, 16, 256, 257, 1500])
def test_specialised_narrow_tile_matches_general(T):
    from blockgtq_b200 import BlockGTQKVManager, _lib
    from blockgtq_b200.layer import decode
    from helpers import HD, synth_head
    gen = torch.Generator().manual_seed(T)
    B, n_kv, gqa = 2, 2, 3
    mgr = BlockGTQKVManager(1, n_kv * gqa, n_kv, HD, max_seq_len=1504, batch_size=B, k_avg_bits=5.0, v_bits=4, device=DEV,
                            k_mixed=True, v_nibble=True)
    cal = [synth_head(gen, 256, gqa) for _ in range(n_kv)]
    mgr.calibrate(0, torch.stack([c[0] for c in cal]).float(), torch.stack([c[1] for c in cal]).float())
    mgr.init_from_cache([tuple(torch.randn(B, n_kv, T, HD, generator=gen).half().to(DEV) for _ in range(2))])
    q = torch.randn(B, n_kv * gqa, HD, generator=gen).half().to(DEV)
    lt, cache = mgr._layers[0], (mgr._k_packed[0], mgr._k_norms[0], mgr._v_packed[0], mgr._v_norms[0])
    po, pl = decode(lt, q, *cache, 0, T, n_splits=5, flags=mgr._dec_flags)
    go, gl = decode(lt, q, *cache, 0, T, n_splits=5, flags=mgr._dec_flags | _lib.DEC_GENERIC)
    live = torch.isfinite(gl)
    assert live.any() and torch.equal(pl, gl) and torch.equal(po[live], go[live])


@pytest.mark.parametrize("T", [1, 31, 512, 513, 3000])
def test_specialised_2bit_values_match_general(T):
    """2-bit values: the specialised kernel's 64-bit lookups (two dims of two tokens) against the general kernel's pairs."""
    from blockgtq_b200 import BlockGTQKVManager, _lib
    from blockgtq_b200.layer import decode
    from helpers import HD, synth_head
    gen = torch.Generator().manual_seed(T)
    B, n_kv, gqa = 2, 3, 4
    mgr = BlockGTQKVManager(1, n_kv * gqa, n_kv, HD, max_seq_len=3008, batch_size=B, k_avg_bits=2.0, v_bits=2, device=DEV)
    cal = [synth_head(gen, 256, gqa) for _ in range(n_kv)]
    mgr.calibrate(0, torch.stack([c[0] for c in cal]).float(), torch.stack([c[1] for c in cal]).float())
    mgr.init_from_cache([tuple(torch.randn(B, n_kv, T, HD, generator=gen).half().to(DEV) for _ in range(2))])
    q = torch.randn(B, n_kv * gqa, HD, generator=gen).half().to(DEV)
    lt, cache = mgr._layers[0], (mgr._k_packed[0], mgr._k_norms[0], mgr._v_packed[0], mgr._v_norms[0])
    wide = mgr._dec_flags & ~_lib.DEC_NARROW
    po, pl = decode(lt, q, *cache, 0, T, n_splits=3, flags=wide)
    go, gl = decode(lt, q, *cache, 0, T, n_splits=3, flags=wide | _lib.DEC_GENERIC)
    no, nl = decode(lt, q, *cache, 0, T, n_splits=3, flags=wide | _lib.DEC_NARROW)          # the other tile: other sums
    live = torch.isfinite(gl)
    assert live.any() and torch.equal(pl, gl) and torch.equal(po[live], go[live])
    assert torch.equal(torch.isfinite(nl), live) and (no[live] - go[live]).abs().max() < 1e-3 and (nl[live] - gl[live]).abs().max() < 1e-3
