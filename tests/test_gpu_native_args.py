"""Arguments of the natively taken calls in the forms in which Python programs write them."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("flag", [1, np.bool_(True), torch.tensor(True), "yes"])
def test_true_flags_of_other_types_ask_for_the_lse(flag):
    from blockgtq_b200 import BlockGTQKVManager, fused_blockgtq_decode_attention
    from helpers import HD, synth_head
    gen = torch.Generator().manual_seed(3)
    mgr = BlockGTQKVManager(1, 4, 1, HD, max_seq_len=64, device=DEV)
    qs, ks = synth_head(gen, 256, 4)
    mgr.calibrate(0, qs.float(), ks.float())
    mgr.init_from_cache([tuple(torch.randn(1, 1, 40, HD, generator=gen).half().to(DEV) for _ in range(2))])
    q = torch.randn(1, 4, 1, HD, generator=gen).half().to(DEV)
    want = mgr.attend(0, q, want_partial=True)
    assert all(torch.equal(a, b) for a, b in zip(mgr.attend(0, q, want_partial=flag), want))
    assert mgr.attend(0, q, want_partial=0)[1:] == (None, None)
    qz = mgr.quantizers[0][0]
    ka = qz.build_kernel_args()
    cache = [t[0, :, :, :40].contiguous() for t in (mgr._k_packed, mgr._k_norms, mgr._v_packed, mgr._v_norms)]
    args = (qz.rotate_q_for_packed_kernel(q), cache[0], cache[1], ka["codebook_flat"], ka["lut_offset"], ka["norm_group"],
            ka["segments_b"], cache[2], cache[3], qz.v_lut)
    kw = dict(v_bits=3, v_rotation=qz._v_rot)
    out, lse = fused_blockgtq_decode_attention(*args, return_lse=flag, **kw)
    ref = fused_blockgtq_decode_attention(*args, return_lse=True, **kw)
    assert torch.equal(out, ref[0]) and torch.equal(lse, ref[1])


def test_ranges_may_be_any_whole_numbers():
    from blockgtq_b200 import BlockGTQKVManager
    from helpers import HD, synth_head
    gen = torch.Generator().manual_seed(4)
    mgr = BlockGTQKVManager(1, 2, 1, HD, max_seq_len=64, device=DEV)
    qs, ks = synth_head(gen, 256, 2)
    mgr.calibrate(0, qs.float(), ks.float())
    mgr.init_from_cache([tuple(torch.randn(1, 1, 40, HD, generator=gen).half().to(DEV) for _ in range(2))])
    q = torch.randn(1, 2, 1, HD, generator=gen).half().to(DEV)
    want = mgr.attend(0, q, token_range=(3, 39), n_splits=2)[0]
    for lo, hi, n in ((np.int64(3), np.int32(39), np.int64(2)), (3.0, 39.0, 2.0), (torch.tensor(3), torch.tensor(39), torch.tensor(2))):
        assert torch.equal(mgr.attend(0, q, token_range=(lo, hi), n_splits=n)[0], want)
    for n in (0, -1):
        with pytest.raises(RuntimeError, match="bad argument"):
            mgr.attend(0, q, n_splits=n)


def test_one_query_head_cut_out_of_a_larger_tensor():
    """(B, 1, 1, 128) views whose head dim of one has another tensor's stride: one query head per KV head."""
    from blockgtq_b200 import fused_blockgtq_decode_attention
    from blockgtq_b200.quantizer import BlockGTQQuantizer
    from helpers import HD, synth_head
    gen = torch.Generator().manual_seed(5)
    qz = BlockGTQQuantizer(HD, avg_bits=3.0, device=torch.device(DEV))
    qs, ks = synth_head(gen, 256, 1)
    qz.calibrate(qs.float(), ks.float())
    qz.init_v_quantizer(v_bits=3, seed=42)
    ka = qz.build_kernel_args()
    kp, kn, _ = qz.compress_packed(torch.randn(1, 1, 50, HD, generator=gen).half().to(DEV))
    vp, vn = qz.compress_v_packed(torch.randn(1, 1, 50, HD, generator=gen).half().to(DEV))
    q = torch.randn(1, 1, 9, HD, generator=gen).half().to(DEV)[:, :, 4:5]
    assert q.is_contiguous() and q.stride(1) != HD

    def run(q):
        return fused_blockgtq_decode_attention(q, kp, kn.half(), ka["codebook_flat"], ka["lut_offset"], ka["norm_group"], ka["segments_b"],
                                               vp, vn, qz.v_lut, v_bits=3, v_rotation=qz._v_rot)

    assert torch.equal(run(q), run(q.clone()))
