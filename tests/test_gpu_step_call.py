"""The one-call layer step reads the caller's rows where they lie: every way of handing them over gives the step's
bits, and so does the step on the static buffers."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("batch,n_q,n_kv,T,window", [(1, 8, 8, 0, 0), (3, 6, 2, 511, 0), (2, 16, 2, 700, 0), (2, 8, 2, 300, 64)])
def test_step_call_input_layouts(batch, n_q, n_kv, T, window):
    from blockgtq_b200 import BlockGTQKVManager
    from helpers import HD, synth_head
    gen = torch.Generator().manual_seed(17)
    mgr = BlockGTQKVManager(1, n_q, n_kv, HD, max_seq_len=T + 8, batch_size=batch, device=DEV,
                            n_sink=4 if window else 0, recent_window=window)
    cal = [synth_head(gen, 256, n_q // n_kv) for _ in range(n_kv)]
    mgr.calibrate(0, torch.stack([c[0] for c in cal]).float(), torch.stack([c[1] for c in cal]).float())
    if T:
        mgr.init_from_cache([tuple(torch.randn(batch, n_kv, T, HD, generator=gen).half().to(DEV) for _ in range(2))])
    q, k, v = (torch.randn(batch, n, 1, HD, generator=gen).half().to(DEV) for n in (n_q, n_kv, n_kv))
    row = T if not window else max(0, T - 4 - window)

    def state():
        return [t[0, :, :, row].clone() for t in (mgr._k_packed, mgr._k_norms, mgr._v_packed, mgr._v_norms)]

    for dst, src in zip(mgr.static_inputs(0), (q, k, v)):
        dst.copy_(src)
    mgr.layer_step(0)
    want = mgr.static_outputs()[0].clone()
    rows = state()
    wide = torch.cat([q, k, v], dim=1).transpose(1, 2).contiguous().transpose(1, 2)        # a fused projection's layout
    forms = {"as is": (q, k, v),
             "views": (wide[:, :n_q], wide[:, n_q:n_q + n_kv], wide[:, n_q + n_kv:]),
             "fp32": (q.float(), k.float(), v.float()),
             "last dim strided": tuple(t.transpose(2, 3).contiguous().repeat_interleave(2, dim=2)[:, :, ::2].transpose(2, 3)
                                       for t in (q, k, v))}
    for name, args in forms.items():
        mgr.static_outputs().fill_(float("nan"))
        out = mgr.append_and_attend(0, *args)
        assert out.shape == (batch, n_q, 1, HD)
        assert torch.equal(out[:, :, 0], want), name
        assert all(torch.equal(a, b) for a, b in zip(state(), rows)), name
    torch.cuda.synchronize()
    mgr.check_status()
