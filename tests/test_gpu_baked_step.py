"""Layer steps with queries that arrive in the packed basis (rotations baked into the projection), on the static buffers and
on the caller's tensors in several layouts: the step of the original queries, rotated ahead."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("batch,n_q,n_kv,T", [(1, 4, 2, 300), (3, 6, 2, 300), (2, 3, 3, 0)])
def test_baked_queries(batch, n_q, n_kv, T):
    from blockgtq_b200 import BlockGTQKVManager
    from blockgtq_b200.layer import rotate_q
    from helpers import HD, synth_head
    gen = torch.Generator().manual_seed(23)
    mgr = BlockGTQKVManager(1, n_q, n_kv, HD, max_seq_len=T + 8, batch_size=batch, device=DEV)
    cal = [synth_head(gen, 256, n_q // n_kv) for _ in range(n_kv)]
    mgr.calibrate(0, torch.stack([c[0] for c in cal]).float(), torch.stack([c[1] for c in cal]).float())
    if T:
        mgr.init_from_cache([tuple(torch.randn(batch, n_kv, T, HD, generator=gen).half().to(DEV) for _ in range(2))])
    q, k, v = (torch.randn(batch, n, 1, HD, generator=gen).half().to(DEV) for n in (n_q, n_kv, n_kv))
    want = mgr.append_and_attend(0, q, k, v).clone()
    q = rotate_q(mgr._layers[0], q).unsqueeze(2)
    for qz in mgr.quantizers[0]:
        qz._q_perm_baked = True
    wide = torch.cat([q, k, v], dim=1)
    for args in ((q, k, v), (wide[:, :n_q], wide[:, n_q:n_q + n_kv], wide[:, n_q + n_kv:]), (q.float(), k.float(), v.float())):
        mgr.static_outputs().fill_(float("nan"))
        assert torch.equal(mgr.append_and_attend(0, *args), want)
    for dst, src in zip(mgr.static_inputs(0), (q, k, v)):
        dst.copy_(src)
    mgr.static_outputs().fill_(float("nan"))
    mgr.layer_step(0)
    assert torch.equal(mgr.static_outputs()[0].unsqueeze(2), want)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        mgr.layer_step(0)
    mgr.static_outputs().fill_(float("nan"))
    g.replay()
    assert torch.equal(mgr.static_outputs()[0].unsqueeze(2), want)
    mgr.check_status()
