"""The bulk query rotation under torch's transforms and on the CPU: there it is made of torch's own operators."""
import pytest
import torch

from blockgtq_b200.layer import LayerTables, rotate_q_bulk
from helpers import HD, tables_for

DEVICES = ["cpu", pytest.param("cuda:0", marks=pytest.mark.gpu)]


def _case(dev, n_kv=2, gqa=3, S=5):
    tabs = [tables_for("a3_1to8", h % 2) for h in range(n_kv)]
    lt = LayerTables([t[0] for t in tabs], [t[1] for t in tabs], dev)
    gen = torch.Generator().manual_seed(1)
    q = torch.randn(2, n_kv * gqa, S, HD, generator=gen).half().to(dev)
    M = torch.zeros(n_kv, HD, HD, device=dev)       # q -> q[perm] @ rot as one matrix per KV head
    for h in range(n_kv):
        M[h, lt.head_perm[h]] = lt.rot_k[h]
    want = torch.einsum("bhgsd,hdp->bhgsp", q.view(2, n_kv, gqa, S, HD).double(), M.double()).reshape(q.shape)
    return lt, q, M.repeat_interleave(gqa, dim=0), want


def _close(a, b):
    # one rounding to fp16 of an fp32 sum of 128 terms (2^-11 relative, with room for the sum's own error)
    return ((a.double() - b).abs() <= 1e-4 + b.abs() * 2.0 ** -10).all()


@pytest.mark.parametrize("dev", DEVICES)
def test_plain(dev):
    lt, q, _, want = _case(dev)
    for x in (q, q.float(), q.double()):
        out = rotate_q_bulk(lt, x)
        assert out.dtype == torch.float16 and _close(out, want)
    assert rotate_q_bulk(lt, q[:, :, :0]).shape == (2, 6, 0, HD)


@pytest.mark.parametrize("dev", DEVICES)
def test_gradients_forward_mode_and_vmap(dev):
    lt, q, M, want = _case(dev)
    x = q.clone().requires_grad_()
    y = rotate_q_bulk(lt, x)
    assert _close(y.detach(), want)
    g = torch.randn(q.shape, generator=torch.Generator().manual_seed(2)).half().to(dev)
    y.backward(g)
    grad = torch.einsum("bnsp,ndp->bnsd", g.double(), M.double())
    assert ((x.grad.double() - grad).abs() <= 1e-4 + grad.abs() * 2.0 ** -10).all()
    with torch.no_grad():
        assert not rotate_q_bulk(lt, x).requires_grad
    with torch.autograd.forward_ad.dual_level():
        out = torch.autograd.forward_ad.unpack_dual(rotate_q_bulk(lt, torch.autograd.forward_ad.make_dual(q, g)))
        assert _close(out.tangent, torch.einsum("bnsd,ndp->bnsp", g.double(), M.double()))
    many = torch.stack([q, 2 * q])
    assert _close(torch.vmap(lambda t: rotate_q_bulk(lt, t))(many), torch.stack([want, 2 * want]))
