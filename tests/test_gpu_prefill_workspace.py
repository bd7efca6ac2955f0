"""Prefill attention when its workspace meets a limit: the library's bound on one launch, or a device without room."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _case(B, n_kv, gqa, T, S_q):
    from blockgtq_b200.layer import LayerTables, encode, rotate_q_bulk
    from helpers import HD, tables_for
    tabs = [tables_for("a3_1to8", h % 2) for h in range(n_kv)]
    lt = LayerTables([t[0] for t in tabs], [t[1] for t in tabs], DEV)
    gen = torch.Generator(device=DEV).manual_seed(T)
    q, k, v = (torch.randn(B, n, s, HD, generator=gen, device=DEV).half() for n, s in ((n_kv * gqa, S_q), (n_kv, T), (n_kv, T)))
    cache = (torch.zeros(B, n_kv, T, lt.max_tpb, dtype=torch.uint8, device=DEV), torch.zeros(B, n_kv, T, lt.max_ng, dtype=torch.float16, device=DEV),
             torch.zeros(B, n_kv, T, lt.vpb, dtype=torch.uint8, device=DEV), torch.zeros(B, n_kv, T, dtype=torch.float16, device=DEV))
    encode(lt, k, v, 0, *cache)
    return lt, rotate_q_bulk(lt, q), cache


@pytest.mark.parametrize("B,n_kv,gqa,T,S_q,tiles", [(1, 3, 2, 700, 33, 13), (1, 8, 1, 260, 260, 5), (3, 3, 4, 300, 7, 4), (5, 2, 3, 130, 5, 9),
                                                    (2, 2, 1, 500, 64, 1)])
def test_launches_within_the_bound(B, n_kv, gqa, T, S_q, tiles, monkeypatch):
    """``tiles``: tile workspaces (128 tokens of one head) that a launch may take; the last case cannot keep to it."""
    from blockgtq_b200 import _lib, layer
    lt, q_rot, cache = _case(B, n_kv, gqa, T, S_q)
    L = _lib.lib()
    for rot in (lt.v_rot, None):
        args = dict(q_pos_offset=T - S_q, causal=True, v_rot=rot)
        want = layer.prefill_attention(lt, q_rot, *cache, T, **args).float()
        fixed = L.bgtq_prefill_workspace_bytes(1, gqa, 1, S_q, T, T - S_q, 1, rot is not None) - -(-T // 128) * 128 * 768
        bound = tiles * 128 * 768 + fixed
        seen = []
        empty = torch.empty
        monkeypatch.setattr(layer, "_PREFILL_WORKSPACE", bound)
        monkeypatch.setattr(torch, "empty", lambda *a, **k: seen.append(a) or empty(*a, **k))
        before = _lib.launches
        got = layer.prefill_attention(lt, q_rot, *cache, T, **args).float()
        monkeypatch.undo()
        sizes = [a[0] for a in seen if isinstance(a[0], int) and len(a) == 1]
        assert len(sizes) == 1 and _lib.launches - before > 2       # one workspace, several launches
        one = L.bgtq_prefill_workspace_bytes(1, gqa, 1, S_q, T, T - S_q, 1, rot is not None)
        assert sizes[0] <= max(bound, one)
        # the cut of the cache among CTAs may differ with the launch: partial results are added in another order
        assert ((got - want).abs() <= 1e-3 + want.abs() * 2.0 ** -10).all()
    assert L.bgtq_prefill_tcgen05_status() == 0


def test_no_room_for_the_workspace():
    from blockgtq_b200 import _lib, layer
    B, n_kv, gqa, T, S_q = 2, 4, 2, 40000, 16
    lt, q_rot, cache = _case(B, n_kv, gqa, T, S_q)
    args = dict(q_pos_offset=T - S_q, causal=True, v_rot=lt.v_rot)
    want = layer.prefill_attention(lt, q_rot, *cache, T, flags=_lib.PF_NO_TCGEN05, **args)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    ws = _lib.lib().bgtq_prefill_workspace_bytes(1, gqa, 1, S_q, T, T - S_q, 1, 1)
    fill = []
    try:
        torch.cuda.set_per_process_memory_fraction(torch.cuda.memory_reserved() / total)
        size = 1 << 30
        while size > 4 << 20:                   # what the allocator's blocks still hold
            try:
                fill.append(torch.empty(size, dtype=torch.uint8, device=DEV))
            except torch.OutOfMemoryError:
                size //= 2
        # room for the results, not for the tiles of one head of one batch entry
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (8 << 20)) / total)
        for bound in (layer._PREFILL_WORKSPACE, ws):
            with pytest.MonkeyPatch.context() as m:
                m.setattr(layer, "_PREFILL_WORKSPACE", bound)
                before = _lib.launches
                got = layer.prefill_attention(lt, q_rot, *cache, T, **args)
            assert _lib.launches - before == 1                      # mma.sync, not the tcgen05 form's two
            assert torch.equal(got, want)
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
        del fill
    again = layer.prefill_attention(lt, q_rot, *cache, T, **args).float()
    assert ((again - want.float()).abs() <= 1e-3 + want.float().abs() * 2.0 ** -10).all()


def test_entry_point_without_a_workspace():
    """bgtq_prefill_attention takes its workspace from the stream's pool; a pool that cannot give it changes the kernel."""
    from blockgtq_b200 import _lib
    from helpers import HD
    rt = pytest.importorskip("cuda.bindings.runtime")
    B, n_kv, gqa, T, S_q = 1, 2, 3, 60000, 50
    lt, q_rot, (kp, kn, vp, vn) = _case(B, n_kv, gqa, T, S_q)

    def run(flags):
        out = torch.full((B, n_kv * gqa, S_q, HD), float("nan"), device=DEV)
        rc = _lib.lib().bgtq_prefill_attention(
            lt.desc_dev.data_ptr(), q_rot.data_ptr(), *q_rot.stride()[:3], kp.data_ptr(), *kp.stride()[:3], kn.data_ptr(), *kn.stride()[:3],
            vp.data_ptr(), *vp.stride()[:3], vn.data_ptr(), *vn.stride()[:3], B, n_kv * gqa, n_kv, S_q, T, T - S_q, 1, 1.0 / HD ** 0.5, flags,
            out.data_ptr(), torch.cuda.current_stream().cuda_stream)
        assert rc == 0
        torch.cuda.synchronize()
        return out

    mma, t5 = run(_lib.PF_NO_TCGEN05), run(0)
    assert not torch.equal(mma, t5) and ((t5 - mma).abs() <= 1e-3 + mma.abs() * 2.0 ** -10).all()
    props = rt.cudaMemPoolProps()
    props.allocType = rt.cudaMemAllocationType.cudaMemAllocationTypePinned
    props.location.type, props.location.id = rt.cudaMemLocationType.cudaMemLocationTypeDevice, 0
    props.maxSize = 1 << 20                     # (pools grow in steps of some 32 MB; the workspace takes 92)
    err, small = rt.cudaMemPoolCreate(props)
    assert err == rt.cudaError_t.cudaSuccess
    err, usual = rt.cudaDeviceGetMemPool(0)
    assert err == rt.cudaError_t.cudaSuccess
    try:
        assert rt.cudaDeviceSetMemPool(0, small)[0] == rt.cudaError_t.cudaSuccess
        assert torch.equal(run(0), mma)
    finally:
        rt.cudaDeviceSetMemPool(0, usual)
        rt.cudaMemPoolDestroy(small)
    assert torch.equal(run(0), t5)


def test_rotation_in_any_layout():
    """V's rotation as a transposed view, as a matrix of its own for one head, as rows of all heads; another type is an error."""
    from blockgtq_b200 import layer
    from helpers import HD
    for n_kv in (1, 3):
        lt, q_rot, cache = _case(1, n_kv, 2, 300, 40)
        args = dict(q_pos_offset=260, causal=True)
        want = layer.prefill_attention(lt, q_rot, *cache, 300, v_rot=lt.v_rot, **args)
        turned = lt.v_rot.transpose(1, 2).contiguous().transpose(1, 2)
        for rot in [turned, lt.v_rot.reshape(n_kv * HD, HD)] + ([lt.v_rot[0], turned[0]] if n_kv == 1 else []):
            assert torch.equal(layer.prefill_attention(lt, q_rot, *cache, 300, v_rot=rot, **args), want)
        for bad in (lt.v_rot.half(), lt.v_rot[:, :, :64], lt.v_rot.cpu()):
            with pytest.raises((TypeError, RuntimeError)):
                layer.prefill_attention(lt, q_rot, *cache, 300, v_rot=bad, **args)
