"""The decode operator's tables belong to the contents of its codebook and V LUT, not to the address they had once."""
import numpy as np
import torch

from blockgtq_b200.attention import _layer_for

SEGS = [[3, 0, 128, 0, 0, 0]]


def _codebook(lt):
    return np.array(lt.desc_host[0].codebook[:8], dtype=np.uint16).view(np.float16)


def test_tables_follow_the_contents():
    lut = torch.arange(8).half()
    for i in range(20):         # freed and made anew: the allocator gives the same address again when it can
        cb = torch.full((8,), float(i), dtype=torch.float16)
        lt = _layer_for(SEGS, cb, lut, 3, 1, torch.device("cpu"))
        assert (_codebook(lt) == i).all(), i
        assert _layer_for(SEGS, cb, lut, 3, 1, torch.device("cpu")) is lt
        assert _layer_for(SEGS, cb.clone(), lut.clone(), 3, 1, torch.device("cpu")) is lt         # equal contents share them
    cb.mul_(2)                  # written in place
    assert (_codebook(_layer_for(SEGS, cb, lut, 3, 1, torch.device("cpu"))) == 38).all()
    lut[3] = 99.0
    assert np.array(_layer_for(SEGS, cb, lut, 3, 1, torch.device("cpu")).desc_host[0].v_lut[:8], dtype=np.uint16).view(np.float16)[3] == 99
    wide = torch.arange(16).half()
    a, b = (_layer_for(SEGS, c, lut, 3, 1, torch.device("cpu")) for c in (wide[:8], wide[::2]))        # the same address, other strides
    assert (_codebook(a) == np.arange(8)).all() and (_codebook(b) == 2 * np.arange(8)).all()
    with torch.inference_mode():
        inf = torch.full((8,), 3.0, dtype=torch.float16)
    assert (_codebook(_layer_for(SEGS, inf, lut, 3, 1, torch.device("cpu"))) == 3).all()
