"""CPU: split schedules hold every tile once, and are shorter than whole items where one is chosen."""
import ctypes

import pytest

from test_gpu_split import fwd_tiles


def plan(entry, ctas, **kw):
    from flamia_blackwell_attention_b200 import _lib as L
    a, s = L.AttnArgs(), L.Split()
    a.b, a.s_q, a.s_k, a.h, a.h_kv, a.d = (kw[n] for n in ("b", "sq", "sk", "h", "hk", "d"))
    a.flags = L.FL_A_CAUSAL if kw["causal"] else 0
    a.window_left_p1 = kw["left"] + 1 if kw.get("left") is not None else 0
    assert getattr(L.load(), entry)(ctypes.byref(a), ctas, ctypes.byref(s)) == 0
    return [(x >> L.SPLIT_TILE_BITS, x & ((1 << L.SPLIT_TILE_BITS) - 1)) for x in s.at[:s.parts + 1]] if s.parts else None


SHAPES = [dict(b=b, sq=sq, sk=sk, h=h, hk=hk, d=128, causal=causal)
          for b, sq, sk, h, hk in ((1, 128, 8192, 1, 1), (1, 4096, 4096, 4, 2), (2, 256, 256, 2, 2), (4, 512, 8192, 32, 8), (1, 8832, 8832, 2, 2),
                                   (1, 1152, 640, 3, 1), (2, 2048, 2048, 16, 4), (1, 128, 128, 1, 1))
          for causal in (True, False)]


@pytest.mark.parametrize("ctas", [148, 132, 16])
@pytest.mark.parametrize("kw", SHAPES)
def test_forward_schedule(kw, ctas):
    tiles = fwd_tiles(kw["b"], kw["sq"], kw["sk"], kw["h"], kw["causal"])
    check(plan("fl_fwd_split_plan", ctas, **kw), tiles, ctas)


def check(at, tiles, ctas):
    if at is None:
        return
    assert len(at) - 1 <= ctas and at[0] == (0, 0) and at[-1] == (len(tiles), 0)
    loads = []
    for (i, a), (j, b) in zip(at, at[1:]):
        assert (i, a) < (j, b)
        assert a == 0 or 0 < a < tiles[i]
        loads.append(sum(tiles[i:j]) - a + b)
    assert sum(loads) == sum(tiles)
    whole = max(sum(tiles[c::ctas]) for c in range(ctas))
    assert max(loads) < max(whole, max(tiles))


def test_few_items_are_cut_and_many_are_not():
    big = dict(h=16, hk=16, d=128, causal=True)
    assert plan("fl_fwd_split_plan", 148, b=4, sq=4096, sk=4096, **big) is None
    assert plan("fl_fwd_split_plan", 148, b=1, sq=256, sk=256, **big) is None
    assert plan("fl_fwd_split_plan", 148, b=1, sq=512, sk=16384, **big) is not None
    assert plan("fl_fwd_split_plan", 148, b=1, sq=512, sk=16384, left=4000, **big) is None
