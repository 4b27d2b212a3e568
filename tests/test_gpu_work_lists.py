"""Work lists made by a block of the quantiser's launch against those of a launch of their own."""
import pytest
import torch

from inputs import attention_inputs
from launches import launches
from test_gpu_call_path import _state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lens,kw", [
    ([1], {}),
    ([128, 129, 1, 127, 256, 257], {}),
    ([1] * 127 + [128 * 130], {}),                                     # more tiles than threads, a document over several chunks
    ([700, 3, 1300, 129], dict(window_size=(200, 0))),
    ([640, 128, 256], dict(deterministic=True)),                       # document order
    ([1] * 1536, {}),                                                  # the most documents that the quantiser's block takes at one head
    ([1] * 1537, {}),
    ([1] * 4096, {}),
    ([1] * 4097, {}),
])
def test_lists_equal_those_of_their_own_launch(lens, kw):
    from flamia_blackwell_attention_b200 import _lib as L, kernels as K
    q, k, v, _ = (t[0].cuda() for t in attention_inputs(1, sum(lens), 1, 1, 64, seed=7))
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device="cuda")
    _, _, st = _state("fp8", q, k, v, [cu, cu], cu_seqlens_q=cu, cu_seqlens_k=cu, max_seqlen_q=max(lens), max_seqlen_k=max(lens), **kw)
    start, length, row_map, _, _, got = st[-7:-1]
    want, status = torch.empty_like(got), torch.zeros(1, dtype=torch.int32, device="cuda")
    left = kw["window_size"][0] + 1 if "window_size" in kw else 0
    L.check(L.load().fl_doc_work(L.ptr(start), L.ptr(length), len(lens), row_map.numel(), left, 0, 1, int(kw.get("deterministic", False)),
                                 L.ptr(want), L.ptr(status), K._stream()), "fl_doc_work")
    assert status.item() == 0 and torch.equal(got[:4], want[:4])
    tiles = row_map.numel() // 128
    for part, n in enumerate(got[:2].tolist()):
        a, b = (x[4:4 + 8 * tiles].view(2, tiles, 4)[part, :n].tolist() for x in (got, want))
        assert sorted(a) == sorted(b)              # (equal costs may change places, except in document order)
        if kw.get("deterministic"):
            assert a == b


@pytest.mark.parametrize("docs,rows,h,d,own", [
    (1536, 128, 1, 64, False), (1537, 128, 1, 64, True), (2048, 128, 4, 64, True), (2048, 128, 6, 64, False), (4096, 128, 6, 64, True),
    (4096, 128, 8, 64, False), (4097, 128, 8, 64, True),
    (2200, 64, 1, 64, False), (2300, 64, 1, 64, True), (2561, 1, 1, 64, True), (4096, 1, 2, 64, False), (4096, 32, 2, 64, True),
    (3000, 128, 1, 128, True), (2048, 128, 1, 128, False), (4096, 128, 2, 128, False),
])
def test_long_lists_of_few_heads_are_a_launch_of_their_own(docs, rows, h, d, own, tmp_path):
    import flamia_blackwell_attention_b200 as F
    n = docs * rows
    q, k, v = (torch.zeros(n, i, d, dtype=torch.bfloat16, device="cuda") for i in (h, 1, 1))
    maps = F.DocMaps.from_cu_seqlens(torch.arange(0, n + 1, rows, dtype=torch.int32), padded_size=docs * 128).to("cuda")
    with torch.no_grad():
        names = [name for name, _, _ in launches(lambda: F.flash_attn_fp8(q, k, v, causal=True, doc_maps=maps), tmp_path)]
    assert any("quant_rows" in name for name in names) and any("doc_work" in name for name in names) == own, names
