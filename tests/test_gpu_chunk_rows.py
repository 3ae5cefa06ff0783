"""Rows handed to the chunk form of the expert kernels: they may begin at any float, as long as their stride is a multiple of four."""
import numpy as np
import pytest
import torch

import dwarfstar_red_lite_b200 as rc
from dwarfstar_red_lite_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hidden,ffn", [(512, 256), (1024, 512)])
@pytest.mark.parametrize("shift", [0, 1, 2, 3])
def test_unaligned_rows(hidden, ffn, shift, monkeypatch):
    monkeypatch.setenv("RC_MOE_TC_MIN", "1")
    ntok, n_expert, k = 40, 8, 4
    m = rc.MoeLayer(synth.moe_layer(9, synth.MoeDims(hidden=hidden, n_expert=n_expert, top_k=k, ffn=ffn, ffn_sh=256)), max_tokens=ntok)
    rng = np.random.default_rng(shift)
    stride = hidden + 4
    x = torch.from_numpy(rng.normal(0, 1, size=(ntok, hidden)).astype(np.float32)).cuda()
    ids = torch.from_numpy(np.stack([rng.choice(n_expert, k, replace=False) for _ in range(ntok)]).astype(np.int32)).cuda()
    w = torch.from_numpy(rng.uniform(0.1, 1, size=(ntok, k)).astype(np.float32)).cuda()
    buf = torch.zeros(ntok * stride + 4, device="cuda")
    rows = buf[shift:shift + ntok * stride].view(ntok, stride)
    rows[:, :hidden] = x
    want, got = torch.empty(ntok, hidden, device="cuda"), torch.empty(ntok, hidden, device="cuda")
    s = torch.cuda.current_stream().cuda_stream
    m.partial_device(ntok, x.data_ptr(), hidden, ids.data_ptr(), w.data_ptr(), k, want.data_ptr(), s)
    m.partial_device(ntok, rows.data_ptr(), stride, ids.data_ptr(), w.data_ptr(), k, got.data_ptr(), s)
    torch.cuda.synchronize()
    assert torch.equal(want, got)
    m.close()
