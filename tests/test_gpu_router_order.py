"""Router logits of a small batch request their weights ahead of the wait for the kernel before them; the rows they multiply are what that
kernel writes, and must be read behind it."""
import pytest
import torch

import dwarfstar_red_lite_b200 as rc
from dwarfstar_red_lite_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ntok", [2, 8, 16])
@pytest.mark.parametrize("hidden", [256, 2048])
def test_rows_of_the_kernel_before(ntok, hidden):
    dims = synth.MoeDims(hidden=hidden, n_expert=32, top_k=4, ffn=256, ffn_sh=256)
    layers = [rc.MoeLayer(synth.moe_layer(40 + i, dims), max_tokens=ntok) for i in range(3)]
    g = torch.Generator(device="cuda")
    g.manual_seed(ntok)
    rows = torch.empty(4, ntok, hidden, device="cuda")
    s = torch.cuda.Stream()

    def chain(wait):
        for i, m in enumerate(layers):       # a layer's rows are the outputs of the layer before
            m.forward_device(ntok, rows[i].data_ptr(), rows[i + 1].data_ptr(), s.cuda_stream)
            if wait:
                s.synchronize()
        s.synchronize()
        return rows.clone()

    for _ in range(20):
        rows[0] = torch.randn(ntok, hidden, device="cuda", generator=g)
        torch.cuda.synchronize()
        want = chain(True)
        rows[1:].zero_()
        torch.cuda.synchronize()
        assert torch.equal(chain(False), want)
    for m in layers:
        m.close()
