"""A layer's forward of a few tokens replayed from a CUDA graph: the side stream's join and the kernels that are launched ahead of their
predecessor's end must stay ordered in the graph, for inputs that change between replays."""
import pytest
import torch

import dwarfstar_red_lite_b200 as rc
from dwarfstar_red_lite_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("t", [synth.IQ2_XXS, synth.IQ3_S])
@pytest.mark.parametrize("ntok", [1, 2, 3, 6, 16, 17])
def test_replayed_forward(t, ntok):
    dims = synth.MoeDims(hidden=1024, n_expert=32, top_k=10, ffn=512, ffn_sh=512, type_gu=t, type_down=t)
    layers = [rc.MoeLayer(synth.moe_layer(20 + i, dims), max_tokens=ntok) for i in range(2)]
    g = torch.Generator(device="cuda")
    g.manual_seed(ntok)
    x, mid, out, resid = (torch.randn(ntok, dims.hidden, device="cuda", generator=g) for _ in range(4))
    s = torch.cuda.Stream()

    def step():
        layers[0].forward_device(ntok, x.data_ptr(), mid.data_ptr(), s.cuda_stream, resid_ptr=resid.data_ptr())
        layers[1].forward_device(ntok, mid.data_ptr(), out.data_ptr(), s.cuda_stream)

    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        step()
        s.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s):
            step()
        for _ in range(4):
            x.copy_(torch.randn(ntok, dims.hidden, device="cuda", generator=g))
            step()
            want = out.clone()
            out.zero_(), mid.zero_()
            graph.replay()
            graph.replay()
            s.synchronize()
            assert torch.equal(out, want)
    del graph
    for m in layers:
        m.close()
