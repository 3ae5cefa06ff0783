"""What the host calls for a layer of a small batch beside its launches: a kernel's attributes are set when the layer is created, except the
two of the expert kernels."""
import pytest
import torch

import dwarfstar_red_lite_b200 as rc
from dwarfstar_red_lite_b200 import synth

pytestmark = pytest.mark.gpu


def test_attributes_are_not_set_at_every_launch():
    from torch.profiler import ProfilerActivity, profile
    dims = synth.MoeDims(hidden=512, n_expert=16, top_k=4, ffn=256, ffn_sh=256)
    m = rc.MoeLayer(synth.moe_layer(5, dims), max_tokens=6)
    x = torch.randn(6, dims.hidden, device="cuda")
    out = torch.empty_like(x)
    stream = torch.cuda.current_stream().cuda_stream
    calls = 4
    m.forward_device(6, x.data_ptr(), out.data_ptr(), stream)
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as p:
        for _ in range(calls):
            m.forward_device(6, x.data_ptr(), out.data_ptr(), stream)
        torch.cuda.synchronize()
    m.close()
    names = [e.name for e in p.events()]
    if not any(n.startswith("cudaLaunchKernel") for n in names):
        pytest.skip("the profiler sees no runtime calls here")
    assert sum(n == "cudaFuncSetAttribute" for n in names) <= 2 * calls


def test_the_router_of_a_chunk_sets_none(monkeypatch):
    from torch.profiler import ProfilerActivity, profile
    monkeypatch.setenv("RC_ROUTER_I8_MIN", "2")
    dims = synth.MoeDims(hidden=256, n_expert=128, top_k=2, ffn=256, ffn_sh=256)
    m = rc.MoeLayer(synth.moe_layer(5, dims), max_tokens=300)
    x = torch.randn(300, dims.hidden, device="cuda")
    ids, w = torch.empty(300, 2, dtype=torch.int32, device="cuda"), torch.empty(300, 2, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    m.route_device(300, x.data_ptr(), ids.data_ptr(), w.data_ptr(), stream)
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CPU, ProfilerActivity.CUDA]) as p:
        m.route_device(300, x.data_ptr(), ids.data_ptr(), w.data_ptr(), stream)
        torch.cuda.synchronize()
    m.close()
    names = [e.name for e in p.events()]
    if not any(n.startswith("cudaLaunchKernel") for n in names):
        pytest.skip("the profiler sees no runtime calls here")
    assert "cudaFuncSetAttribute" not in names
