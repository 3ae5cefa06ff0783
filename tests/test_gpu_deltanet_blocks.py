"""The DeltaNet step at every number of blocks per value head that its launch rule knows (value heads x batch against the chip), and
with clusters of 3, 5, 6, 7 and 8 blocks."""
import numpy as np
import pytest

import dwarfstar_red_lite_b200 as rc
import oracle_lib as ol

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("groups,rank,batch", [(16, 32, 1), (16, 32, 3), (16, 32, 4), (16, 32, 5), (16, 32, 6), (16, 32, 7), (16, 32, 9), (16, 32, 10), (16, 32, 14), (16, 16, 7), (8, 24, 3), (2, 6, 1),
                                               (8, 32, 5), (2, 10, 2), (3, 18, 2), (1, 7, 2), (2, 16, 2)])
@pytest.mark.parametrize("d_conv", [4, 3])
def test_blocks_per_head(groups, rank, batch, d_conv):
    S = 128
    rng = np.random.default_rng(batch + rank + d_conv)
    d_inner, channels = rank * S, 2 * S * groups + rank * S
    f = lambda *s, k=1.0: (rng.normal(0, 1, size=s) * k).astype(np.float32)  # noqa: E731
    p = dict(d_conv=d_conv, d_state=S, n_group=groups, dt_rank=rank, d_inner=d_inner, channels=channels, rms_eps=1e-6, conv_kernel=f(channels, d_conv, k=0.5), dt_bias=f(rank),
             ssm_a=-np.exp(f(rank, k=0.5)), ssm_norm=1.0 + f(S, k=0.1))
    qkv, z, ba = f(batch, channels), f(batch, d_inner), f(batch, 2 * rank)
    conv, rec = f(batch, channels, d_conv - 1), f(batch, rank, S, S, k=0.05)
    cg, rg = conv.copy(), rec.copy()
    out = rc.deltanet_step(p, qkv, z, ba, cg, rg)
    for b in range(batch):
        ref = ol.deltanet_mid(p, qkv[b], z[b], ba[b], conv[b], rec[b])
        assert np.array_equal(cg[b], conv[b])                                        # the oracle moved its window in place
        # tolerances of the reference's stage tools (native/redlite_native_deltanet_state_cli.c:267-269); the output adds a norm over the head
        assert np.all(np.abs(rg[b] - rec[b]) <= 3e-6 + 3e-5 * np.abs(rec[b]))
        assert np.max(np.abs(out[b] - ref)) <= 2e-5 * np.max(np.abs(ref)) + 1e-7


@pytest.mark.parametrize("batch", [1, 3])
def test_output_in_the_input(batch):
    """out may lie in qkv: every block's inputs are read before any output is written."""
    import ctypes as C
    import torch
    from dwarfstar_red_lite_b200 import redcuda
    S, groups, rank = 128, 16, 32
    d_inner, channels = rank * S, 2 * S * groups + rank * S
    g = torch.Generator(device="cuda")
    g.manual_seed(batch)
    r = lambda *s: torch.randn(*s, device="cuda", generator=g)  # noqa: E731
    arr = [r(channels, 4) * 0.5, r(rank), -torch.exp(r(rank) * 0.5), 1.0 + 0.1 * r(S)]
    P = redcuda.DeltanetParams(4, S, groups, rank, d_inner, channels, 1e-6, *[C.cast(a.data_ptr(), redcuda.f32p) for a in arr])
    qkv, z, ba, conv, rec = r(batch, channels), r(batch, d_inner), r(batch, 2 * rank), r(batch, channels, 3), r(batch, rank, S, S) * 0.05
    lib = rc.lib()

    def step(inputs, out_ptr):
        c, s = conv.clone(), rec.clone()
        torch.cuda.synchronize()
        assert lib.redcuda_deltanet_step_noalloc(C.byref(P), batch, inputs.data_ptr(), z.data_ptr(), ba.data_ptr(), c.data_ptr(), s.data_ptr(), out_ptr, None) == 1
        torch.cuda.synchronize()
        return c, s

    out, buf = torch.empty(batch, d_inner, device="cuda"), qkv.clone()
    c0, s0 = step(qkv, out.data_ptr())
    c1, s1 = step(buf, buf.data_ptr())
    got = buf.view(-1)[:batch * d_inner].view(batch, d_inner)
    assert torch.equal(c0, c1)
    # the forms differ in the order of a few 32-bit sums only
    assert torch.allclose(s0, s1, rtol=3e-5, atol=3e-6) and torch.max(torch.abs(got - out)) <= 2e-5 * torch.max(torch.abs(out))
