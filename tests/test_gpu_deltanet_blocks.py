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
