"""The one-launch DeltaNet step: one to eight value heads per key head, state sizes 32 to 128, other conv lengths, and the forms
beyond it (nine value heads per key head, state size 256)."""
import numpy as np
import pytest

import dwarfstar_red_lite_b200 as rc
import oracle_lib as ol

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S,groups,rank,d_conv", [(128, 2, 4, 4), (128, 3, 3, 4), (64, 2, 16, 4), (32, 4, 8, 4), (128, 2, 4, 3), (64, 2, 2, 2), (32, 1, 9, 4), (256, 2, 4, 4)])
@pytest.mark.parametrize("batch", [1, 3])
def test_deltanet_step_forms(S, groups, rank, d_conv, batch):
    rng = np.random.default_rng(S + rank + d_conv)
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
