"""Batch form of the expert kernels, against the CPU oracle: items of every size from one pair to more than a full one, the row lengths
the layout takes, runs that leave blocks without work and runs that cut an item, and the shared expert's batch kernel, with its
columns staged at once and in several panels. Bounds: operands are exact, activations are 24-bit fixed point per row and sums of up to 4096 products are
fp32, so a layer output is good to a few 1e-6 of its range; 2e-5 leaves room for the order of the sums."""
import numpy as np
import pytest

import dwarfstar_red_lite_b200 as rc
import oracle_lib as ol
import q6k_panels_lib as qp
from dwarfstar_red_lite_b200 import synth

pytestmark = pytest.mark.gpu


def _check(dims, ntok, seed, same_experts):
    layer = synth.moe_layer(seed, dims)
    x = np.random.default_rng(seed + 1).normal(0, 1, size=(ntok, dims.hidden)).astype(np.float32)
    logits = None
    if same_experts:                           # every token picks the same experts: items as full as ntok makes them
        logits = np.tile(np.random.default_rng(seed + 2).normal(0, 1, size=(1, dims.n_expert)), (ntok, 1)).astype(np.float32)
    m = rc.MoeLayer(layer, max_tokens=ntok)
    out = m.forward(x, logits_in=logits)
    m.close()
    for t in range(0, ntok, max(1, ntok // 4)):
        ref = ol.moe_ffn(layer, x[t], threads=4, logits_in=None if logits is None else logits[t])[0]
        assert np.max(np.abs(out[t] - ref)) <= 2e-5 * np.max(np.abs(ref)), t


@pytest.mark.parametrize("ntok", [2, 3, 4, 5, 7, 8, 9, 17])
def test_item_sizes(ntok):
    _check(synth.MoeDims(hidden=512, n_expert=16, top_k=4, ffn=512, ffn_sh=256), ntok, 700 + ntok, True)


@pytest.mark.parametrize("hidden,ffn", [(256, 256), (256, 1024), (1024, 256), (1024, 2048), (2048, 512)])
@pytest.mark.parametrize("ntok", [2, 40])
def test_row_lengths(hidden, ffn, ntok):
    _check(synth.MoeDims(hidden=hidden, n_expert=32, top_k=8, ffn=ffn, ffn_sh=256), ntok, 800 + ntok, False)


@pytest.mark.parametrize("hidden,ffn_sh", [(256, 512), (768, 256), (2048, 768), (2304, 256), (4096, 512)])
@pytest.mark.parametrize("ntok", [3, 8, 9, 37])
def test_shared_expert_panels(hidden, ffn_sh, ntok):
    _check(synth.MoeDims(hidden=hidden, n_expert=8, top_k=2, ffn=256, ffn_sh=ffn_sh), ntok, 900 + ntok, False)


# hidden, ffn_sh, tokens, panels of gate/up and of down: the second panel whole and ragged, column splits without work in a panel
@pytest.mark.parametrize("hidden,ffn_sh,ntok,panels", [(2048, 2048, 75, (2, 2)), (2048, 2048, 127, (2, 2)), (2048, 4096, 64, (2, 2)), (2048, 1536, 99, (2, 1)),
                                                      (4352, 512, 8, (2, 1)), (5120, 512, 8, (2, 1)), (8192, 256, 9, (2, 1))])
def test_shared_expert_in_several_panels(hidden, ffn_sh, ntok, panels):
    cut = lambda pair, nrows, ncols: -(-ncols // qp.plan(pair, nrows, ncols, ntok)["panel"])  # noqa: E731
    assert (cut(1, ffn_sh, hidden), cut(0, hidden, ffn_sh)) == panels
    _check(synth.MoeDims(hidden=hidden, n_expert=8, top_k=2, ffn=256, ffn_sh=ffn_sh), ntok, 1000 + ntok, False)
