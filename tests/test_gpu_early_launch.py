"""Kernels that are launched ahead of their predecessor's end give what they give when launched behind it (RC_PDL=0), for batches of every
form, with a new batch right behind the one before."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SIZES = (2, 3, 9, 40, 130)
CODE = """
import sys
import numpy as np
import torch
import dwarfstar_red_lite_b200 as rc
from dwarfstar_red_lite_b200 import synth
outs = []
for t in (synth.IQ2_XXS, synth.IQ3_S):
    dims = synth.MoeDims(hidden=512, n_expert=32, top_k=8, ffn=512, ffn_sh=256, type_gu=t, type_down=t)
    layers = [rc.MoeLayer(synth.moe_layer(70 + i, dims), max_tokens=%d) for i in range(2)]
    for n in %r:
        g = torch.Generator(device="cuda")
        g.manual_seed(n)
        x = torch.randn(16, n, 512, device="cuda", generator=g)
        mid, out = torch.empty_like(x), torch.empty_like(x)
        s = torch.cuda.current_stream().cuda_stream
        for i in range(16):
            layers[0].forward_device(n, x[i].data_ptr(), mid[i].data_ptr(), s)
            layers[1].forward_device(n, mid[i].data_ptr(), out[i].data_ptr(), s)
        torch.cuda.synchronize()
        outs.append(out.cpu().numpy())
np.savez(sys.argv[1], *outs)
""" % (max(SIZES), SIZES)


def test_same_results_launched_early_and_late(tmp_path):
    got = []
    for name, env in (("early", {}), ("late", {"RC_PDL": "0"})):
        path = str(tmp_path / (name + ".npz"))
        clean = {k: v for k, v in os.environ.items() if k != "RC_PDL"}
        subprocess.run([sys.executable, "-c", CODE, path], check=True, cwd=ROOT, env=dict(clean, **env), timeout=300)
        got.append(np.load(path))
    for k in got[0].files:
        assert np.array_equal(got[0][k], got[1][k]), k
