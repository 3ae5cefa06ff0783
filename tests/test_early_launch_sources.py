"""A kernel may be launched ahead of its predecessor's end and waits for it inside. What the predecessor may have written is then not
memory that nobody writes while the kernel runs, which a const __restrict__ argument would let the compiler take it for (non-coherent loads, which
move across the wait). So only weights that were in place before are such arguments; of the file-layout kernels every input is, as they follow
copies, which end first."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dwarfstar_red_lite_b200", "csrc")
RESIDENT = {"k_router_logits": {"w"}, "k_vec_sigmoid": {"w"}, "k_rmsnorm": {"w"}, "k_attn_prep": {"qn", "kn"}, "k_embed_row": {"base"}, "k_dn_prep": {"conv_kernel", "dt_bias", "ssm_a"},
            "k_dn_tail": {"norm_w"}, "k_dn_step": {"conv_kernel", "dt_bias", "ssm_a", "norm_w"}, "k_dn_prep_seq": {"conv_kernel", "dt_bias", "ssm_a"},
            "k_nib_repack": {"raw"}}      # never launched early
KERNEL = re.compile(r"__global__[^;{]*?\b(k_\w+)\(([^{]*?)\)\s*\{", re.S)
CONST_RESTRICT = re.compile(r"const\s+[\w:]+\s*\*\s*__restrict__\s+(\w+)")


def test_inputs_of_kernels_are_read_behind_the_wait():
    kernels, wrong = 0, []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        if path.endswith("redcuda_kquants.cu"):
            continue
        for name, params in KERNEL.findall(open(path).read()):
            kernels += 1
            wrong += [(name, p) for p in CONST_RESTRICT.findall(params) if p not in RESIDENT.get(name, ())]
    assert kernels >= 40 and not wrong, wrong
