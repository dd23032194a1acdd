"""What holds of every kernel source, on the CPU."""
import os
import re

from mini_inference_b200.ops.build import CSRC


def kernels(name):
    """{kernel: its parameters, one per entry} of a file of csrc/."""
    with open(os.path.join(CSRC, name)) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    out = {}
    for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*)?(\w+)\s*\(", text):
        depth, end = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[end], 0)
            end += 1
        out[m.group(1)] = [" ".join(p.split()) for p in text[m.end():end - 1].split(",")]
    return out


def test_what_the_kernel_ahead_writes_is_not_promised_to_stay():
    """A kernel that starts while the one ahead runs may not have a __restrict__ pointer to what that one writes: its loads could be moved ahead of the wait."""
    for file, kernel, names in (("state_chunks.cu", "chunk_scan_kernel", ("sums",)), ("state_chunks.cu", "chunk_out_kernel", ("before",)),
                                ("gemm_f32_tc.cu", "gemm_f32_tc_kernel", ("token_flag",))):
        params = kernels(file)[kernel]
        for name in names:
            (param,) = [p for p in params if re.search(rf"\b{name}$", p)]
            assert "__restrict__" not in param, (file, kernel, param)
