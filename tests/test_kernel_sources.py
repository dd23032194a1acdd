"""What holds of every kernel source, on the CPU."""
import os
import re

from mini_inference_b200.ops.build import CSRC


def kernels(name):
    """{kernel: (its parameters, its body)} of a file of csrc/."""
    with open(os.path.join(CSRC, name)) as f:
        text = re.sub(r"//[^\n]*", "", f.read())
    out = {}
    for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*)?(\w+)\s*\(", text):
        def closing(at, pair):
            depth = 1
            while depth:
                depth += (text[at] == pair[0]) - (text[at] == pair[1])
                at += 1
            return at
        end = closing(m.end(), "()")
        body = text.index("{", end)
        out[m.group(1)] = ([" ".join(p.split()) for p in text[m.end():end - 1].split(",")], text[body:closing(body + 1, "{}")])
    return out


def test_what_the_kernel_ahead_writes_is_not_promised_to_stay():
    """A kernel that starts while the one ahead runs may not have a __restrict__ pointer to what that one writes: its loads could be moved ahead of the wait."""
    for file, kernel, names in (("state_chunks.cu", "chunk_scan_kernel", ("sums",)), ("state_chunks.cu", "chunk_out_kernel", ("before",)),
                                ("gemm_f32_tc.cu", "gemm_f32_tc_kernel", ("token_flag",))):
        params, _ = kernels(file)[kernel]
        for name in names:
            (param,) = [p for p in params if re.search(rf"\b{name}$", p)]
            assert "__restrict__" not in param, (file, kernel, param)


# what a kernel with a bare wait may read by __restrict__ pointers: weights and a step's metadata, and what was complete before the kernel ahead began
THERE_BEFORE = {"attn_prefill_tc_kernel": {"tiles", "seg_q_start", "seg_pos0", "block_table", "table_rows"}, "gemm_f32_tc_kernel": {"A", "W"},
                "gemm_skinny_kernel": {"W"}, "chunk_scan_kernel": {"decay", "seg_q_start", "seg_slot"}, "chunk_out_kernel": {"in", "decay", "seg_q_start"}}


def test_waits_name_what_the_kernel_ahead_writes():
    """... where pointers to it are __restrict__ ones: pdl_wait(pointers) ends what the compiler knows of them."""
    waiting = 0
    for file in sorted(f for f in os.listdir(CSRC) if f.endswith(".cu")):
        for kernel, (params, body) in kernels(file).items():
            if "pdl_wait(" not in body:
                continue
            waiting += 1
            read = {p.split()[-1] for p in params if "__restrict__" in p and p.startswith("const")}
            named = [w for w in re.findall(r"pdl_wait\(([^)]*)\)", body)]
            if not all(named):
                assert read <= THERE_BEFORE.get(kernel, set()), (file, kernel, read)
            for name in (n.strip() for w in named for n in w.split(",") if w):
                assert re.search(rf"\b{name}\b", " ".join(params)) or re.search(rf"\*\s*{name} =", body), (file, kernel, name)
    assert waiting > 25
