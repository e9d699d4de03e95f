"""Kernels that may start before the kernels in front of them have ended (they call pdl_wait) read what those write by ordinary
loads through ordinary pointers: __ldg and const __restrict__ promise data that nobody writes during the kernel's life, and
neither the read-only path nor a load through a __restrict__ pointer is held back by griddepcontrol.wait.  Nothing here runs a
kernel: the sources are read."""

import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gpt_triton_b200", "csrc")
PARAMETERS = {"w", "b", "wte", "wpe", "gain", "bias", "fbias", "sink", "lambda"}  # of a model: no kernel of a pass writes them
OUTPUTS = {"out", "stats", "ext", "lse_out"}  # written, never read
# written as well as read, so never by the read-only path, and every read depends on a position that is loaded behind the wait
BEHIND_POSITION = {("attention_decode_kernel", "cache")}


def sources():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        text = re.sub(r"//[^\n]*", "", open(path).read())
        yield os.path.basename(path), text


def kernels(text):
    """(name, parameter list, body) of every __global__ function."""
    for m in re.finditer(r"__global__[^;{]*?\b(\w+)\(((?:[^(){}]|\([^()]*\))*)\)\s*\{", text):
        depth, i = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        yield m.group(1), m.group(2), text[m.end():i]


def early_kernels():
    return [(f, n, p) for f, t in sources() for n, p, body in kernels(t) if "pdl_wait()" in body]


def test_the_kernels_are_found():
    names = {n for _, n, _ in early_kernels()}
    assert {"gemm_tn_kernel", "gemm_narrow_kernel", "gemm_few_kernel", "ln_stats_few_rows_kernel", "attention_decode_kernel", "layernorm_vec_kernel",
            "embedding_kernel", "attention_sm100_kernel", "pair_attention_sm100_kernel", "argmax_reduce_kernel"} <= names


def test_no_restrict_on_what_other_kernels_write():
    for file, name, params in early_kernels():
        for prm in params.split(","):
            if "__restrict__" in prm:
                ident = re.search(r"(\w+)\s*$", prm).group(1)
                if (name, ident) in BEHIND_POSITION:
                    body = next(b for f, t in sources() if f == file for n, _, b in kernels(t) if n == name)
                    assert "const" not in prm and re.search(r"pdl_wait\(\);\s*const int pos = pos_dev\[0\];", body)
                    continue
                assert ident in (PARAMETERS if "const" in prm else OUTPUTS), f"{file}: {name}({prm.strip()})"


def test_read_only_loads_of_parameters_only():
    for file, text in sources():
        if "pdl_wait()" not in text:
            continue
        for arg in re.findall(r"__ldg\(((?:[^()]|\([^()]*\))*)\)", text):
            assert PARAMETERS & set(re.findall(r"\w+", arg)), f"{file}: __ldg({arg})"


def test_every_kernel_with_the_attribute_waits():
    """What LaunchSetup launches (it sets the attribute) calls pdl_wait, unless the call switches the attribute off."""
    early = {n for _, n, _ in early_kernels()}
    for file, text in sources():
        for m in re.finditer(r"LaunchSetup ls\((?P<args>[^;]*)\);(?P<rest>.{0,700})", text, re.S):
            if re.search(r",\s*false$", m.group("args")):
                continue
            launched = re.findall(r"(?:cudaLaunchKernelEx\(&ls\.cfg,\s*)(\w+)", m.group("rest").split("LaunchSetup")[0])
            launched = set(launched)
            if "kernel" in launched:  # (a variable that names the instantiation)
                launched = launched - {"kernel"} | set(re.findall(r"\bkernel = (\w+)<", text))
            assert launched and launched <= early, (file, launched)
