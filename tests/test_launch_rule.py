"""Kernels that are launched behind one another without waiting for the earlier one's flush (launch_after) must wait for it themselves, first of all, and must not let
their successor start before their end: read from the sources."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "fasttalk_llm_microservice_b200", "csrc")


def sources():
    return {f: re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, f)).read()) for f in sorted(os.listdir(CSRC)) if f.endswith((".cu", ".cuh"))}


def body_from(text, at):
    """The text between the first brace behind `at` and the one that closes it."""
    start = text.index("{", at)
    depth = 0
    for i in range(start, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[start + 1:i]
    raise AssertionError("no closing brace")


def kernel_bodies(text):
    found = {}
    for m in re.finditer(r"__global__\s+void\s+(?:__\w+__\s*\((?:[^()]|\((?:[^()]|\([^()]*\))*\))*\)\s*)*(\w+)\s*\(", text):
        found[m.group(1)] = body_from(text, m.end())
    return found


def launched_behind(text):
    """Names that reach launch_after: its first argument, and the kernels handed to a helper that passes them on."""
    names = set(re.findall(r"launch_after\(\s*(\w+)", text)) - {"void"}
    if "kernel" in names:
        names.remove("kernel")
        names |= {m for m in re.findall(r"\bstep\((\w+)<", text)}
    return names


def test_kernels_launched_behind_others_wait_first_and_release_nobody():
    seen = 0
    for f, text in sources().items():
        kernels = kernel_bodies(text)
        for name in launched_behind(text):
            if f == "common.cuh":
                continue
            assert name in kernels, (f, name)
            body = kernels[name]
            assert "pdl_wait();" in body, (f, name)
            assert "pdl_launch_dependents" not in body and "launch_dependents" not in body, (f, name)
            # ahead of the wait: nothing that could read or write global memory.  Most kernels wait in their first line; those on the tensor cores first set up their
            # barriers and tensor memory
            ahead = body[:body.index("pdl_wait();")]
            if ahead.strip():
                assert "tmem_alloc" in ahead, (f, name)
                for word in ("tma_load", "tma_tile", "tma_bulk", "cp_async", "__ldg", "__ldcg", "atomic", "load_f4", "reinterpret_cast<const"):
                    assert word not in ahead, (f, name, word)
            seen += 1
    assert seen > 40


def test_programmatic_launches_elsewhere_wait_as_well():
    """Every kernel of a file that asks for a programmatic launch by its own attribute waits somewhere, and the few-token product of a cluster, which runs between kernels
    that are launched behind one another, releases nobody."""
    seen = set()
    for f, text in sources().items():
        if "cudaLaunchAttributeProgrammaticStreamSerialization" in text and f != "common.cuh":
            bodies = kernel_bodies(text)
            for name in re.findall(r"cudaLaunchKernelEx\(&cfg,\s*(?:[^,?]*\?\s*)?(\w+)", text):
                assert "pdl_wait();" in bodies[name], (f, name)
                seen.add(name)
            if f == "gemm_plain.cu":
                assert "launch_dependents" not in bodies["gemm_plain_few_kernel"]
    assert seen >= {"attn_decode_kernel", "attn_prefill_kernel", "attn_prefill_tc_kernel", "gemm_bf16_tcgen05_kernel", "gemm_pair_kernel", "gemm_plain_few_kernel"}, seen
