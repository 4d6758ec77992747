"""Rules of the hardware that no result shows reliably, checked on the kernels' source: each would be undefined behaviour or a
hang that depends on what else is resident."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "scratchy_b200", "csrc")


def sources():
    out = {}
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cuh")):
            with open(os.path.join(CSRC, name)) as f:
                out[name] = re.sub(r"//[^\n]*", "", f.read())
    return out


def block(text, start):
    """The braces' content that opens first from `start` on."""
    lo = at = text.index("{", start)
    depth = 0
    while True:
        depth += {"{": 1, "}": -1}.get(text[at], 0)
        at += 1
        if depth == 0:
            return text[lo:at]


def kernels():
    """(file, name, body, the device functions of the repository that it calls, asm text included)"""
    texts = sources()
    functions = {}
    for text in texts.values():
        for m in re.finditer(r"__device__ __forceinline__ [\w:<> ]+?[ *&](\w+)\(", text):
            functions.setdefault(m.group(1), []).append(block(text, m.end()))
    for name, text in texts.items():
        for m in re.finditer(r"__global__[^;{]*?\b(\w+_kernel)\(", text):
            body = block(text, m.end())
            called = "".join(f for n in sorted(set(re.findall(r"\b(\w+)\(", body))) for f in functions.get(n, []))
            yield name, m.group(1), body, body + called


def test_warps_are_whole_at_aligned_barriers():
    """`barrier.cluster.*.aligned` and tcgen05's `.sync.aligned` forms are executed by a whole warp: where single lanes had roles
    of their own before, a __syncwarp, or a barrier of the CTA, comes first."""
    texts = sources()
    syncs = {m.group(1) for t in texts.values() for m in re.finditer(r"(\w+)\(\) \{\s*asm volatile\(\"barrier\.cluster\.arrive\.release\.aligned", t)}
    assert len(syncs) >= 6
    checked = 0
    for file, kernel, body, _ in kernels():
        lone = [m.end() for m in re.finditer(r"if \((?:\(?threadIdx\.x == 0|lane [=<]=? ?\w+|lane == 0 && \w+ == 0)\)", body)]
        calls = [m.start() for s in syncs for m in re.finditer(rf"\b{s}\(\)", body)] + [m.start() for m in re.finditer(r"\bskinny_finish\(", body)]
        for at in calls:
            before = [p for p in lone if p < at]
            if not before:
                continue
            # the nearest convergence before the barrier, past the last role of a single lane
            gap = body[before[-1]:at]
            assert re.search(r"__syncwarp\(\)|__syncthreads\(\)|bar\.sync", gap), (file, kernel, body[at - 200:at])
            checked += 1
    assert checked >= 6


def test_dependents_start_after_the_tensor_memory_is_held():
    """A CTA of the next kernel that takes TMEM first would wait for this kernel's end, and this kernel's CTA for that TMEM: a
    kernel lets its dependents start only when the allocation is behind it (or on a way out that takes none)."""
    checked = set()
    for file, kernel, body, _ in kernels():
        if "tmem_alloc" not in body:
            continue
        held = body.index("*tmem_slot")
        for m in re.finditer(r"pdl_trigger\(\)|griddepcontrol\.launch_dependents", body):
            leaves = re.match(r"[^{}]*\breturn;", body[m.end():])
            assert m.start() > held or leaves, (file, kernel)
            checked.add(kernel)
    assert {"latent_prefill_kernel", "window_prefill_kernel", "dense_gemm_kernel", "dense_skinny_kernel", "affine_b4_skinny_kernel"} <= checked
