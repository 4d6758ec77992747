"""The rings of the int4 GEMMs whose stages two groups of warps share: no order in which copies complete lets a group read a
stage before its chunk is there.  Ring sizes and the order of the waits are taken from the kernels' source; the barriers are
modelled by how many phases they have completed, and a parity wait passes whenever that count has the wanted parity."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "scratchy_b200", "csrc")


def size(text, name):
    """Every value a constant takes (a template's depend on its tile)."""
    m = re.search(rf"\b{name} = ([^;,]+)[;,]", text)
    return sorted({int(n) for n in re.findall(r"(?<![=!<>] )\b\d+\b", re.sub(r"TN == \d+", "", m.group(1)))})


def early_reads(packed, expanded, packed_first, chunks=12):
    """Chunks that some interleaving lets a group expand before their copy is complete."""
    passed = lambda done, phase: (done & 1) != (phase & 1)              # try_wait.parity: `done` phases complete
    start = (0, frozenset(), (0, 1), (0, 0), frozenset(), 0)            # copies issued and complete, chunk and stage of the groups, expanded, MMAs
    seen, todo, bad = {start}, [start], set()
    while todo:
        issued, copied, at, step, ready, mmas = todo.pop()
        copies = lambda s: sum(1 for c in copied if c % packed == s)
        freed = lambda s: sum(1 for c in ready if c % packed == s)      # (a group releases a packed stage with its expansion)
        used = lambda s: sum(1 for c in range(mmas) if c % expanded == s)
        after = []
        if issued < chunks and passed(freed(issued % packed), issued // packed + 1):
            after.append((issued + 1, copied, at, step, ready, mmas))
        after += [(issued, copied | {c}, at, step, ready, mmas) for c in range(issued) if c not in copied]
        for g in (0, 1):
            c = at[g]
            if c >= chunks:
                continue
            full = (copies(c % packed), c // packed)
            empty = (used(c % expanded), c // expanded + 1)
            waits = [full, empty] if packed_first else [empty, full]
            put = lambda t, v: tuple(v if i == g else t[i] for i in (0, 1))
            if step[g] < 2:
                if passed(*waits[step[g]]):
                    after.append((issued, copied, at, put(step, step[g] + 1), ready, mmas))
            else:
                if c not in copied:
                    bad.add(c)
                    continue
                after.append((issued, copied, put(at, c + 2), put(step, 0), ready | {c}, mmas))
        if mmas < chunks and mmas in ready:
            after.append((issued, copied, at, step, ready, mmas + 1))
        for s in after:
            if s not in seen:
                seen.add(s)
                todo.append(s)
    return bad


def test_the_model_sees_an_odd_ring_that_waits_for_its_copy_first():
    assert early_reads(3, 3, True) and not early_reads(4, 3, True) and not early_reads(3, 3, False)


@pytest.mark.parametrize("source,packed,expanded,full,empty", [
    ("affine_b4_gemm.cu", "A4G_SP", "A4G_SA", "pfull(s),", "aempty(grp)"),
    ("affine_b4_gemm_pair.cu", "A4P_SP", "A4P_SD", "pfull(sp)", "dempty(sd)"),
    ("affine_b4_skinny.cu", "kSP", "kSA", "pfull(s),", "aempty(a)")])
def test_no_group_reads_a_stage_before_its_copy(source, packed, expanded, full, empty):
    with open(os.path.join(CSRC, source)) as f:
        text = f.read()
    waits = [text.index("mbar_wait(" + name) for name in (full, empty)]
    for p in size(text, packed):
        for e in size(text, expanded):
            assert not early_reads(p, e, waits[0] < waits[1]), (p, e)
