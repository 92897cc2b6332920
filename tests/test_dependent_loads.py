"""Kernels whose launches overlap must not read, with non-coherent loads, what the launch before them writes (the rule at
``grid_dependency_wait``): every such load in the sources is listed here with the reason why it may stay."""

import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "miniworld_b200" / "csrc"

# (file, text of the line) -> why the operand is older than the direct predecessor
ALLOWED = {
    ("backward.cuh", "asm volatile(\"ld.global.nc.v8.b32"): "the load of ldg_32B, whose only caller is ldg_chunks",
    ("backward.cuh", "for (int c = 0; c < CHUNKS; ++c) out[c] = __ldg(p + c);"): "ldg_chunks",
    ("backward.cuh", "ldg_chunks(reinterpret_cast<const uint4*>(p.drop_scale"): "an argument; the set-up launch starts after it is written",
    ("backward.cuh", "__ldg((u < 4 ? t0 : t1) + at"): "the forward's tri; likewise",
    ("backward.cuh", "const float4 st = __ldg(sp + q)"): "statistics, written three launches before",
    ("backward.cuh", "tv[k] = __ldg(t + base"): "the forward's tri",
    ("backward.cuh", "rstd_in = __ldg(p.rstd"): "written by the epilogue's backward, contractions in between",
    ("backward.cuh", "? __ldg(dy + i + u * step)"): "the set-up launch, which does not overlap",
    ("transition_backward.cuh", "rstd_in = __ldg(p.rstd + gp);"): "written by the first of four launches, read by the last",
}


def test_non_coherent_loads_are_the_listed_ones():
    found = []
    for path in sorted(CSRC.glob("*.cuh")) + sorted(CSRC.glob("*.inc")) + sorted(CSRC.glob("*.cu")):
        for line in path.read_text().splitlines():
            code = line.split("//")[0]
            if re.search(r"__ldg\(|ld\.global\.nc|ldg_chunks\(", code) and "__forceinline__" not in code:
                if code.strip() == "asm volatile(":
                    continue
                found.append((path.name, code.strip()))
    unknown = [f for f in found if not any(f[0] == a[0] and a[1] in f[1] for a in ALLOWED)]
    assert not unknown, unknown
    unused = [a for a in ALLOWED if not any(f[0] == a[0] and a[1] in f[1] for f in found)]
    assert not unused, unused


def test_packed_constants_are_read_past_l1():
    """What one call of a chain of overlapped launches packs, the next one on the same workspace packs again, with no ordinary launch
    in between that would empty L1."""
    reads = []
    for path in sorted(CSRC.glob("prologue*")) + sorted(CSRC.glob("epilogue*")):
        for line in path.read_text().splitlines():
            code = line.split("//")[0]
            if re.search(r"\bp\.(c3|c3_a|c3_b|d1|ln_w|ln_b)\b", code):
                reads.append((path.name, code.strip()))
    assert {name for name, _ in reads} == {"prologue_stats.inc", "prologue_epilogue.inc", "epilogue.cuh", "epilogue_wide.cuh"}
    assert not [r for r in reads if "__ldcg(" not in r[1]]
