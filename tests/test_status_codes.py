"""The code that a kernel records when it gives up on a bounded wait names the kernel: no two sources share one."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "savanna_b200", "csrc")


def test_status_codes_are_disjoint():
    sources = {os.path.basename(f): open(f).read() for f in glob.glob(os.path.join(CSRC, "*.cu*"))}
    # enum constants and constexpr words, and the largest number added to each
    bases = [(name, int(v, 0), f) for f, s in sources.items()
             for name, v in re.findall(r"\b(ST_[A-Z_]+) = (0x[0-9a-f]+|\d+)", s)]
    assert {"ST_OK", "ST_ATTN", "ST_MX", "ST_MR_FWD", "ST_MR_BWD"} <= {n for n, _, _ in bases}
    owner = {}
    for name, base, where in bases:
        added = [int(n) for s in sources.values() for n in re.findall(rf"\b{name} \+ (\d+)", s)]
        if name == "ST_MR_BWD":                           # numbered in the calls of the kernel's own wait()
            added += [int(n) for n in re.findall(r"wait\([A-Z][^;]*?, (\d+)\)", sources["mr_conv_umma.cu"])]
            assert len(set(added)) >= 11
        for code in range(base, base + max(added, default=0) + 1):
            assert code < 256 and code not in owner, f"{code:#x} of {name} in {where} is {owner.get(code)}'s"
            owner[code] = name
