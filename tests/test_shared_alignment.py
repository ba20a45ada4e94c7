"""ld, ldg and st (csrc/field.cuh) move a field element as two 16-byte words, but
the element's own type is aligned to four: a static shared array that they (or
the warp-per-point formulas of csrc/curve.cuh, which use them) access must ask
for 16 bytes itself.  Read from the sources: a misaligned access faults."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "halo2-gpu_b200", "csrc")
DECL = re.compile(r"^\s+__shared__\s+(__align__\((\d+)\)\s+)?(Fr|Fq|F|G1Xyzz|G1Affine)\s+(\w+)(\[[^;]*)?;")


def test_shared_elements_moved_by_vectors_are_aligned():
    seen, bad = 0, []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu*"))):
        lines = open(path).read().split("\n")
        for i, line in enumerate(lines):
            m = DECL.match(line)
            if not m:
                continue
            end = next(j for j in range(i, len(lines)) if lines[j].startswith("}"))
            name = m.group(4)
            vec = re.compile(r"\b(ld|ldg|st|ld_xyzz|st_xyzz|st_xyzze)\(&%s\b|\bsl_\w+\(%s\b|uint4\s*\*>\(&?%s\b"
                             % (name, name, name))
            if vec.search("\n".join(lines[i + 1:end])):
                seen += 1
                if int(m.group(2) or 0) < 16:
                    bad.append(f"{os.path.basename(path)}:{i + 1}: {line.strip()}")
    assert seen > 0 and not bad, bad
