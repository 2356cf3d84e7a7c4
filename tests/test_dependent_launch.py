"""A kernel that calls dep_wait() is resident while the kernel before it still
writes.  __restrict__ on a parameter tells the compiler that nobody else writes
the array while the kernel runs, so its loads may be moved above the wait or take
the read-only path: only arrays that no kernel of the chain writes may have it."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "gundam_gb300" / "csrc"
# set before the chain begins: observed data, standardisation, prior, proposal factor
CONSTANT = {"data", "mean", "scale", "m", "icov", "Lt"}


def _kernels(text):
    text = re.sub(r"//[^\n]*", "", text)
    for g in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\([^)]*\)\s*)?(\w+)\s*\(", text):
        depth, i = 1, g.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        params = text[g.end():i - 1]
        j = text.index("{", i)
        depth, k = 1, j + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[k], 0)
            k += 1
        yield g.group(1), params, text[j:k]


def test_restrict_only_on_arrays_constant_over_the_chain():
    seen = 0
    for path in sorted(CSRC.glob("*.cu")):
        for name, params, body in _kernels(path.read_text()):
            if "dep_wait()" not in body and "gemm_tile" not in body:
                continue
            seen += 1
            bad = set(re.findall(r"__restrict__\s+(\w+)", params)) - CONSTANT
            assert not bad, (path.name, name, bad)
    assert seen >= 16
