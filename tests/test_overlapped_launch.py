"""Kernels that start before their predecessor has ended and wait for it inside:
what the predecessor writes must be read by loads that see other SMs' stores, so
no such pointer is a const __restrict__ parameter (which allows the read-only
path and lets the compiler move the load above the wait)."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "gnss_gpu_b200" / "csrc"
# inputs that no kernel of such a chain writes
INPUTS = {"k_broadcast_orbits": {"recs", "idx", "times"}, "k_glo_table": {"recs"}}


def _kernels(text):
    """(name, parameters, body) of each __global__ function."""
    for m in re.finditer(r"__global__[^;{]*?\b(k_\w+)\s*\(", text):
        i, depth = m.end(), 1
        while depth:
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        params, j = text[m.end():i - 1], text.index("{", i)
        k, depth = j + 1, 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[k], 0)
            k += 1
        yield m.group(1), params, text[j:k]


def test_waiting_kernels_read_their_predecessors_results_coherently():
    seen = set()
    for path in sorted(CSRC.glob("*.cu*")):
        for name, params, body in _kernels(path.read_text()):
            if not re.search(r"\w*pdl_wait\(\)", body):
                continue
            seen.add(name)
            ro = set(re.findall(r"const\s+\w+\s*\*\s*__restrict__\s+(\w+)", params))
            assert ro <= INPUTS.get(name, set()), f"{path.name}: {name} reads {sorted(ro)} through __restrict__"
    assert {"k_mlp_grad", "k_mlp_reduce", "k_broadcast_orbits", "k_glo_table", "k_estimate"} <= seen
