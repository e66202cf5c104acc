"""Kernels launched before their predecessor on the stream has ended must not
read through __restrict__ pointers: such loads may take the read-only path or
move above the wait, while the predecessor still writes the data."""
import os
import re

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "agent-ray_b200", "csrc", "poisson.cu")


def test_chained_kernels_read_through_plain_pointers():
    text = re.sub(r"//[^\n]*", "", open(SRC).read())
    chained = set(re.findall(r"launch_chained\((k_\w+)", text))
    assert {"k_sor_sweeps", "k_cg_direction", "k_cg_update"} <= chained
    for name in chained:
        m = re.search(r"__global__[^;{]*?\b" + name + r"\(([^)]*)\)\s*\{(.*?)\n\}", text, re.S)
        params, body = m.groups()
        # the wait comes first, the shared arrays' declarations apart
        assert re.match(r"\s*(__shared__[^;]*;\s*)*after_previous\(\);", body), name
        for p in params.split(","):
            if "__restrict__" not in p:
                continue
            var = p.split()[-1]
            assert "const" not in p, f"{name}: {var} is read through __restrict__"
            uses = re.findall(r"\b" + var + r"\b\[[^\]]*\]\s*(.{1,2})", body)
            assert uses and all(u[0] == "=" and u != "==" for u in uses), f"{name}: {var} is not only stored to"
