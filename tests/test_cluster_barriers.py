"""Barriers in inline PTX whose form asks for the whole warp together (.aligned, and bar.sync,
which is): each directly behind a __syncwarp or a vote over the full mask. Read from the
sources: a warp that arrives in parts cannot be shown on the CPU, and must not be on the GPU."""
import os
import re

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cfd-craft_gb300", "csrc")


def statements(text):
    text = re.sub(r"//[^\n]*", "", text)
    return [" ".join(s.split()) for s in re.split(r"(?<=[;{}])\s*\n", text)]


def test_aligned_barriers_follow_a_convergence_point():
    found = 0
    for name in sorted(os.listdir(SRC)):
        if not name.endswith((".cu", ".cuh")):
            continue
        st = [s for s in statements(open(os.path.join(SRC, name)).read()) if s]
        for k, s in enumerate(st):
            if not re.search(r'asm volatile\(\s*"(bar\.sync|bar\.arrive|barrier\.[^"]*\.aligned)', s):
                continue
            found += 1
            before = st[k - 1]
            if before == "}":  # the end of a loop: its condition is what ran last
                depth, q = 1, k - 2
                while depth:
                    depth += (st[q].count("}") - st[q].count("{"))
                    q -= 1
                before = st[q + 1]
            assert "__syncwarp();" in before or "while (__any_sync(0xffffffffu" in before, (name, before, s)
    assert found >= 3
