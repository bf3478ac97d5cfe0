"""Rules of the CUDA sources, checked on their text: those for kernels which
may be resident while the kernel before them still writes (sgm_launch.h:
launch_after), and the list of the checked build's sites."""
import glob
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pyrsgm_gb300", "csrc")


def _code():
    """The sources without comments, by file name."""
    out = {}
    for f in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        with open(f) as h:
            out[os.path.basename(f)] = re.sub(r"//[^\n]*|/\*.*?\*/", "", h.read(), flags=re.S)
    return out


def _body(text, start):
    """The braces block from the first '{' at or after start."""
    i = text.index("{", start)
    depth, j = 0, i
    while True:
        depth += {"{": 1, "}": -1}.get(text[j], 0)
        j += 1
        if depth == 0:
            return text[i:j]


def test_no_read_only_loads():
    """__ldg promises that nothing writes the memory while the kernel lives;
    the kernel before may."""
    bad = [(f, n) for f, t in _code().items() for n in ("__ldg", "ld.global.nc", "__restrict__") if n in t]
    assert not bad


def test_kernels_let_in_early_wait_for_the_one_before():
    """Every kernel launched with launch_after has the wait, before any return
    and any access through its descriptor's buffers."""
    code = _code()
    launched = {m for t in code.values() for m in re.findall(r"launch_after\((?:pg::)?(k_\w+)", t)}
    kernels = {}
    for t in code.values():
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\([^;{]*?\)\s+)?(k_\w+)\(", t):
            kernels[m.group(1)] = _body(t, m.end())
    assert len(launched) >= 15 and launched <= set(kernels)
    for k in launched:
        before, wait, _ = kernels[k].partition("after_previous();")
        assert wait, k
        # (an early return waits in its own block)
        assert "return" not in before and not re.search(r"J\.\w+\s*\[|cp16|tile_cp16|atomic", before), k


def test_check_sites_are_the_listed_ones():
    """The sites that check.h lists are those of the kernels, each its number,
    and every kernel that writes or reads a volume has one."""
    with open(os.path.join(CSRC, "check.h")) as h:
        text = re.sub(r"\n//", " ", h.read())
    listed = text[text.index("Sites: "):text.index("#pragma once")]
    listed = re.sub(r"\([^)]*\)", "", listed)
    numbers = {int(n) for n in re.findall(r"(?<![\w-])(\d+)(?=[ ,])", listed)}
    used = {int(n) for f, t in _code().items() for n in re.findall(r"PG_IN\((?:[^;{]*?), (\d+)\)", t)}
    assert used == numbers == set(range(1, max(numbers) + 1))
    for k in ("k_seg", "k_rowadd", "k_grow", "k_gtb", "k_gtbw", "k_post", "k_features", "k_cost_census",
              "k_cost_bt_tiled", "k_cost_bt_strip", "k_path_signed", "k_wta_group"):
        assert re.search(r"\b" + k + r"\b", listed), k
