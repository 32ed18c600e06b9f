"""The margins of the parallel hull's check (csrc/k_felz.cu), worked out from its
constants in units of e = 2^-24, half a float's last place: a vertex that
counts as clear stays clear after everything that the check lets pass and all
rounding, its own and the reference's."""
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_clear_vertices_stay_clear():
    src = open(os.path.join(ROOT, "distance-occlusion_b200", "csrc", "k_felz.cu")).read()
    e = 2.0 ** -24
    const = lambda name: float.fromhex(re.search(r"constexpr float %s = (0x1p-\d+)f;" % name, src).group(1)) / e
    turns = int(re.search(r"constexpr int kFelzTurns = (\d+);", src).group(1))
    # a boundary: a rounded difference and a division
    check = src[src.index("const float s1 ="):src.index("const float gap =")]
    division = {"__fdiv_rn": 1, "__fdividef": 4}[re.search(r"= (\w+)\(hq", check).group(1)]   # 2 ulp = 4 e
    boundary = 1 + division
    gap = 2 * boundary + 2          # of two boundaries, and its own rounding (at most twice the size)
    clear, off, sure = const("kFelzClear"), const("kFelzOff"), const("kFelzSure")
    assert sure >= gap              # a vertex that is no turn has a gap above zero in truth
    back = (turns + 1) * (off + gap)   # what boundaries can fall back by, to one side
    reference = 2 * 2               # its two boundaries
    assert clear - gap - 2 * back > reference + 1
