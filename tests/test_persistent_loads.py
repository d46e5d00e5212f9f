"""The persistent substep kernel reads what it writes with plain loads.

A read-only load (__ldg) is for data that nothing writes while the kernel runs. The bodies that the persistent
kernel shares with the launched kernels therefore choose the load by their template argument.
"""

import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "libclsph_gb300" / "csrc"
CONSTANT = {"test_face", "nearest_hit"}  # a scene's mesh does not change during a launch


def _functions():
    """name -> body of every device function that is not itself a kernel."""
    out = {}
    for name in ("clsph_common.cuh", "clsph_radix.cuh", "clsph_kernels.cuh", "clsph_persistent.cuh"):
        text = re.sub(r"//[^\n]*", "", (CSRC / name).read_text())
        for m in re.finditer(r"^__device__ __forceinline__ [^;{]*?\b(\w+)\([^;]*?\) \{\n(.*?)^\}", text, re.M | re.S):
            out.setdefault(m[1], "")
            out[m[1]] += m[2]
    return out


def test_shared_bodies_have_no_fixed_read_only_loads():
    functions = _functions()
    text = (CSRC / "clsph_persistent.cuh").read_text()
    seen, todo = set(), [text[text.index("k_substeps_persistent(PersistArgs"):]]
    while todo:
        body = todo.pop()
        for name in re.findall(r"\b(\w+)(?:<[^<>()]*>)?\(", body):
            if name in functions and name not in seen:
                seen.add(name)
                todo.append(functions[name])
    assert {"density_cells_team", "density_particle_warp", "forces_particle", "cell_lookup", "ld_step"} <= seen
    bare = {n for n in seen if "__ldg(" in functions[n]} - CONSTANT - {"ld_step"}
    assert not bare
    for body, callee in ((text, "density_cells_team"), (text, "forces_particle")):
        assert re.search(rf"\b{callee}<true>\(", body)
    for caller, callee in (("density_cells_team", "cell_lookup"), ("density_cells_team", "facing_slots"),
                           ("density_cells_team", "density_particle_warp"), ("density_particle_warp", "cell_lookup"),
                           ("forces_particle", "forces_particle_warp"), ("forces_particle_warp", "cell_lookup")):
        assert re.search(rf"\b{callee}<kLive>\(", functions[caller]) and not re.search(rf"\b{callee}\(", functions[caller])
