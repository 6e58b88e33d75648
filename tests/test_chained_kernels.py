"""Kernels that start beside the launch before them (those that call previous_done) read what launches
write with ordinary loads only: the non-coherent path is for data that nothing writes while the kernel
is resident. Checked on their sources, and on those of the device functions they read it through."""

import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "autan_b200" / "csrc"
# a read of primitives, reconstruction or boundary states, and whether it takes the ordinary path
READS = [
    (re.compile(r"\bload5<([^>]*)>\(d\.prim"), "P, true"),
    (re.compile(r"\bload_prim<([^>]*)>\("), "P, true"),
    (re.compile(r"\bload_recon<([^>]*)>\("), "P, true"),
    (re.compile(r"\bcell_recon<([^>]*)>\("), "P, SECOND, true"),
    (re.compile(r"\bload_words<([^>]*)>\(d\.(?:prim|prim_b|recon)\b"), "P, true, true"),
]
NEVER = re.compile(r"__ldg\(\s*d\.(prim|prim_b|recon|u|stage|racc|dt_local|ctl)\b")


def functions():
    """name -> text of every device function and kernel, from its name to the next one's."""
    out = {}
    for name in ("euler_device.cu", "cell_blocks.cuh", "face_blocks.cuh"):
        text = (CSRC / name).read_text()
        for part in re.split(r"^(?=__global__|__device__)", text, flags=re.M)[1:]:
            head = re.sub(r"__launch_bounds__\((?:[^()]|\([^()]*\))*\)", "", part)
            m = re.search(r"\b(\w+)\(", head)
            out[m.group(1)] = head[m.end() :]
    return out


def test_chained_kernels_read_mutable_data_with_ordinary_loads():
    bodies = functions()
    chained = {n for n, b in bodies.items() if "previous_done()" in b}
    assert {"k_gradients_split", "k_faces_block", "k_spectral", "k_begin"} <= chained
    # cell_time_step is k_spectral's alone; cell_recon and load_recon hand their path on
    assert sum("cell_time_step(" in b for b in bodies.values()) == 1
    for name in chained | {"cell_time_step"}:
        assert not NEVER.search(bodies[name]), name
        for pattern, want in READS:
            for m in pattern.finditer(bodies[name]):
                assert m.group(1) == want, (name, m.group(0))
    reads = sum(len(p.findall(bodies[n])) for n in chained | {"cell_time_step"} for p, _ in READS)
    assert reads >= 7
    for name, inner in (("cell_recon", "MUT"), ("load_recon", "MUT"), ("load_prim", "MUT"), ("load5", "MUT")):
        assert inner in bodies[name], name
