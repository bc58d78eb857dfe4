"""Every kernel that is launched with programmatic stream serialization may start while its predecessor on the stream still
runs, so it has to wait for it (grid_dep_wait) before its first store.  Read from the sources: a kernel without the wait shows
only now and then on a GPU."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "spbitnet_b200" / "csrc"
# launched without the attribute: a cooperative launch and two self-tests
WITHOUT_ATTRIBUTE = {"decode_persistent_kernel", "pd_barrier_selftest_kernel", "ws_wait_selftest_kernel"}


def kernels():
    """(name, body) of every __global__ function that is defined in the library's sources."""
    for path in sorted(CSRC.glob("*.cu")) + sorted(CSRC.glob("*.cuh")):
        text = re.sub(r"//[^\n]*", "", path.read_text())
        for m in re.finditer(r"__global__", text):
            start = text.index("{", m.end())
            head = text[m.end():start]
            if ";" in head:
                continue  # a declaration
            depth, end = 0, start
            while True:
                depth += {"{": 1, "}": -1}.get(text[end], 0)
                end += 1
                if depth == 0:
                    break
            name = next(w for w in re.findall(r"(\w+)\s*\(", head) if w != "__launch_bounds__")
            yield name, text[start:end]


def test_kernels_wait_for_their_predecessor():
    found = dict(kernels())
    assert len(found) > 40 and WITHOUT_ATTRIBUTE <= set(found)
    missing = [n for n, body in found.items() if "grid_dep_wait()" not in body and n not in WITHOUT_ATTRIBUTE]
    assert not missing, missing


def test_waits_behind_a_predecessor_are_bounded_from_its_end():
    """Weights are on their way before a grid's predecessors are done; what follows from the activations comes after them, and their
    time must not count towards the bound of such a wait."""
    for name, barriers in {"gemm_tcsp_ws.cu": ["w_free + 8 * w.s", "bbar", "a_free + 8 * sA"], "half_gemm_tc.cu": ["full + 8 * c.s"]}.items():
        text = (CSRC / name).read_text()
        for b in barriers:
            assert f"ws_wait_dep({b}," in text and f"ws_wait({b}," not in text, (name, b)
