"""Promises that the device code must not make, read off its source (no GPU, no compiler)."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "kernelmatrices.jl_gb300" / "csrc"


def kernels(text):
    """(name, parameters, body) of every __global__ function of a source."""
    for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\([^;{]*?\)\s+)?(\w+)\(", text):
        depth, i = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        depth, j = 1, text.index("{", i) + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[j], 0)
            j += 1
        yield m.group(1), text[m.end():i - 1], text[i:j]


def test_kernels_that_start_early_do_not_restrict_their_vectors():
    """__restrict__ promises that nobody else writes the vectors while the kernel runs, and allows loads by the
    read-only path; the kernel in front of one that starts early still does."""
    early = [(name, args) for f in CSRC.glob("*.cu") for name, args, body in kernels(f.read_text())
             if "wait_for_previous()" in body or "griddepcontrol.wait" in body]
    assert {name for name, _ in early} == {"k_up", "k_down"}
    assert [name for name, args in early if "__restrict__" in args] == []


def test_cluster_permission_is_set_per_device():
    """The permission for clusters above 8 belongs to a kernel on a device: one place asks for it, by device."""
    users = {f.name for f in CSRC.glob("*.cu*") if "NonPortableClusterSizeAllowed" in f.read_text()}
    assert users == {"km_probe.cu"}
    body = (CSRC / "km_probe.cu").read_text().split("int cluster_limit(", 1)[1]
    assert "known[{func, dev}]" in body


def test_waits_count_polls():
    """A bounded wait counts polls, as km_set_wait_limit documents: the clock also runs while another process has
    the GPU."""
    assert [f.name for f in CSRC.glob("*.cu*") if re.search(r"\bclock(64)?\(|globaltimer", f.read_text())] == []
