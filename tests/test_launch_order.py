"""Kernels launched by launch_after may be set up before the kernel in front of
them has ended, so each has to wait as its first statement.  A source file uses
launch_after for all of its launches or for none, and no kernel is launched from
another file: then every kernel of the former waits."""
import pathlib
import re

CSRC = pathlib.Path(__file__).resolve().parents[1] / "fluidsurfacereconstructiongpu_gb300" / "csrc"


def test_every_chained_kernel_waits_first():
    chained = {}
    for path in CSRC.glob("*.cu"):
        text = path.read_text()
        if "launch_after(" not in text:
            continue
        assert "<<<" not in text, path.name
        bodies = re.findall(r"__global__[^;{]*?\b(k_\w+)\s*\([^{;]*?\)\s*\n\{\n\s*(\S[^\n]*)", text)
        assert len(bodies) == len(re.findall(r"^(?:template <[^\n]*>\n)?__global__", text, flags=re.M)), path.name
        chained.update((name, first.strip()) for name, first in bodies)
    assert len(chained) >= 35
    assert {name for name, first in chained.items() if first != "after_launch();"} == set()
