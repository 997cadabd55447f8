"""The loads of the collide kernels, by reading their source.

A collide kernel may be resident while the update before it still writes phi, f and g (it
waits for that update before its first access). The read-only data path is for data that
nothing writes during the kernel's whole life, so the only data read through it are the case
descriptions."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "multic-bubble-cuda_gb300" / "csrc"
SOURCES = ("kernels.cuh", "kernels_pair.cuh")


def _code(name):
    text = (CSRC / name).read_text()
    return re.sub(r"//[^\n]*", "", re.sub(r"/\*.*?\*/", "", text, flags=re.S))


@pytest.mark.parametrize("name", SOURCES)
def test_read_only_loads_are_of_the_case_table_alone(name):
    code = _code(name)
    others = [m.group(0) for m in re.finditer(r"__ldg\w*\(\s*(?!&cd->|&cs\[mid\]\.)[^;\n]*", code)]
    assert others == []
    assert re.findall(r"ld\.global\.\w*\.?nc|\btex\w*\(|__ldlu|__ldcs", code) == []


@pytest.mark.parametrize("name", SOURCES)
def test_no_input_of_an_update_is_declared_read_only(name):
    assert re.findall(r"const\s+[\w:]+\s*\*\s*__restrict__[^;\n]*", _code(name)) == []


@pytest.mark.parametrize("name", SOURCES)
def test_the_first_load_of_the_lattice_follows_the_wait(name):
    code = _code(name)
    assert code.index("grid_wait();") < code.index("issue(t.zb - 2 + p);")
