"""The masks of the kernels' exchanges name their threads: a warp intrinsic's
mask is an expression on the thread's place, never a question of who is active
(after code whose turns differ by thread, a partner may not be there yet)."""
import pathlib
import re

CSRC = pathlib.Path(__file__).resolve().parent.parent / "pentago_b200" / "csrc"


def code(path):
    """A source file without its comments."""
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", path.read_text(), flags=re.S)


def test_no_mask_comes_from_the_active_threads():
    files = sorted(p for p in CSRC.iterdir() if p.suffix in (".cu", ".cuh", ".h", ".cc"))
    assert any("_sync(" in code(p) for p in files)
    found = [f"{p.name}:{k + 1}" for p in files for k, line in enumerate(code(p).split("\n")) if "__activemask" in line]
    assert not found, found
