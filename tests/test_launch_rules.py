"""Launch rules follow the device: no count of SMs is written into the sources."""
import pathlib
import re

CSRC = pathlib.Path(__file__).resolve().parent.parent / "cudagfx_gb300" / "csrc"


def test_no_sm_counts_as_literals():
    # 152 SMs, two blocks for each, four schedulers each
    for f in sorted(CSRC.glob("*.cu*")):
        code = re.sub(r"//[^\n]*|/\*.*?\*/", "", f.read_text(), flags=re.S)
        assert not re.search(r"(?<![\w.])(152|304|608)(?![\w.])", code), f.name
