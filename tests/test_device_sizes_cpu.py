"""Launch rules count their blocks by the device's own number of multiprocessors: no code line of the kernels holds
the 152 of the device they were tuned on, or a multiple of it."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "em_lab_gb300" / "csrc"


def test_no_multiprocessor_count_in_the_code():
    found = []
    for f in sorted(CSRC.iterdir()):
        text = re.sub(r"/\*.*?\*/", "", f.read_text(), flags=re.S)
        for n, line in enumerate(text.splitlines(), 1):
            code = line.split("//")[0]
            if re.search(r"(?<![\w.])(152|304|456|608)(?![\w.])", code):
                found.append(f"{f.name}:{n}: {line.strip()}")
    assert not found, found
