"""How the linked restart cycle (csrc/linked.cuh) reads and writes its cells.

A cell is one 64-bit word per 32 bits of value, each with the number of the
iteration beside it, and a reader has no fence or flag: it relies on getting a
value together with its own number.  PTX promises that only within one element of
an access (a vector access is one access per element, in no given order), so every
element stored and loaded has to be a whole 64-bit word.
"""
import re
from pathlib import Path

import pytest

SOURCE = Path(__file__).resolve().parents[1] / "mipx_b200" / "csrc" / "linked.cuh"


@pytest.mark.parametrize("access", ["ld", "st"])
def test_cells_are_accessed_in_whole_words(access):
    forms = re.findall(rf"\b{access}\.relaxed\.gpu\.global\.([\w.]+)", SOURCE.read_text())
    assert len(forms) == 2, "one access for FP64 cells and one for FP32 cells"
    assert sorted(forms) == ["b64", "v2.b64"]
