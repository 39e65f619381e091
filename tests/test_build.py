"""What the built library costs a process that loads it."""
from __future__ import annotations

import os


def test_the_library_stays_small_enough_to_load():
    """A kernel's first launch loads its unit of the library, so a process's first product pays for the library's bytes:
    27 ms at 84 MB (with the line tables of the generated codelets), 7 ms at 41 MB."""
    from rooftop_mom_b200 import build

    assert os.path.getsize(build.build()) < 56e6
