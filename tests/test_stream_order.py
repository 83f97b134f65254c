"""The runtime's streams are non-blocking, so nothing that it puts on the legacy default stream
is ordered before its kernels (cudaMemset of device memory returns before it is done): its
sources must name a stream for every copy and fill."""
from __future__ import annotations

import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "chemps2_gb300" / "csrc"


def test_no_copy_or_fill_on_the_legacy_stream():
    found = []
    for path in sorted((CSRC / "dmrg").rglob("*")) + sorted((CSRC / "device").rglob("*")):
        if path.suffix in (".cpp", ".hpp", ".cu", ".cuh"):
            for i, line in enumerate(path.read_text().splitlines(), 1):
                if re.search(r"\bcudaMem(set|cpy)(2D|3D|ToSymbol|FromSymbol)?\(", line):
                    found.append(f"{path.name}:{i}: {line.strip()}")
    assert not found, "\n".join(found)
