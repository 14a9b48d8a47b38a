"""The library's calls take their device and pinned memory from the caller
("hot calls never allocate"): its sources call no allocation, release or
registration function of CUDA, which would also synchronise the device."""
import re
from pathlib import Path

import renormalizer_b200

CALLS = re.compile(r"\b(cuda(Malloc|Free|HostAlloc|HostRegister|HostUnregister|MemPool)|cuMem(Alloc|Free))\w*\s*\(")


def test_sources_allocate_nothing():
    src = Path(renormalizer_b200.__file__).parent / "csrc"
    files = sorted(src.glob("*.cu")) + sorted(src.glob("*.cuh"))
    assert len(files) > 10
    found = [(f.name, n + 1, line.strip()) for f in files for n, line in enumerate(f.read_text().splitlines())
             if CALLS.search(line)]
    assert not found
