"""Rules of the kernel sources whose breach one GPU does not show in a test."""
import re
from pathlib import Path

import pytest

KERNELS = Path(__file__).resolve().parent.parent / "ferrotorch_b200" / "csrc" / "kernels"


@pytest.mark.parametrize("path", sorted(p for p in KERNELS.iterdir() if p.suffix in (".cu", ".cuh")), ids=lambda p: p.name)
def test_shared_memory_limits_are_set_on_every_device(path):
    """The limit of a kernel's dynamic shared memory belongs to a device: a launcher that remembers having set it keeps a flag per device."""
    lines = path.read_text().splitlines()
    for i, line in enumerate(lines):
        if "cudaFuncAttributeMaxDynamicSharedMemorySize" in line or "ft_allow_shared(" in line:
            assert not any(re.search(r"static\s+(bool|int|cudaError_t)\s+\w+\s*=", x) for x in lines[max(0, i - 6): i]), f"{path.name}:{i + 1}"
