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


def test_the_weight_stream_starts_its_limits_behind_the_kernel_before():
    """Every role of the weight stream passes the wait for the kernel before it ahead of its first bounded wait: what that kernel takes is not a wait that ran out."""
    code = (KERNELS / "decode.cu").read_text()
    body = code[code.index("gemm_stream_kernel(const __grid_constant__"):]
    body = body[: body.index("\n}\n")]
    roles = re.split(r"\n  (?:if \(warp == 0\) \{\n|\} else if \(warp == 1\) \{\n|\} else \{\n)", body)[1:]
    assert len(roles) == 3
    for role in roles:
        assert 0 <= role.find("pdl_wait()") < role.index("ws_wait(")


@pytest.mark.parametrize("name", ["ft_flash_fwd", "ft_flash_bwd_ws", "ft_embedding_bwd_sorted"])
def test_launchers_that_were_shipped_stay_in_the_c_interface(name):
    from ferrotorch_b200 import _lib
    header = (KERNELS.parent / "include" / "ferrotorch" / "kernels.h").read_text()
    assert f"int {name}(" in header and hasattr(_lib.kernels(), name)


def test_benchmarks_name_launchers_that_the_package_calls():
    """A row of a benchmark's table is keyed by the launcher's name: one that nothing calls loses its figures without a word."""
    root = KERNELS.parents[2]
    called = set(re.findall(r'"(ft_[a-z0-9_]+)"', "".join(p.read_text() for p in (root / "ferrotorch_b200").rglob("*.py"))))
    named = {n for p in (root / "benchmarks").glob("*.py") for n in re.findall(r'"(ft_[a-z0-9_]+)"', p.read_text())}
    assert named and named <= called, sorted(named - called)
