"""Rules of the kernel sources that no run can show reliably."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "clean-lm_b200" / "csrc"


@pytest.mark.parametrize("path", sorted(CSRC.glob("*.cu")), ids=lambda p: p.name)
def test_tensor_memory_loads_are_named_by_their_wait(path):
    """The registers of a tensor-memory load go through the wait behind it.  Where the wait does not name them nothing keeps
    arithmetic on them behind it: the fused SwiGLU epilogue once read registers that the load had not filled."""
    pending = set()
    for i, line in enumerate(path.read_text().splitlines(), 1):
        at = f"{path.name}:{i}"
        assert not re.search(r'"tcgen05.(wait::)?ld', line), f"{at}: belongs in ptx.cuh"
        loaded = re.search(r"tmem_ld(?:16|32)\(.*, (\w+)(?:\[\w+\])?\);", line)
        assert loaded or "tmem_ld" not in line, f"{at}: load not understood"
        if loaded:
            pending.add(loaded.group(1))
        waited = re.search(r"tmem_wait_ld\(([^)]*)\);", line)
        if waited and not line.lstrip().startswith("else "):  # (else: of an if whose branch waits for more)
            named = {re.sub(r"\[\d\]", "", r.strip()) for r in waited.group(1).split(",")}
            assert pending <= named, f"{at}: the wait does not name {sorted(pending - named)}"
            pending.clear()
    assert not pending, f"{path.name}: no wait for {sorted(pending)}"
