"""What the library's sources may not contain."""
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "thunder-refactor-expectation_gb300" / "csrc"


@pytest.mark.parametrize("path", sorted(CSRC.glob("*.cu*")), ids=lambda p: p.name)
def test_no_cluster_loads(path):
    """No copy or commit that reaches the other CTAs of a cluster: the library
    is loaded by every rank of a run on several GPUs."""
    assert "multicast" not in path.read_text().lower()
