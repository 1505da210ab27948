"""The C++ frontend's fused ops against its own libtorch formulation (examples/cpp/check_fused.cc)."""
import subprocess
from pathlib import Path

import pytest

CHECKER = Path(__file__).resolve().parents[1] / "infinitrain_b200" / "bin" / "itb_check_fused"


@pytest.mark.gpu
@pytest.mark.skipif(not CHECKER.exists(), reason="the C++ frontend has not been built")
def test_fused_ops_of_the_cpp_frontend():
    r = subprocess.run([str(CHECKER)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-3000:] + r.stderr[-1000:]
    assert "swiglu, gradient off boundary" in r.stdout
