"""An item's status from the flags its kernel collected, compiled for the host."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = """
#include <cstdio>
#include "item_status.cuh"
int main() {
  for (int i = 0; i < 16; ++i)
    std::printf("%d %d %d %d %d\\n", i & 1, i >> 1 & 1, i >> 2 & 1, i >> 3 & 1, item_status(i & 1, i >> 1 & 1, i >> 2 & 1, i >> 3 & 1));
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_an_expired_wait_is_not_reported_as_a_singular_block(tmp_path):
    from dpnegf_b200 import _lib
    (tmp_path / "s.cpp").write_text(SRC)
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "dpnegf_b200", "csrc"), "s.cpp", "-o", "s"],
                   cwd=tmp_path, check=True)
    out = subprocess.run([str(tmp_path / "s")], check=True, capture_output=True, text=True).stdout
    seen = 0
    for line in out.splitlines():
        bad, inv_lost, tc_lost, finite, status = map(int, line.split())
        if bad:
            want = _lib.NEGF_ERR_TIMEOUT if inv_lost else _lib.NEGF_ERR_SINGULAR
        elif tc_lost:
            want = _lib.NEGF_ERR_TIMEOUT
        else:
            want = _lib.NEGF_OK if finite else _lib.NEGF_ERR_NONFINITE
        assert status == want, line
        seen += 1
    assert seen == 16


def test_the_exception_of_an_expired_wait():
    import torch
    from dpnegf_b200 import _lib, rgf_plan
    with pytest.raises(_lib.NegfError, match="wait"):
        rgf_plan.check_status(torch.tensor([0, _lib.NEGF_ERR_TIMEOUT], dtype=torch.int32))
    with pytest.raises(torch.linalg.LinAlgError, match="singular"):
        rgf_plan.check_status(torch.tensor([0, _lib.NEGF_ERR_SINGULAR], dtype=torch.int32))
