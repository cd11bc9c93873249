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
  for (int inv = 0; inv < 4; ++inv)
    for (int lost = 0; lost < 2; ++lost)
      for (int fin = 0; fin < 2; ++fin) std::printf("%d %d %d %d\\n", inv, lost, fin, item_status(inv, lost, fin));
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_an_expired_wait_is_not_reported_as_a_singular_block(tmp_path):
    from dpnegf_b200 import _lib
    (tmp_path / "s.cpp").write_text(SRC)
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "dpnegf_b200", "csrc"), "s.cpp", "-o", "s"],
                   cwd=tmp_path, check=True)
    got = {}
    for line in subprocess.run([str(tmp_path / "s")], check=True, capture_output=True, text=True).stdout.splitlines():
        inv, lost, fin, st = map(int, line.split())
        got[inv, lost, fin] = st
    singular, expired = 1, 2
    for lost in (0, 1):
        for fin in (0, 1):
            assert got[expired, lost, fin] == got[expired | singular, lost, fin] == _lib.NEGF_ERR_TIMEOUT
            assert got[singular, lost, fin] == _lib.NEGF_ERR_SINGULAR
            assert lost == 0 or got[0, 1, fin] == _lib.NEGF_ERR_TIMEOUT
    assert got[0, 0, 1] == _lib.NEGF_OK and got[0, 0, 0] == _lib.NEGF_ERR_NONFINITE


def test_the_exception_of_an_expired_wait():
    import torch
    from dpnegf_b200 import _lib, rgf_plan
    with pytest.raises(_lib.NegfError, match="wait"):
        rgf_plan.check_status(torch.tensor([0, _lib.NEGF_ERR_TIMEOUT], dtype=torch.int32))
    with pytest.raises(torch.linalg.LinAlgError, match="singular"):
        rgf_plan.check_status(torch.tensor([0, _lib.NEGF_ERR_SINGULAR], dtype=torch.int32))
