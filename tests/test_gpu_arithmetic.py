"""The branch-free operations that stand for IEEE ones in the replays and the per-cell
quantities: rcp_normal and sqrt_normal over every significand (both exponent parities
and the ends of their range), log_ratio over its whole range, div_by over 2^28 seeded
pairs of each of its four uses (significands next to one, to two and of all ones among
them). No result may differ from the correctly rounded one."""
import subprocess

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu


def test_branch_free_operations_are_correctly_rounded(tmp_path):
    from illcrawl_b200 import build
    exe = str(tmp_path / "arith_check")
    subprocess.run([build.nvcc()] + build.NVCC_FLAGS
                   + ["-I", build.CSRC, ROOT + "/tests/cpp/arith_check.cu", "-o", exe],
                   check=True, timeout=300)
    out = subprocess.run([exe], check=True, timeout=300, capture_output=True, text=True).stdout
    checks = [line.split() for line in out.splitlines()]
    assert [c[0] for c in checks] == ["rcp_normal", "sqrt_normal"] * 3 + ["log_ratio"] \
        + ["div_by"] * 4, out
    for name, n, bad in checks:
        assert int(n) > 4_000_000 and int(bad) == 0, out
