"""The error code that a GEMM leaves is that of the wait which ran out first.

A role that gives up makes the others give up behind it: the MMA issuer and the epilogue see its abort flag, and a CTA that sends no
parts lets the waits of its cluster run out.  Making a wait run out needs a GPU that stalls, so the sources are held to the rule instead.
"""
import re

from sharq_b200._build import CSRC
from tests.test_dependent_launch_cpu import _block, _code

CODE = _code(CSRC / "gemm.cu")


def test_a_later_code_does_not_replace_the_first():
    writes = [m.group() for m in re.finditer(r"atomic\w+\s*\([^;]*error_flag[^;]*;|\*\s*p\.error_flag\s*=[^;]*;", CODE)]
    assert writes == ["atomicCAS(error_flag, 0, code);"]
    assert len(set(re.findall(r"report\(p\.error_flag, (\d+)\)", CODE))) == 7


def test_the_code_of_the_receiving_slots_means_their_wait():
    """It is raised where one of their waits has failed, not where the producer had given up before."""
    loop = _block(CODE, CODE.index("for (int s = slot0;"))
    assert "report(p.error_flag, 6)" in loop and CODE.count("report(p.error_flag, 6)") == 1
