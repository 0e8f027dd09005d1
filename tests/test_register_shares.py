"""The pair kernels' register shares (csrc/launch.h): what the host lets run.  An increase of a warpgroup's registers past what the launch brought waits for good,
so a build with fewer registers per thread than the shares add up to is refused ahead of its first launch; that is shown here, on the host's own condition."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "qserve_b200", "csrc")


def _holds(condition, tmp_path):
    src = tmp_path / "shares.cpp"
    src.write_text('#include "launch.h"\nusing namespace qs;\nstatic_assert(%s);\n' % condition)
    return subprocess.run(["g++", "-std=c++17", "-fsyntax-only", "-I", CSRC, str(src)], capture_output=True, text=True)


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
@pytest.mark.parametrize("per_thread,fits", [(96, True), (95, False), (88, False), (80, False), (0, False)])
def test_launches_that_bring_too_few(tmp_path, per_thread, fits):
    r = _holds("%spair_registers_suffice(%d)" % ("" if fits else "!", per_thread), tmp_path)
    assert r.returncode == 0, r.stderr


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_the_shares_are_the_launch_s(tmp_path):
    # a multiprocessor's 65536 registers hold the launch, shares come in eights, and 640 threads cannot be launched with more than 96 registers each
    r = _holds("kPairRoundsThreads == 5 * 128 && kPairRoundsThreads * 96 <= 65536 && kPairRoundsThreads * 104 > 65536 && kPairLoadRegs % 8 == 0 && "
               "kPairUnpackRegs % 8 == 0 && kPairEpilogueRegs % 8 == 0", tmp_path)
    assert r.returncode == 0, r.stderr
