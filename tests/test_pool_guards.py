"""The pool's rule: when a buffer from it goes out of scope, by an exception
too, no work that uses it is pending. A function that declares such buffers
declares the guard that waits (Drain, PoolStream, Wait) right after them, ahead
of any work; a failed check between an upload and the call's own wait would
hand the buffer to the next thread with the copy under way."""
import os
import re

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "pyqcm_gb300", "csrc")
BUFFER = re.compile(r"^\s+(PoolBuf|PinnedBuf)<[^;]*;")
GUARD = re.compile(r"^\s+(Drain|PoolStream|Wait) \w+")
WORK = re.compile(r"<<<|MemcpyAsync|MemsetAsync|\.upload\(")


@pytest.mark.parametrize("name", ["qcmg_api.cu", "qcmg_band.cu", "qcmg_chip.cu", "qcmg_chip_band.cu", "qcmg_lattice.cu"])
def test_buffers_are_guarded_before_work_is_queued(name):
    with open(os.path.join(CSRC, name)) as f:
        lines = f.readlines()
    found = [i for i, line in enumerate(lines) if BUFFER.match(line)]
    assert found
    for i in found:
        for line in lines[i + 1:]:
            if GUARD.match(line):
                break
            # (work on a lambda's or a launch's line after the guard is not reached here)
            assert not WORK.search(line), (name, i + 1, line)
        else:
            assert False, (name, i + 1)
