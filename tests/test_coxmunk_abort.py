"""The bulk copies that the Cox-Munk projection may have in flight when it gives up
(csrc/coxmunk_tc.cu): one per stage of the table ring, each of which the issuing warp
must wait for before its CTA leaves and the shared memory is another's.

The issuing warp's copies and waits are replayed here for every chunk at which a wait
can run out: a copy for each chunk up to a ring ahead, a wait for the chunk at hand.
What is then in flight must lie within the copies the exit loop names."""
import os
import re

import pytest

import ocrt_gb300

SRC = os.path.join(os.path.dirname(ocrt_gb300.__file__), "csrc", "coxmunk_tc.cu")


def _waited_at_exit(copied, nbst):
    """Chunks the exit code waits for, by its loop bounds in the source."""
    text = open(SRC).read()
    tail = text[text.index("land before the CTA leaves"):text.index("umma_commit(fin)")]
    m = re.search(r"for \(int k = max\(0, copied - NBST\); k < copied; \+\+k\) \(void\)mbar_wait\(&bfull\[k % NBST\], "
                  r"\(k / NBST\) & 1\);", tail)
    return set(range(max(0, copied - nbst), copied)) if m else {copied - 1}


@pytest.mark.parametrize("nbst", [1, 2])
def test_every_copy_in_flight_is_waited_for(nbst):
    nchunk = 5
    for fail in range(nchunk):                    # the wait for this chunk's table runs out
        issued, landed, copied = set(), set(), 0
        for c in range(fail + 1):
            while copied < nchunk and copied < c + nbst:
                issued.add(copied)
                copied += 1
            if c < fail:
                landed.add(c)
        assert issued - landed <= _waited_at_exit(copied, nbst), (nbst, fail)
