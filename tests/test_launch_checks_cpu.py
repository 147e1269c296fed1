"""A kernel launch that the runtime refuses (too much shared memory, say) shows in
cudaGetLastError only until the next call that succeeds, so a status read after several
launches can miss it and a build lose a quartet class: in every source, the statement after
a launch reads its status.
"""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), 'polymer_b200', 'csrc')
SOURCES = sorted(glob.glob(os.path.join(CSRC, '*.cu')) + glob.glob(os.path.join(CSRC, '*.cuh')))
# a branch of an if chain may leave it to the statement after the chain
CHECK = re.compile(r'\s*(//[^\n]*\n\s*)*(note_launch\(\);|PFE_CUDA\((cudaGetLastError|launch_status)\(\)\);|else\b)')


def _ends(text):
    """Where the statement of each launch ends."""
    for m in re.finditer('<<<', text):
        k = text.index('(', text.index('>>>', m.start()))
        depth = 1
        while depth:
            k += 1
            depth += (text[k] == '(') - (text[k] == ')')
        yield m.start(), text.index(';', k) + 1


def test_there_are_launches_to_check():
    assert sum(open(f).read().count('<<<') for f in SOURCES) > 80


@pytest.mark.parametrize('path', SOURCES, ids=os.path.basename)
def test_every_launch_is_followed_by_a_look_at_its_status(path):
    text = open(path).read()
    missed = [text.count('\n', 0, at) + 1 for at, end in _ends(text) if not CHECK.match(text[end:])]
    assert missed == []
