"""
How the warps of the tensor-core kernel (csrc/corr_tc.cuh) hand the pairs' entries to each other, as its source
states it: what goes wrong without these lines is a matter of timing, which no run shows for certain.
"""
import os
import re

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), 'slipcam_b200', 'csrc', 'corr_tc.cuh')


def code():
    with open(SOURCE) as f:
        return re.sub(r'//[^\n]*', '', f.read())


def test_entry_is_read_before_it_is_given_back():
    """Between the epilogue's reads of an entry and the store that lets the setup warp overwrite it stands a barrier."""
    text = code()
    stores = [m.start() for m in re.finditer(r's_taken\) = n \+ 1;', text)]
    assert len(stores) == 1
    barrier = text.rindex('bar.sync 1,', 0, stores[0])
    end = text.index('\n    } else {\n', stores[0])   # of the epilogue's role
    assert not re.search(r'\be\.\w', text[barrier:end])
    assert re.search(r'\be\.q\b', text[:barrier])


def test_a_warp_decides_as_one():
    """No vote over the lanes that happen to be active: whole warps vote with the full mask, a lane by itself not at all."""
    text = code()
    assert '__activemask' not in text
    assert text.count('tc_entry_one(e, n, ab)') == 1 and re.search(r'if \(lane == 0\) \{[^{}]*(\{[^{}]*)?tc_entry_one\(e, n, ab\)', text)
