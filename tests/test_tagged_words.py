"""Border cells that carry their own tag (the epoch or the number of the sweep) instead of a flag: a reader that sees the
tag takes the value with it, with no fence between them. PTX keeps an access whole only up to its element type, and a
vector access is its elements in any order, so tag and value have to lie in one element. Checked on the CPU: every order
in which a writer's and a reader's elements can meet, for the element widths that the two kernels ask for.
"""
from __future__ import annotations

import itertools
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "fluid-dynamics1_gb300", "csrc")
ACCESS = re.compile(r'"(?:ld|st)\.(?:relaxed|volatile)(?:\.gpu|\.cluster)?(?:\.global|\.shared)?\.v(\d)\.[ub](\d+)')


def stale_value_seen(width: int) -> bool:
    """Whether a reader of a 64-bit cell {value, tag} accessed in elements of `width` bits can see the new tag with
    any part of the old value."""
    parts = range(64 // width)
    for writes, reads in itertools.product(itertools.permutations(parts), itertools.permutations(parts)):
        for cut in itertools.combinations_with_replacement(range(len(parts) + 1), len(parts)):
            # the r-th read happens after cut[r] of the writes
            new = {part: part in writes[:done] for part, done in zip(reads, cut)}
            tag = [p for p in parts if (p + 1) * width > 32]
            value = [p for p in parts if p * width < 32]
            if all(new[p] for p in tag) and not all(new[p] for p in value):
                return True
    return False


def test_only_whole_words_keep_value_and_tag_together():
    assert not stale_value_seen(64)
    assert stale_value_seen(32)


@pytest.mark.parametrize("source", ["cnv_mixed.cu", "cnv_poisson_cells.cu"])
def test_the_kernels_exchange_whole_words(source):
    text = open(os.path.join(CSRC, source)).read()
    accesses = ACCESS.findall(text)
    assert len(accesses) >= 2 and all(not stale_value_seen(int(width)) for _, width in accesses), accesses
