"""The word exchange of the cooperative tridiagonalisation, as a model.

Rows are dealt to CTAs in turn (row r to CTA r % G).  At step j a CTA publishes
the words of its rows >= j with the step's number, in one of two buffers by the
step's parity, leaves if it has no row > j, and otherwise waits until the words of
all rows >= j carry that number.  A word that is overwritten before a reader saw
it leaves that reader waiting until its limit: no order of the CTAs may do that.
"""
import math

import pytest


def starved_readers(n, g, first):
    """(reader, step, row) for words gone before their reader sees them: the
    reader stops between publishing a step and reading it, the other CTAs go on
    as far as they can.  Rows >= j + first are published and waited for."""
    last = [max(range(b, n, g)) for b in range(g)]
    steps = range(n - 2)
    out = []
    for x in range(g):
        for s in steps:
            if last[x] <= s:
                break  # no row > s: the reader has left
            words = {}  # (parity, row): step number
            step, read = [0] * g, [-1] * g  # steps published, last step read
            moved = True
            while moved:
                moved = False
                for b in range(g):
                    j = step[b]
                    if j in steps and read[b] == j - 1 and last[b] >= j:
                        words.update({(j & 1, r): j for r in range(b, n, g) if r >= j + first})
                        step[b] += 1
                        moved = True
                    elif read[b] < j - 1 and last[b] > j - 1 and (b, j - 1) != (x, s) and all(
                            words.get((j - 1 & 1, r)) == j - 1 for r in range(j - 1 + first, n)):
                        read[b] += 1
                        moved = True
            out += [(x, s, r) for r in range(s + first, n) if words.get((s & 1, r), -1) > s]
    return out


@pytest.mark.parametrize("n,g", [(6, 2), (9, 3), (10, 3), (13, 4), (17, 5), (24, 7)])
def test_no_reader_is_overtaken(n, g):
    assert starved_readers(n, g, 0) == []
    # without the word of row j, a CTA that has no row below it is not waited for
    assert bool(starved_readers(n, g, 1)) == (g >= 4)


def test_every_cta_starts_with_rows_to_spare():
    """No CTA leaves at step 0, where row 0 is stored after the gather: the
    launch's CTA count for every n that it takes."""
    sms, chunk = 148, 16
    for n in range(3, 2049):
        g = min(max(math.ceil(8.0 * n * n / (96 * 1024)), -(-n // chunk)), n, sms)
        g = -(-n // -(-n // g))
        assert n // g >= 3, (n, g)
