"""The data-flow smoothing launch's hand-overs between CTAs (flow_schedule.cu), on the host: every value stored
for another CTA is one that some CTA polls for, and the other way round.

A mailbox holds one value, and the order of two stores to it rests on a reader between them. A stored value that
nobody reads has none: its store could land after the next one's, which its reader would then wait for in vain.
"""
import numpy as np
import pytest

import brae_b200.native as b2g
from brae_b200 import cases


def _greedy_colours(c):
    colours = np.full(c.n_cells, -1, np.int32)
    nbr = [[] for _ in range(c.n_cells)]
    for lo, up in zip(c.lower, c.upper):
        nbr[lo].append(up)
        nbr[up].append(lo)
    for cell in range(c.n_cells):
        used = {colours[o] for o in nbr[cell]}
        colours[cell] = next(k for k in range(len(used) + 1) if k not in used)
    return colours


# boxes, a slab and a line of cells; CTAs that cut them anywhere, one cell a CTA at the most
@pytest.mark.parametrize("dims,ranks", [((9, 7, 5), (2, 7, 33)), ((23, 11, 1), (5, 148)), ((40, 1, 1), (3, 40)),
                                        ((16, 15, 14), (4, 148))])
@pytest.mark.parametrize("symmetric", [False, True])
@pytest.mark.parametrize("coloured", [False, True])
def test_every_hand_over_has_a_reader(dims, ranks, symmetric, coloured):
    c = cases.box_case(*dims)
    colours = _greedy_colours(c) if coloured else None
    for r in ranks:
        for sweeps in (1, 2, 4):
            for weight in (1, 4):
                n = b2g.flow_handovers(c.lower, c.upper, c.n_cells, sweeps, r, weight, symmetric, colours)
                assert n["unread"] == 0 and n["missing"] == 0, (r, sweeps, weight, n)
                # with several sweeps every rank reads its neighbours' values
                assert sweeps == 1 or (n["stored"] >= r - 1 and n["taken"] >= n["stored"])
