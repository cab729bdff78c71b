"""The two slots of partial sums that consecutive reductions of a team alternate
between share no word, whatever the reductions on either side publish: a block
that is ahead writes one slot while another still reads the other.  Checked on
the source: the sequence of calls that runs today meets the overlap of unequal
strides on no word that is still read."""
import itertools
import os
import re

from tests.util import ROOT


def _reductions():
    """(slot stride, words published) of every reduction, in units of the grid"""
    src = open(os.path.join(ROOT, "schrodingersem_gb300", "csrc", "sem_cg.cuh")).read()
    consts = {k: int(v) for k, v in re.findall(r"constexpr int (\w+) = (\d+);", src)}
    widths = {int(k) for k in re.findall(r"team_sum<TEAM, (\d)>\(", src)}
    strides = re.findall(r"tm\.partials \+ \(size_t\)slot \* (\w+) \* G", src)
    assert len(strides) == 2 and widths  # team_sum, team_sum64
    for name, ks in zip(strides, (widths, {2})):
        for k in ks:
            yield (k if name == "K" else int(name) if name.isdigit() else consts[name]), k


def test_slots_share_no_word():
    red = list(_reductions())
    for (sa, ka), (sb, kb) in itertools.product(red, red):
        a, b = set(range(0, ka)), set(range(sb, sb + kb))  # slot 0 of one, slot 1 of the other
        assert not a & b, (sa, ka, sb, kb)
