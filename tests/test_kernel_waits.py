"""Bounded waits of the tensor-core kernels, by reading their source: a wait that runs out must take every thread
that later meets in one barrier or one warp-wide instruction the same way.  (On a GPU this shows only when
a wait runs out for some threads and ends well for others.)"""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "yamoe_b200", "csrc")
#: barriers that whole warps wait on; the others are waited on by one thread, or voted on together
WARP_WIDE = {"umma_gemm.cuh": ["bar_tmem_full"], "umma_pair.cuh": ["bar_tmem_full", "bar_tmem_empty", "bar_full", "bar_empty"],
             "umma_f32.cuh": ["bar_acc_full", "bar_w_full", "bar_a_empty"]}


def source(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


@pytest.mark.parametrize("name", sorted(WARP_WIDE))
def test_waits_of_whole_warps_have_one_outcome(name):
    waits = re.findall(r"\b(mbar_wait\w*)\(smem_u32\(&(\w+)\[", source(name))
    for bar in WARP_WIDE[name]:
        used = [fn for fn, b in waits if b == bar]
        assert used and set(used) == {"mbar_wait_warp"}, (bar, used)


def test_warps_that_store_together_leave_together():
    """group_sync joins four warps for every chunk of a tile: they agree on the outcome of the wait before the first."""
    text = source("umma_pair.cuh")
    wait = text.index("mbar_wait_warp(smem_u32(&bar_tmem_full[acc])")
    agree = text.index("if constexpr (kStore) ok = group_all(1 + turn, ok);", wait)
    assert agree < text.index("if (!ok)", wait) < text.index("emit(c, v)", wait)
    assert "bar.red.and.pred q, %1, 128, p;" in text and "bar.sync %0, 128;" in text


def test_commits_are_awaited_before_a_cta_ends():
    """The leader's last commits arrive in both CTAs' shared memory: each barrier they reach is waited on after the
    last tile, by the role that would use what they free."""
    text = source("umma_f32.cuh")
    for bar in ("bar_b_empty", "bar_a_empty"):
        assert len(re.findall(r"mbar_wait\w*\(smem_u32\(&%s\[" % bar, text)) == 2, bar
