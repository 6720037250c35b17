"""Waits of the kernels, by reading their source.  Bounded waits: one that runs out must take every thread that later meets
in one barrier or one warp-wide instruction the same way.  (On a GPU this shows only when a wait runs out for some
threads and ends well for others.)  Waits for the kernel before: nothing that it wrote is loaded as read-only data."""
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


#: kernels that may start before the one before them has ended (launch_pdl_opt), and what each may load by __ldg or take as
#: `const __restrict__`: tensors of the caller that no kernel of the same call writes, read behind another kernel of that call
EARLY = {"misc_kernels.cuh": {"gather_tokens_kernel": ["src"], "gather_grad_tokens_kernel": [], "finish_grads_kernel": [],
                              "combine_padded_kernel": []},
         "gemv.cuh": {"gemv_kernel": []}, "umma_gemm.cuh": {"umma_gemm_kernel": []}, "umma_pair.cuh": {"umma_pair_kernel": []},
         "umma_f32.cuh": {"umma_f32_kernel": []}}


def kernel(text, name):
    start = text.index("\n%s(" % name)
    return text[start:text.index("\n}\n", start)]


def test_early_kernels_are_known():
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cuh", ".cu")) and name != "common.cuh":
            calls = len(re.findall(r"\blaunch_pdl_opt\(", source(name)))
            assert calls == len(EARLY.get(name, {})), name


@pytest.mark.parametrize("name,kern", [(f, k) for f in sorted(EARLY) for k in EARLY[f]])
def test_early_kernels_load_what_others_wrote_behind_the_wait(name, kern):
    body = kernel(source(name), kern)
    wait = body.index("pdl_wait()")
    read_only = re.findall(r"const\s+\w+\s*\*\s*__restrict__\s+(\w+)", body)
    assert read_only == EARLY[name][kern], read_only
    for load in re.findall(r"__ldg\(([^;]*);", body):
        assert any(re.search(r"\b%s\b" % allowed, load) for allowed in EARLY[name][kern]), load
    # pointers are taken behind the wait, and what is loaded past this kernel's own stores comes from one of them
    taken = re.findall(r"(\w+) = after_wait\(", body)
    assert all(m.start() > wait for m in re.finditer(r"after_wait\(", body))
    for load in re.findall(r"ld_written\(reinterpret_cast<const uint4\*>\((\w+)", body):
        assert load in taken, load
    for call in re.findall(r"load_vec<([^;]*);", body):
        assert ", true>(" in call, call


def test_epilogues_of_early_kernels_load_no_read_only_data():
    """Pre-activations come from an earlier GEMM of the same pass."""
    for name in ("umma_pair.cuh", "umma_f32.cuh", "umma_gemm.cuh", "gemv.cuh"):
        assert "__ldg(" not in source(name), name
    assert re.findall(r"load_vec<([^>]*)>\(pre\b", source("epilogues.cuh")) == ["T, 2 * NV, true"]
