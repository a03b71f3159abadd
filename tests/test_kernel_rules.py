"""Rules of the device code that no run can show safely, checked on its source: what a broken one
would cost is a hang or a read of freed memory."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gpu-load-balance_gb300", "csrc")


def source(name):
    text = open(os.path.join(CSRC, name)).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    return re.sub(r"//[^\n]*", "", text)


def body(text, start):
    """The brace block that opens after the match of `start`."""
    i = text.index("{", re.search(start, text).end())
    depth = 0
    for j in range(i, len(text)):
        depth += {"{": 1, "}": -1}.get(text[j], 0)
        if depth == 0:
            return text[i:j + 1]
    raise AssertionError("unbalanced braces")


def test_a_cta_leaves_a_failed_level_as_a_whole():
    """The error flag can be set while a kernel runs; a CTA whose threads each decided for
    themselves could lose some of a named barrier's warps. So the one test of the flag ends in a
    vote of the CTA, and is its only way out."""
    text = source("orb_kernels.cu")
    fail = body(text, r"bool level_failed\(const Level &v\)")
    assert re.findall(r"return\b[^;]*;", fail) == ["return __syncthreads_or(late || ctr->error) != 0;"]
    # and nothing else decides on the flag
    assert not re.search(r"if \([^)]*error\b", text)


def test_an_acquire_is_followed_by_a_barrier():
    """One thread acquires the other CTAs' writes; the threads that read them are ordered behind
    it by a barrier (a shuffle orders no memory)."""
    text = source("orb_kernels.cu")
    calls = [m.end() for m in re.finditer(r"\bacquire\(\);", text)]
    assert len(calls) == 4
    for at in calls:
        assert re.search(r"__sync(threads|warp)\b|__shfl_sync", text[at:]).group() != "__shfl_sync"


def test_a_lost_copy_ends_its_group():
    """A wait for a copy that ran out leaves its barrier in a phase that must not be armed again:
    the barrier behind every wait is followed by the group's way out."""
    text = source("orb_kernels.cu")
    group = body(text, r"bool sub_group\(")
    waits = [m.end() for m in re.finditer(r"\bend_load\(\);", group)]
    assert len(waits) == 3
    for at in waits:
        assert re.match(r"\s*sync\(\);\s*if \((r == 0 && )?sm\.lost\) return leave\(\);", group[at:])
    kernel = body(text, r"void __launch_bounds__\(kSubThreads\) k_subtree\(")
    assert kernel.count("if (!__syncthreads_and(ok)) return;") == 3


def test_a_graph_is_replayed_with_the_buffers_it_was_captured_with():
    """Every device address a captured kernel can read stands in the graph's key: a buffer that
    was freed and allocated elsewhere must not be reached through an older graph."""
    level = body(source("orb_internal.cuh"), r"struct Level ")
    pointers = set(re.findall(r"\*\s*(\w+)(?=\s*[,;])", level))
    assert {"x", "hint", "hint_axis", "win_cnt", "wtot"} <= pointers
    api = source("orb_api.cu")
    keyed = set(re.findall(r"\(const void \*\)v\.(\w+)", body(api, r"level_key\(orb_ctx \*ctx, const Level &v\)")))
    keyed |= set(re.findall(r"key_add\(key, v\.(\w+)\)", api))
    for name, buffer in {"skip": "sub_flag", "sub_list": "sub_list", "slots": "batch_slots", "child_map": "batch_child"}.items():
        assert f"key_add(key, ctx->{buffer}.p)" in api
        keyed.add(name)
    keyed |= {"tot", "tot_next"}  # inside the counters
    keyed |= {"out_counts", "cells_in"}  # service calls, which are not captured
    assert pointers - keyed == set()
