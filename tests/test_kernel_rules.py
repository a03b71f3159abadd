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
    """The classify pass sets the error flag while its other CTAs start, and its warps meet at named
    barriers, which wait for warps that have left: it decides on the level above's count alone,
    which no CTA of it changes. Every other kernel that flags an error is through with its own test
    of the flag: the last of several passes does it, the first one tests."""
    text = source("orb_kernels.cu")
    late = body(text, r"bool level_late\(const Level &v\)")
    assert "done[v.depth - 1]" in late and late.count("error") == 1 and "atomicExch(&v.counters->error" in late
    classify = body(text, r"k_part_classify\(const __grid_constant__ Level v\)")
    assert "if (level_late(v)) return;" in classify and "level_failed" not in classify
    flag = "atomicExch(&v.counters->error, 1u)"
    setters = {m.start() for m in re.finditer(re.escape(flag), text)}
    known = 0
    for start, guard in [(r"bool level_late\(", "threadIdx.x == 0"), (r"k_part_classify\(", "lane == 0"),
                         (r"void resolve_cell\(", "v.pass == v.last_pass"), (r"void __launch_bounds__\(kThreads, 4\) k_whist\(", "v.pass == v.last_pass"),
                         (r"bool sub_group\(", "ti == 0")]:
        block = body(text, start)
        assert re.findall(r"if \(([^()]*)\) " + re.escape(flag), block) == [guard]
        known += 1
    assert len(setters) == known
    for kernel in (r"void __launch_bounds__\(kThreads, 4\) k_whist\(", r"kHistBlocks512 : 1\)\) k_hist\("):
        assert "if (v.pass == 0 && level_failed(v)) return;" in body(text, kernel)


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
    the barrier behind every wait is the group's way out."""
    text = source("orb_kernels.cu")
    group = body(text, r"bool sub_group\(")
    assert len(re.findall(r"\bend_load\(\)", group)) == 3
    assert len(re.findall(r"if \(!come_all\((r > 0 \|\| )?end_load\(\)\)\) return leave\(\);", group)) == 3
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


def test_buffers_are_sized_before_the_key_is_taken():
    """A buffer that grows after its address went into the key would leave a graph under the key
    of the buffer that was freed."""
    api = source("orb_api.cu")
    for build in (r"orb_status build_single\([^;{]*(?=\{)", r"orb_status build_batch_impl\([^;{]*(?=\{)"):
        block = body(api, build)
        key, run = block.index("level_key("), block.index("run_graphed(")
        assert not [b for b in re.findall(r"ctx->(\w+)\.ensure\(", block[key:run]) if f"v.{b}" not in block[key:run]]


def test_the_count_passes_keep_to_their_ctas_per_sm():
    """hist_blocks_per_sm bounds the count passes' CTAs on every level, those of few tiles too, whose
    CTAs are larger and take a tile each."""
    block = body(source("orb_api.cu"), r"orb_status run_bisection\([^{]*(?=\{)")
    most = re.search(r"most = std::min<uint32_t>\(kHistBlocks512, ctx->tune\.hist_blocks_per_sm\);", block)
    assert most and "tiles <= (uint64_t)ctx->num_sms ? 1024 : (tiles <= most * (uint64_t)ctx->num_sms ? 512 : kThreads)" in block
