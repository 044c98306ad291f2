"""Rules of the kernel sources that no output shows reliably: checked on the text of goml_b200/csrc."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "goml_b200", "csrc")


def sources():
    out = {}
    for f in sorted(os.listdir(CSRC)):
        if f.endswith((".cu", ".cuh")):
            with open(os.path.join(CSRC, f)) as fh:
                out[f] = re.sub(r"//[^\n]*|/\*.*?\*/", "", fh.read(), flags=re.S)
    return out


def functions(text):
    """(name, signature + body) of every __global__ / __device__ function of a source."""
    for m in re.finditer(r"__(?:global|device)__[^;{}=]*?(\w+)\s*\([^{};]*\)\s*(?:const\s*)?\{", text):
        depth, at = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[at], 0)
            at += 1
        name = re.sub(r"__launch_bounds__\s*\([^()]*(?:\([^()]*\))?[^()]*\)", "", m.group(0))
        yield re.search(r"(\w+)\s*\(", name).group(1), text[m.start():at]


def plain_launches(text):
    return set(re.findall(r"(\w+)(?:<[^<>;]*>)?<<<", text))


def other_uses(text):
    """The kernels of a source that are named anywhere but in their definition, a plain launch and an attribute: handed to one of
    the overlapped launches (launch_pdl, launch_pdl_stream, a lambda around them, cudaLaunchKernelEx)."""
    rest = re.sub(r"cudaFuncSetAttribute\([^;]*;|\w+(?:<[^<>;]*>)?<<<", "", text)
    kernels = {fn for fn, body in functions(text) if body.startswith("__global__")}
    return {k for k in kernels if len(re.findall(rf"\b{k}\b", rest)) > 1}


# every kernel of a chain of calls, by source
OVERLAPPED = {
    "fa_fwd_sm100.cu": {"fa_fwd_kernel", "v_to_f16_kernel"}, "fa_decode_sm100.cu": {"fa_decode_kernel", "clear_words_kernel"},
    "fp8_gemm_sm100.cu": {"fp8_gemm_tcgen05_kernel"}, "fp8_gemm_skinny.cuh": {"fp8_gemm_skinny_kernel"}, "one_cluster.cuh": {"one_cluster_kernel"},
    "fp8_quantize_sm100.cu": {"clear_word_kernel", "amax_kernel", "quant_kernel"},
    "fp8_block_glue_sm100.cu": {"clear_words_kernel", "rms_stats_kernel", "rms_stats_regs_kernel", "rms_quant_kernel", "qkv_amax_kernel", "qkv_quant_kernel",
                                "dec_q_amax_kernel", "dec_append_kernel", "dec_lengths_kernel", "o_amax_kernel", "o_quant_kernel", "quant_bf16_kernel"},
}


@pytest.mark.parametrize("name", [n for n, t in sources().items() if re.search(r"__global__|__device__", t)])
def test_no_read_only_loads_in_overlapped_kernels(name):
    # a kernel that may start before its predecessor on the stream has drained must not read through the read-only path: only
    # kernels launched plainly (<<<>>>) may
    text = sources()[name]
    assert list(functions(text))
    plain = plain_launches(text)
    for fn, body in functions(text):
        if re.search(r"__ldg\s*\(|__restrict__|ld\.global\.nc|ld\.global\.L1::no_allocate\.nc", body):
            assert fn in plain, f"{name}: {fn} reads through the read-only path"
    assert not plain & other_uses(text)


@pytest.mark.parametrize("name", OVERLAPPED)
def test_overlapped_kernels_are_seen(name):
    text = sources()[name]
    assert other_uses(text) == OVERLAPPED[name]
    # a plain launch added to any of them is one the test above objects to
    for kernel in OVERLAPPED[name]:
        assert plain_launches(f"{text}\n{kernel}<<<1, 1>>>();") & other_uses(f"{text}\n{kernel}<<<1, 1>>>();") == {kernel}


def test_the_lane_that_copies_v_is_ordered_behind_the_lane_that_saw_the_flag():
    # the attention producer: every lane acquires a flag of its own and one elected lane issues the copies; between the vote and
    # the proxy fence stands a warp barrier, which orders memory among the lanes (a vote does not)
    body = dict(functions(sources()["fa_fwd_sm100.cu"]))["wait_v_chunk"]
    assert re.search(r"ld\.acquire\.gpu.*__ballot_sync.*__syncwarp\(\);\s*asm volatile\(\"fence\.proxy\.async", body, flags=re.S)


@pytest.mark.parametrize("name", [n for n, t in sources().items() if "mbar_wait" in t and n != "sm100_ptx.cuh"])
def test_bounded_waits_are_left_by_whole_warps(name):
    # roles run on whole warps: a lane that leaves a loop on its own outcome of a wait strands the others in the loop's next
    # warp-wide operation
    assert not re.search(r"\bmbar_(try_)?wait\s*[(<]", sources()[name])


def test_the_warp_wait_votes():
    body = dict(functions(sources()["sm100_ptx.cuh"]))["mbar_wait_warp"]
    assert re.search(r"__all_sync\(0xffffffffu,\s*mbar_try_wait\(", body) and "mbar_wait(" not in body
    # the only other way out is voted on as well
    assert body.count("return") == 2 and re.search(r"if \(__any_sync\([^;]*\) return false;", body)


def test_calls_on_different_streams_do_not_hold_one_lock_over_their_launches():
    # the lock of a GPU's table of kept buffers guards the look-up; what is held over the launches belongs to the stream
    text = sources()["fa_api.cu"]
    assert re.search(r"lock = std::unique_lock<std::mutex>\(k->busy\)", text)
    assert not re.search(r"unique_lock<std::mutex>\([^)]*shared", text)


def test_a_part_of_the_decode_line_comes_from_one_reading_of_the_lengths():
    # two readings that disagree (a caller that rewrites the lengths while the kernel runs) must not make an address: the sequence
    # that a unit falls in, its length and the units before it are taken from the same values
    body = re.search(r"auto segment_at = .*?\n    \};", sources()["fa_decode_sm100.cu"], flags=re.S).group(0)
    assert body.count("lane_len(") == 1 and "seq_len_of" not in body and "len_of(" not in body.replace("lane_len(", "")


def test_the_first_block_of_a_decode_cluster_outlives_what_its_peers_store():
    # every way out of the cluster form that the first block may take, by whatever it has read of the length, is behind both phases
    text = re.sub(r"//[^\n]*", "", sources()["fa_decode_sm100.cu"])
    kernel = text[text.index("find_piece(false);"):]
    kernel = kernel[:kernel.index("if (!whole) {\n            int parts")]   # behind it: the workspace's merge, not the cluster's
    # no keys, or all of them; a part, behind which a peer may go
    assert re.search(r"if \(CLUSTER && run == 0 && \(nothing \|\| seg\.c_end == seg\.n_chunks\)\) \{\s*__syncwarp\(\);\s*cluster_wait\(\);\s*cluster_here\(\);\s*"
                     r"if \(nothing\) cluster_wait\(\);\s*\}\s*if \(nothing\) return;", kernel)
    assert "if (CLUSTER && !whole) cluster_wait();" in kernel
    tail = kernel[kernel.rindex("if (CLUSTER) {"):]
    assert re.match(r"if \(CLUSTER\) \{\s*__syncwarp\(\);\s*if \(!whole\) cluster_arrive\(\);\s*if \(seg\.c_begin != 0\) return;\s*cluster_wait\(\);\s*if \(whole\) return;",
                    tail)
    # no other way out than these, a lambda's and the end
    assert len(re.findall(r"\breturn;", kernel)) == 5
    assert len(re.findall(r"cluster_(?:wait|arrive|here)\(\)", kernel)) == 6


def decode_cluster(readings, chunks_per_split, stays):
    """The cluster's blocks by what each has read (in chunks): every order in which they may run.  True where a store can meet a block that has gone."""
    size = len(readings)

    def steps(rank, chunks):
        used = -(-chunks // chunks_per_split)
        each = chunks_per_split * -(-used // size)
        begin, end = rank * each, min(chunks, (rank + 1) * each)
        if begin >= end or (begin == 0 and end == chunks):
            return ["arrive", "wait", "arrive", "wait", "gone"] if stays and rank == 0 else ["arrive", "gone"]
        return ["arrive", "wait", "store", "arrive", "gone"] if rank else ["arrive", "wait", "store", "arrive", "wait", "gone"]

    plans = [steps(r, n) for r, n in enumerate(readings)]
    seen, todo, bad = set(), [(0,) * size], False
    arrivals = [[sum(s == "arrive" for s in plan[:i]) for i in range(len(plan) + 1)] for plan in plans]
    while todo:
        at = todo.pop()
        if at in seen:
            continue
        seen.add(at)
        gone = [i == len(p) for i, p in zip(at, plans)]
        moved = False
        for r, plan in enumerate(plans):
            if gone[r]:
                continue
            step = plan[at[r]]
            # a phase ends when every block has arrived at it or gone
            if step == "wait" and not all(g or arrivals[q][at[q]] >= arrivals[r][at[r]] for q, g in enumerate(gone)):
                continue
            bad |= step == "store" and gone[0]
            moved = True
            todo.append(at[:r] + (at[r] + 1,) + at[r + 1:])
        assert moved or all(gone), (readings, at)   # no order stands still
    return bad


@pytest.mark.parametrize("size,chunks_per_split", [(2, 1), (3, 1), (3, 2), (4, 1)])
def test_readings_that_disagree_store_to_no_block_that_has_gone(size, chunks_per_split):
    import itertools
    most = size * chunks_per_split
    readings = list(itertools.product(range(most + 1), repeat=size))
    assert not any(decode_cluster(r, chunks_per_split, True) for r in readings)
    # the model sees the fault of a first block that leaves by its own reading, and only where readings disagree
    assert decode_cluster((1,) + (most,) * (size - 1), chunks_per_split, False)
    assert not any(decode_cluster((n,) * size, chunks_per_split, False) for n in range(most + 1))


@pytest.mark.parametrize("name", sources())
def test_registers_stay_where_a_launch_puts_them(name):
    # an attention form that moved registers between its warps raised illegal accesses after a harmless change of its code, and the
    # cause was not found
    assert "setmaxnreg" not in sources()[name]
