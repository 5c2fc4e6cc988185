"""Orders that the kernels' sources have to keep because no run can be relied on to show that they are broken: a store that comes too
early usually still lands where it should.  The sources are read as text."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "bitsqueeze-llm_b200", "csrc")


def block(text, at):
    """The balanced {...} that opens at or behind `at`."""
    start, depth = text.index("{", at), 0
    for i in range(start, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[start: i + 1]
    raise ValueError("unbalanced braces")


def sources():
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        with open(path) as f:
            text = f.read()
        yield os.path.basename(path), re.sub(r"//[^\n]*", "", re.sub(r"/\*.*?\*/", "", text, flags=re.S))


def kernels():
    """name -> (parameters, body) of every __global__ function."""
    found = {}
    for _, text in sources():
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s+)?(\w+)\s*\(", text):
            end, depth = m.end(), 1
            while depth:
                depth += {"(": 1, ")": -1}.get(text[end], 0)
                end += 1
            found[m.group(1)] = (text[m.end(): end - 1], block(text, end))
    return found


KERNELS = kernels()


def test_kernels_are_found():
    assert {"ring_jacobi_kernel", "block_jacobi_kernel", "cholesky_kernel", "gemm_kernel", "topk_rows_group_kernel"} <= set(KERNELS)


@pytest.mark.parametrize("name", sorted(n for n, (_, body) in KERNELS.items() if "this_cluster()" in body))
def test_clusters_meet_before_they_store_into_one_another(name):
    """CTAs of a cluster are scheduled together but need not have started together: shared memory of another CTA may be touched only
    behind a barrier of the cluster."""
    body = KERNELS[name][1]
    remote = min(m.start() for m in re.finditer(r"map_shared_rank|st\w*_async\w*\(|put_remote", body))
    assert 0 <= body.find("cluster.sync()") < remote


CHAINED = sorted(n for n, (_, body) in KERNELS.items() if "chain_begin()" in body)
# inputs that are complete before the kernel in front of theirs has started: the caller's matrix
COMPLETE = {"frontend_select_kernel": {"in"}, "frontend_encode_kernel": {"in"}}


def test_kernels_launched_chained_wait():
    launched = set()
    for _, text in sources():
        for m in re.finditer(r"launch_chained\(", text):
            target = re.match(r"\s*(\w+)", text[m.end():])
            if target.group(1) != "void":
                launched.add(target.group(1))
    assert len(launched) >= 12 and launched <= set(CHAINED)


def test_no_kernel_lets_the_next_one_in_early():
    """CTAs that wait for a long kernel hold SMs that other streams want: four calls side by side took 1.7 times as long."""
    assert not [name for name, text in sources() if "launch_dependents" in text]


@pytest.mark.parametrize("name", CHAINED)
def test_inputs_of_chained_kernels_are_read_behind_the_wait(name):
    """While a chained kernel waits, the kernel before it may still write its inputs.  A `const ... *__restrict__` parameter promises that
    nobody does, and the compiler may then read it through the read-only path and in front of the wait."""
    params, body = KERNELS[name]
    promised = set(re.findall(r"const\s+\w+\s*\*\s*__restrict__\s*(\w+)", params))
    assert promised <= COMPLETE.get(name, set())
    assert "__ldg(" not in body
    before = body[1: body.index("chain_begin()")]
    assert before.count("{") == before.count("}")                # not in a branch
    assert not re.search(r"\b(?:if|for|while)\s*\(|__syncthreads|cluster\.sync\(\)", before)


def test_raw_slots_are_handed_back_behind_a_proxy_fence():
    """A copy into shared memory is not ordered behind another thread's reads by that thread's arrival on an mbarrier alone."""
    text = dict(sources())["bsq_gemm_tma.cu"]
    assert not re.search(r"mbar_arrive\(&bars\.raw_empty", text) and text.count("raw_read_done(&bars.raw_empty") == 3
    done = block(text, text.index("void raw_read_done"))
    assert 0 <= done.find("fence_proxy_async_smem()") < done.find("mbar_arrive(")


def test_cholesky_announces_every_row_before_it_counts_itself_out():
    """CholeskySync has to be zero between launches also behind a wait that ran out: the warp that announces the last row and the thread
    that clears the words are different ones."""
    body = KERNELS["cholesky_kernel"][1]
    work, count = body.index("cholesky_factor("), body.index("atomicAdd(&sync->done")
    assert re.search(r"(?m)^    __syncthreads\(\);", body[work: count])


def test_ring_waits_for_stores_in_flight_before_it_leaves():
    """A CTA whose wait for a neighbour's column ran out must not give its shared memory back while that column may still come."""
    body = KERNELS["ring_jacobi_kernel"][1]
    leave = body[body.index("float *sv = "):]
    drain, last = leave.find("if (failed)"), leave.rfind("cluster.sync()")
    assert 0 <= drain < last and leave[drain: last].count("mbar_wait_bounded(") == 2


def test_cholesky_cluster_drains_behind_every_wait_that_may_run_out():
    """The thread that looks whether a wait ran out belongs to one warp, the waits to others: without a barrier of the CTA in front it may
    look too early, and a copy that is still under way lands in shared memory that the CTA has given back."""
    body = KERNELS["cholesky_cluster_kernel"][1]
    roles = block(body, body.index("if (warp == 0)"))
    at = body.index("    } else {", body.index(roles))        # the last role
    drain, last = body.index("&& bars->failed)"), body.rindex("cluster.sync()")
    assert at < drain < last
    between = body[body.index("    if (T) {", at): drain]
    inverse = block(between, 0)
    behind = between[between.index(inverse) + len(inverse):]
    assert "__syncthreads();" in behind
    assert block(body, drain).count("cc_wait(") == 4


def test_tensor_memory_is_read_by_whole_warps():
    """tcgen05.ld is executed by all lanes of a warp together: what decides on the way to one is the same in all of them."""
    text = dict(sources())["bsq_gemm_tma.cu"]
    pre = re.search(r"const bool pre = ([^;]*);", text).group(1)
    assert "row - lane + 32 <= g.M" in pre and not re.search(r"\brow <", pre)
    assert "__all_sync(0xffffffffu, mbar_wait_bounded(&bars.acc_full[set]" in text
