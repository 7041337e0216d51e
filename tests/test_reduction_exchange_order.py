"""Order of the shared and global exchanges of the on-chip Householder reductions, read from their
source (CPU only: a race shows on a GPU as a rare wrong column, not as a failing run).

A column of the cluster reduction is: products, sums, remote stores, barrier_arrive, the reflector's
scalars, barrier_wait, vectors, block barrier.  The barrier's wait returns once every warp has
arrived, so whatever a warp reads between its arrive and its wait may already be overwritten by
another warp's code after the wait."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gfn1-rs_b200", "csrc")


def _source(name):
    with open(os.path.join(CSRC, name)) as fh:
        return re.sub(r"//[^\n]*", "", fh.read())


def _index(expression, k):
    """Buffer number of `base + (...) * NW` or `[(...) * NW + wid]` at column k; 0 without one."""
    m = re.search(r"\(\(?k(?: \+ (\d))?\)? & 1\) \* NW", expression)
    return None if not m else (k + int(m.group(1) or 0)) & 1


def test_cluster_scalars_are_not_overwritten_before_they_are_read():
    text = _source("tridiag_cluster.cuh")
    body = text[text.index("cl.barrier_arrive();"):]
    split = body.index("cl.barrier_wait();")
    overlapped, after = body[:split], body[split:body.index("cluster_write_out<C>(O, k, sm);")]
    reads = re.findall(r"tree_sum<NW>\((red\w*[^;,]*?)\)[,;]", overlapped)
    writes = re.findall(r"(red\w*\[[^\]]*\]) =", after)
    assert reads and writes
    for r in reads:
        for w in writes:
            if re.match(r"\w+", r).group() != re.match(r"\w+", w).group():
                continue
            for k in (0, 1):
                assert _index(r, k) is not None and _index(w, k) is not None, (r, w)
                assert _index(r, k) != _index(w, k), (r, w)  # read at column k, written for column k + 1
                assert _index(r, k + 1) == _index(w, k)


def test_cluster_shared_memory_holds_its_buffers():
    text = _source("tridiag_cluster.cuh")
    body = text[text.index("cluster_phase("):]
    assert "xyc = redxy + NW" in body and "redxy = red + 2 * NW" in body
    assert "3 * NW + 2 * C + kOut" in text


def test_grid_readers_fence_between_the_marks_and_the_reuse_of_their_slots():
    """Marks are made in phase C of column 0 (modulo kMark), published by the owner's fence before its
    values of a later column p, seen by a reader with that column's values, and needed before the
    look at column kMark.  So a reader fences in every thread after its wait of a column in
    p .. kMark - 1, at least once per kMark columns."""
    text = _source("tridiag_grid.cuh")
    const = {m.group(1): int(m.group(2)) for m in re.finditer(r"(k\w+) = (\d+)\b", text)}
    mark, ring = const["kMark"], const["kRing"]
    assert ring == 2 * mark
    body = text[text.index("__forceinline__ bool grid_phase("):text.index("__forceinline__ bool grid_tridiag(")]
    fences = re.findall(r"if \((wid == 0 && )?\(k & \(GS::kMark - 1\)\) == (?:GS::)?(\w+)\) (?:ring_fence|__threadfence)\(\);",
                        body)
    column = {bool(owner): int(const.get(c, c)) for owner, c in fences}
    assert set(column) == {True, False}, "one fence by the owner's publishing warp, one by every reading thread"
    published = column[True] + 1  # the first values stored after the owner's fence
    assert 1 <= column[True] and published <= column[False] < mark
    at = body.index("ring_fence();", body.index("double2 g[NQ];"))
    wait, reader = body.index("if (wait) {"), body.rindex("ring_fence();")
    assert at < wait < reader < body.index("double xy = 0.0;")
    assert re.search(r"fence\.acq_rel\.gpu", text)


def test_every_run_starts_with_clear_error_flags():
    """A wait that gave up raises the flag of its slot for the run it belongs to: the kernel that begins
    a run clears both barriers of every slot, before the reductions poll them."""
    text = _source("wide.cuh")
    body = text[text.index("__global__ void wide_begin_kernel("):]
    body = body[:body.index("\n}\n")]
    assert re.search(r"w\.sync\[0\] = w\.sync\[1\] = GroupSync\{0u, 0u, 0, 0\};", body)
    run = text[text.index("cudaError_t run_wide("):]
    assert run.index("wide_begin_kernel<<<") < run.index("wide_autotune(") < run.index("reduce_all(")


def test_no_list_is_uploaded_that_the_run_does_not_wait_for():
    """The lists of active slots are copied from one pinned array that the next run sorts anew; a list whose
    copy is still under way when run_wide returns may be read half sorted.  So the kernels that write the
    results, after the last synchronisation, take the list that the binding of the slots uploaded."""
    text = _source("wide.cuh")
    run = text[text.index("cudaError_t run_wide("):]
    run = run[:run.index("\n}\n")]
    results = run[run.index("X.act = R.d_all"):]
    assert "upload_act(" not in results and "wide_pw_kernel<<<" in results and "wide_results_kernel<<<" in results
    assert "wide_pw_kernel<<<" not in run[:run.index("X.act = R.d_all")]
