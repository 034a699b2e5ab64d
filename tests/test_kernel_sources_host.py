"""Rules of the CUDA programming model that no run can show to be kept, checked
on the kernels' sources."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tensormesh_gb300", "csrc")


def body(path, head):
    """Source of the function whose text starts at ``head``, comments removed."""
    src = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, path)).read())
    at = src.index("{", src.index(head))
    depth = 0
    for i in range(at, len(src)):
        depth += {"{": 1, "}": -1}.get(src[i], 0)
        if depth == 0:
            return src[at:i]
    raise AssertionError(head)


def test_clusters_meet_before_they_write_each_others_shared_memory():
    """A CTA may write into another's shared memory only after that one has
    started: a cluster barrier stands before every kernel's first cluster_sum."""
    solve = body("pcg_sell.cu", "pcg_sell_hs_kernel(int64_t n")
    assert solve.index("cluster_barrier()") < solve.index("cluster_sum<")
    batch = body("batched.cu", "batched_assemble_pcg_kernel(BatchArgs A)")
    assert batch.index("cl.sync()") < batch.index("cluster_sum<")


def test_a_refused_cluster_size_leaves_no_error_for_the_launch():
    """A CUDA error stays until it is read.  Every refusal inside the search
    for a cluster size reads it, so that a smaller size launches cleanly."""
    search = body("pcg_sell.cu", "int sell_launch(int64_t n_slices")
    loop = search[search.index("for (int nb = 16"):search.index("how.mode = kCluster")]
    refusals = re.findall(r"if \(([^;{]*cuda[^;{]*)\) \{\s*cudaGetLastError\(\);\s*continue;\s*\}", loop)
    calls = re.findall(r"cuda(?:FuncSetAttribute|OccupancyMaxActiveClusters)\(", loop)
    assert len(calls) == 3 and sum(c.count("cudaSuccess") for c in refusals) == 3
