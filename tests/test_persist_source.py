"""Rules of the device code that no run can show reliably, checked in the
source.

A block of a cluster may only touch a peer's shared memory once that peer
runs; nothing but a cluster barrier says so (CUDA programming guide,
distributed shared memory).  The sums of the single-cluster solves store into
every block before their own barrier, so the scope's constructor has to hold
one, after the block's own initialisation."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cufoam_gb300", "csrc")


def _body(text, start):
    """The brace-balanced body that opens at or after `start`."""
    i = text.index("{", start)
    depth, j = 0, i
    while True:
        depth += {"{": 1, "}": -1}.get(text[j], 0)
        j += 1
        if depth == 0:
            return text[i:j]


def _code(name):
    text = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*|/\*.*?\*/", "", text, flags=re.S)


def test_cluster_occupancy_is_asked_for_the_launched_kernel_and_size():
    """A kernel's cluster may fit where another's does not (registers, static
    and dynamic shared memory): the query names the kernel of the launch and
    the largest dynamic size a launch may have, and every choice of the single
    cluster asks it."""
    text = _code("persist.cu")
    fits = _body(text, text.index("bool persist_cluster_fits("))
    assert "cfg.dynamicSmemBytes = persist_smem_limit(true);" in fits
    assert "cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg)" in fits
    for name in ("persist.cu", "persist_mixed.cu"):
        code = _code(name)
        uses = re.findall(r"if \(([^{]*CF_PERSIST_CLUSTER_ROWS[^{]*)\) \{", code)
        assert uses and all("persist_cluster_fits(ctx, " in u and "kScopeCluster" in u for u in uses)


def test_cluster_scope_waits_for_its_blocks_before_the_first_remote_store():
    text = _code("persist.cuh")
    scope = _body(text, text.index("struct ClusterSync"))
    ctor = _body(scope, re.search(r"ClusterSync\(const PersistGrid &[^)]*\)[^{]*", scope).end() - 1)
    assert "st.shared::cluster" not in ctor
    last = [line.strip() for line in ctor.strip("{} \n").splitlines() if line.strip()][-1]
    assert last == "barrier();", last
    barrier = _body(scope, scope.index("bool barrier()"))
    assert barrier.index("barrier.cluster.arrive.release") < barrier.index("barrier.cluster.wait.acquire")


def test_fast_order_reductions_carry_no_scratch_of_the_reference_order():
    """Static shared memory of the CSR passes comes out of their L1: callers
    that never sum in the reference order say so at compile time."""
    calls = [c for name in ("solve_fast.cu", "mixed.cu", "distributed.cu")
             for c in re.findall(r"grid_reduce<([^>]*)>\(([^;{]*?)\) &&", _code(name))]
    assert calls and all(args.split(",")[-1].strip() == "false" for args, _ in calls)


def test_the_in_place_scan_may_alias():
    """The slice lengths are turned into offsets in place: the kernel that
    reads and writes them must not promise the compiler distinct arrays (such
    loads may go through the read-only cache)."""
    text = _code("matrix.cu")
    in_place = re.search(r"exclusive_scan\(ctx, [^,]*, (\w+->s_off\.as<int32_t>\(\)), \1,", text)
    scan = re.search(r"void k_scan_blocks\(([^)]*)\)", text).group(1)
    assert in_place and "__restrict__" not in scan


def test_reference_order_products_keep_their_registers():
    """Without a bound of four blocks per SM the compiler takes 48 registers
    and spills in these two (a sequential sum is a call): 4% to 13% at large
    sizes."""
    text = _code("solve_fp64.cu")
    for kernel in ("k_cg_spmv", "k_rich_step"):
        assert f"__launch_bounds__(kBlock, 4) {kernel}(" in text
