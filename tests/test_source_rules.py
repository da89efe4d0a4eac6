"""Rules that the device code keeps and that no run shows: what they guard against is a
wait that runs out, or a load that a compiler may but need not turn into a stale one. They
are checked on the sources, without a GPU."""
import os
import re

from conftest import ROOT

CSRC = os.path.join(ROOT, "libisdf_b200", "csrc")


def _functions(name):
    """The top-level functions of a source, each from its first line to its closing brace."""
    text = open(os.path.join(CSRC, name)).read()
    text = re.sub(r"//[^\n]*", "", text)
    return [f for f in re.split(r"(?m)^}.*$", text) if "(" in f]


def test_symmetric_products_report_a_wait_that_ran_out():
    """Whoever queues a symmetric product reads its error flag back afterwards."""
    users = [f for f in _functions("check.cu") if "dsyrk_store(" in f]
    assert len(users) == 3  # the check, the sampled check, the Coulomb matrix
    for f in users:
        assert "products_done(" in f[f.rindex("dsyrk_store("):], f


def test_no_warp_of_a_tile_leaves_before_a_barrier():
    """A tile's run() gives each warp its own answer where a wait runs out: one may
    have its product while another has none. A kernel with a barrier behind run()
    must not let the second one return before it, or the first waits for ever."""
    early = re.compile(r"if \(!\w+\.run\((?:[^;{]|\n)*?\)\)\s*return")
    seen = 0
    for name in ("fit.cu", "qrcp.cu", "check.cu"):
        for f in _functions(name):
            if ".run(" not in f:
                continue
            seen += 1
            behind = f[f.index(".run("):]
            if "bar.sync" in behind or "__syncthreads" in behind:
                assert not early.search(f), f
    assert seen >= 4


def test_early_kernels_read_no_loop_data_as_read_only():
    """A kernel that begins with after_previous() is resident while the kernel before it
    still writes. A __restrict__ pointer lets the compiler read through the read-only
    path, which is valid for data that does not change in the kernel's lifetime: the
    loops' constant operands, and outputs that the kernel does not read."""
    constant = {"qrcp.cu": {"Ac", "Bc"}, "kmeans.cu": {"pidx"}}
    written = {"k_normalise": {"Q", "Qm"}}
    early = 0
    for name, allowed in constant.items():
        for f in _functions(name):
            is_early = "after_previous();" in f
            early += is_early
            if not is_early and ("__global__" in f or "__device__" not in f):
                continue  # a kernel launched in order, or host code
            kernel = re.search(r"(\w+)\s*\((?:const|int|double|bool)", f)
            ok = allowed | written.get(kernel.group(1) if kernel else "", set())
            found = set(re.findall(r"__restrict__\s+(\w+)", f))
            assert found <= ok, (name, found - ok)
    assert early == 12


def test_launches_ahead_of_a_loop_are_checked():
    """Making a loop's graph clears the errors it meets itself, so the launches issued
    ahead of it are checked before it."""
    text = open(os.path.join(CSRC, "loop_graph.h")).read()
    start = text[text.index("int start("):text.index("int finish(")]
    assert start.index("round(") < start.index("ISDF_CHECK_LAUNCH();")
    for name in ("kmeans.cu", "qrcp.cu"):
        text = open(os.path.join(CSRC, name)).read()
        assert len(re.findall(r"loop(?:\.|->)finish\(", text)) == \
            len(re.findall(r"loop(?:\.|->)start\(", text)) > 0


def test_mapping_host_memory_clears_only_its_own_error():
    """An earlier launch's error may be waiting to be seen when a host buffer is mapped:
    only the branch of a refused mapping clears the last error."""
    text = open(os.path.join(CSRC, "readback.cu")).read()
    assert text.count("cudaGetLastError()") == 1
    helper = text[text.index("bool map_host("):]
    helper = helper[:helper.index("\n}\n")]
    assert "return true;" in helper[:helper.index("cudaGetLastError()")]
    assert text.count("cudaHostAlloc(") == 1
