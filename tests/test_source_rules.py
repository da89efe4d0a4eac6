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
