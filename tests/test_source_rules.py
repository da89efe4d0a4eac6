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
