import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
for p in (ROOT, os.path.join(ROOT, "graph500-bfs_b200"), os.path.join(ROOT, "oracle")):
    if p not in sys.path:
        sys.path.insert(0, p)


def reference_program(name):
    """Path of one of the reference's own programs (oracle/ref/Makefile).  They
    are built where the reference tree is: a test that needs one is skipped
    where none could be, and fails where the tree was there and it is missing."""
    out = os.path.join(ROOT, "oracle", "_ref")
    path = os.path.join(out, name)
    if not os.path.exists(path):
        if os.path.exists(os.path.join(out, "stock", ".tree")):
            pytest.fail("%s missing: `make -C oracle/ref`" % name)
        pytest.skip("%s: no reference tree to build it from" % name)
    return path


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (B200)")


@pytest.fixture(scope="session")
def built():
    import __graft_entry__

    __graft_entry__.build()
    return True
