import json
import os
import sys

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
sys.path.insert(0, ROOT)
sys.path.insert(0, HERE)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (B200, sm_100a)")
    config.addinivalue_line("markers", "last: runs after every other test of the session")


def _needs_a_dropin_that_cannot_be_had(item):
    """The drop-in library is asked for (fixture gpu_lib), but is neither built nor are the parser
    sources there that it is built from: such a test fails in its set-up."""
    ref = os.environ.get("HEVC_REF_DIR", os.path.join(os.path.dirname(ROOT), "reference"))
    return "gpu_lib" in getattr(item, "fixturenames", ()) and not os.path.isdir(os.path.join(ref, "src")) and \
        not os.path.exists(os.path.join(ROOT, "hevc.js_b200", "libhevcdec_gpu.so"))


def pytest_collection_modifyitems(session, config, items):
    """Tests marked `last`, then those whose drop-in library cannot be had, run at the end (in
    their collected order), so that under -x a failure there stops nothing else."""
    def rank(item):
        return 2 if _needs_a_dropin_that_cannot_be_had(item) else 1 if item.get_closest_marker("last") else 0
    items.sort(key=rank)


@pytest.fixture(scope="session")
def hb():
    import __graft_entry__ as ge
    mod = ge.load_package()
    from hevc_b200 import build
    build.build_synth()
    return mod


@pytest.fixture(scope="session")
def port(hb):
    import oracle
    if not os.path.exists(oracle.PORT_SO):
        oracle.build(with_ref=False)
    return oracle.port()


@pytest.fixture(scope="session")
def golden():
    with open(os.path.join(HERE, "golden", "digests.json")) as f:
        return json.load(f)["cases"]


@pytest.fixture(scope="session")
def gpu_ctx(hb):
    from hevc_b200 import build
    build.build_gpu()
    ctx = hb.Context(0)
    yield ctx
    ctx.close()
