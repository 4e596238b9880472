"""A call that was refused for want of device memory leaves nothing behind: the calls after it run."""
import ctypes
import os
import sys

import pytest

sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
from golden_sets import compare, golden_case, load_digests  # noqa: E402

from graphaligner_gb300._lib import GAError  # noqa: E402
from graphaligner_gb300.align import Aligner, preset  # noqa: E402
from graphaligner_gb300.extend import DeviceGraph, Extender, ExtendParams  # noqa: E402

pytestmark = pytest.mark.gpu

TOO_MUCH = 1 << 50


def refused(dgraph):
    with pytest.raises(GAError, match="out of memory"):
        Extender(dgraph, arena_bytes=TOO_MUCH)


def test_calls_after_a_refused_extender(cuda_lib):
    g, batch = golden_case("vg50k")
    dgraph = DeviceGraph(g)
    ext = Extender(dgraph, arena_bytes=256 << 20)
    refused(dgraph)
    assert not compare(ext.run(ExtendParams(bandwidth=10), batch), load_digests("vg50k", 10))
    refused(dgraph)
    again = DeviceGraph(g)
    refused(again)
    Aligner(Extender(again, arena_bytes=64 << 20), g, preset("vg")).close()


def test_upload_after_another_call_of_the_process_failed(cuda_lib):
    # the library's own CUDA runtime, found among the process's symbols or beside it
    for name in (None, "libcudart.so.13", "libcudart.so"):
        try:
            malloc = ctypes.CDLL(name).cudaMalloc
            break
        except (OSError, AttributeError):
            continue
    else:
        pytest.skip("no CUDA runtime to call")
    p = ctypes.c_void_p()
    assert malloc(ctypes.byref(p), ctypes.c_size_t(TOO_MUCH)) != 0
    DeviceGraph(golden_case("vg50k")[0])
