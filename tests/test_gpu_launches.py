"""The number of kernels that a call is said to launch, against the kernels of its graph."""

import ctypes

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from cubam_b200 import _lib, bgzf as G  # noqa: E402
from cubam_b200.batch import inflate_launches  # noqa: E402


def _kernels(graph) -> int:
    cu, handle = ctypes.CDLL("libcuda.so.1"), ctypes.c_void_p(graph.raw_cuda_graph())
    n = ctypes.c_size_t()
    assert cu.cuGraphGetNodes(handle, None, ctypes.byref(n)) == 0
    nodes = (ctypes.c_void_p * n.value)()
    assert cu.cuGraphGetNodes(handle, nodes, ctypes.byref(n)) == 0
    kinds = []
    for node in nodes:
        kind = ctypes.c_int()
        assert cu.cuGraphNodeGetType(ctypes.c_void_p(node), ctypes.byref(kind)) == 0
        kinds.append(kind.value)
    return kinds.count(0)


@pytest.mark.parametrize("check_crc", [True, False])
@pytest.mark.parametrize("pipeline", [-1, 0, 2])
@pytest.mark.parametrize(("form", "jobs"), [(1, 5), (2, 5), (3, 0), (3, 1), (3, 39), (3, 700), (3, 4000), (3, 65_536)])
def test_launches_are_counted(form, jobs, pipeline, check_crc):
    table = torch.zeros((max(jobs, 1), 4), dtype=torch.int64, device="cuda")  # not run: only captured
    summ = torch.zeros(64, dtype=torch.uint8, device="cuda")
    out = torch.zeros(64, dtype=torch.uint8, device="cuda")
    ws = torch.empty(G.inflate_workspace_bytes(jobs, 64, form), dtype=torch.uint8, device="cuda")
    _lib.lib.cb_set_param(_lib.PARAM_DECODE_PIPELINE, pipeline)
    try:
        g = torch.cuda.CUDAGraph(keep_graph=True)
        with torch.cuda.graph(g):
            G.launch_inflate(table.data_ptr(), jobs, out.data_ptr(), 64, check_crc, summ.data_ptr(), ws, form)
        assert inflate_launches(form, jobs, 64, check_crc, captured=True) == _kernels(g)
        eager = inflate_launches(form, jobs, 64, check_crc)
        two = form == 3 and (pipeline == 2 and jobs >= 2 or pipeline == -1 and jobs >= 20 * 148)
        assert eager == _kernels(g) + (two and pipeline == -1 and jobs < 65_536) * (eager - 4) // 2
    finally:
        _lib.lib.cb_set_param(_lib.PARAM_DECODE_PIPELINE, -1)
