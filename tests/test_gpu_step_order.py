"""Launches whose order the kernels behind them rely on: a step's metadata is complete before anything that reads it early may start."""
import ctypes as C

import pytest

from ingot_b200 import models as M

pytestmark = pytest.mark.gpu


class EdgeData(C.Structure):
    """CUgraphEdgeData; type 0: an ordinary edge (all of the work before is over and seen), 1: a programmatic one."""
    _fields_ = [("from_port", C.c_ubyte), ("to_port", C.c_ubyte), ("type", C.c_ubyte), ("reserved", C.c_ubyte * 5)]


def edge_types(raw):
    """Types of the edges of a captured graph."""
    edges = C.CDLL("libcuda.so.1").cuGraphGetEdges_v2
    n = C.c_size_t(0)
    assert edges(C.c_void_p(raw), None, None, None, C.byref(n)) == 0
    a, b, data = (C.c_void_p * n.value)(), (C.c_void_p * n.value)(), (EdgeData * n.value)()
    assert edges(C.c_void_p(raw), a, b, data, C.byref(n)) == 0
    return [d.type for d in data]


@pytest.mark.parametrize("table_kind", ["rows of whole pieces", "odd rows", "two tables"])
def test_nothing_starts_before_the_metadata_is_there(table_kind):
    """Captured only, as a step's first two launches: the second one hangs on the fetch by an ordinary edge."""
    import torch
    L = M.lib()
    n = 62 if table_kind == "odd rows" else 64
    host, meta = torch.zeros(64, dtype=torch.int32, pin_memory=True), torch.empty(64, dtype=torch.int32, device="cuda")
    table, out = torch.zeros(8, n, dtype=torch.bfloat16, device="cuda"), torch.empty(4, n, device="cuda")
    words = torch.zeros(1, dtype=torch.int32, device="cuda")
    p, graph, stream = C.c_void_p, torch.cuda.CUDAGraph(keep_graph=True), torch.cuda.Stream()
    with torch.cuda.graph(graph, stream=stream):
        s, status = p(stream.cuda_stream), p(words.data_ptr())
        assert L.ingot_support_fetch(p(meta.data_ptr()), p(host.data_ptr()), C.c_size_t(16), s) == 0
        if table_kind == "two tables":
            rc = L.ingot_support_embed_sum_bf16(p(out.data_ptr()), None, p(table.data_ptr()), 8, p(meta.data_ptr()), p(table.data_ptr()), 8, p(meta.data_ptr()), n, 4,
                                                C.c_float(1), status, s)
        else:
            rc = L.ingot_support_embed_rows_bf16(p(out.data_ptr()), p(table.data_ptr()), n, 8, p(meta.data_ptr()), 4, C.c_float(1), status, s)
        assert rc == 0
    assert edge_types(graph.raw_cuda_graph()) == [0]
