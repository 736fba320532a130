"""ecs_rhs_noalloc forms the mean in the block of its first kernel that finishes
last, by a completion count that outlives the call.

A call whose second kernel never runs (its launch can fail) must leave the
count at 0: otherwise no block of the next call is the last one, and a mean of
an earlier call is subtracted.  The first kernel is made to run alone through a
captured call whose last node is taken out of the graph.
"""
import ctypes

import numpy as np
import pytest

import ecsprt_gb300 as E
from ecsprt_gb300 import _lib
from oracle import oracle as orc
from test_zz_no_alloc import _cudart, _rel_inf, _rhs_noalloc

pytestmark = pytest.mark.gpu


def _first_kernel_alone(rt, p, moments):
    """Captures a call, drops its tail node (the mean's subtraction) and launches the rest."""
    m = np.ascontiguousarray(moments, dtype=np.float64)
    dm, db, stream, graph, gexec = (ctypes.c_void_p() for _ in range(5))
    assert rt.cudaMalloc(ctypes.byref(dm), ctypes.c_size_t(m.nbytes)) == 0
    assert rt.cudaMalloc(ctypes.byref(db), ctypes.c_size_t(m.nbytes // 4)) == 0
    assert rt.cudaMemcpy(dm, m.ctypes.data_as(ctypes.c_void_p), ctypes.c_size_t(m.nbytes), 1) == 0
    assert rt.cudaStreamCreateWithFlags(ctypes.byref(stream), 1) == 0
    assert rt.cudaStreamBeginCapture(stream, 1) == 0
    assert _lib.gpu().ecs_rhs_noalloc(ctypes.byref(p), dm, db, stream) == 0
    assert rt.cudaStreamEndCapture(stream, ctypes.byref(graph)) == 0
    count = ctypes.c_size_t(8)
    nodes = (ctypes.c_void_p * 8)()
    assert rt.cudaGraphGetNodes(graph, nodes, ctypes.byref(count)) == 0
    assert count.value == 2
    heads = ctypes.c_size_t(8)
    head = (ctypes.c_void_p * 8)()
    assert rt.cudaGraphGetRootNodes(graph, head, ctypes.byref(heads)) == 0
    assert heads.value == 1
    tail = [n for n in nodes[:2] if n != head[0]]
    assert rt.cudaGraphDestroyNode(ctypes.c_void_p(tail[0])) == 0
    assert rt.cudaGraphInstantiate(ctypes.byref(gexec), graph, ctypes.c_ulonglong(0)) == 0
    assert rt.cudaGraphLaunch(gexec, stream) == 0
    assert rt.cudaStreamSynchronize(stream) == 0
    rt.cudaGraphExecDestroy(gexec)
    rt.cudaGraphDestroy(graph)
    rt.cudaStreamDestroy(stream)
    rt.cudaFree(dm)
    rt.cudaFree(db)


@pytest.mark.parametrize("grid", [(5, 4, 6), (33, 31, 29)], ids=str)  # one block, and many
def test_call_after_a_failed_second_launch(built, grid):
    nx, ny, nz = grid
    p = E.params_from_options(f"-Nx {nx} -Ny {ny} -Nz {nz} -dx 1 -dy 1 -dz 1 -qi 1 -mi 1 -B0 0.1 -viT 1 -nue 8.79e9 "
                              "-Te 11604.5 -E0 0.3 -zBC inject-reflect")
    rng = np.random.default_rng(11)
    m = rng.standard_normal((nz, ny, nx, 4))  # ghosts beyond the walls: the mean is far from 0
    m[..., 0] += 16.0
    rt = _cudart()
    want = orc.Oracle(p).rhs(m)
    other = m.copy()
    other[..., 0] *= 3.0
    assert _rel_inf(_rhs_noalloc(rt, p, other), orc.Oracle(p).rhs(other)) <= 1e-14
    _first_kernel_alone(rt, p, other)
    assert _rel_inf(_rhs_noalloc(rt, p, m), want) <= 1e-14
