"""The graph of a stand-alone solve request keeps the kernels that it was built
with, so the context's flag that picks them (EcsCtx::mom_quanta: the moments are
a mixed deposit's) has to be cleared before the graph is built.  A context that
had deposited ions before its first request kept the kernels for whole quanta,
slower on a density that is not.  The values are the same, so the order is read
from the source."""
from ecsprt_gb300 import build as b


def test_flag_is_cleared_before_the_request_graph_is_built():
    text = (b.CSRC / "ecs_solver.cu").read_text()
    start = text.index("int ecs_request_launch(")
    body = text[start:text.index("\n}\n", start)]
    assert body.index("mom_quanta = false") < body.index("build_request_graph<")
