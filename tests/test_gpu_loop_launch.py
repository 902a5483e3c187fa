"""The drop-in's float64 loop in one launch (small grids, eager) against one
launch per subcycle (as a captured graph replays it)."""
import pytest

from tests.test_gpu_small_grids import lib, prepared  # noqa: F401

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

OPTIONS = {"basalDragK2": 15.0, "useAdaptiveEVP": True, "noSlip": False}


# one CTA, two-row pieces, pieces of eight rows and the first of nine
@pytest.mark.parametrize("nx,ny", ((4, 4), (33, 35), (90, 40), (236, 124), (251, 133)))
@pytest.mark.parametrize("n,settings,plain", ((1, {}, False), (2, {}, True), (7, {}, False), (6, OPTIONS, False)))
def test_one_launch_matches_a_graph_of_subcycles(lib, nx, ny, n, settings, plain):  # noqa: F811
    from veris_gb300.state import Call
    st = prepared(nx, ny, nx + n, **settings)
    if plain:   # a state of the plain tile
        st.variables.k1AtC[3, 3] = 1e-7
    c = Call(st)
    g_, p_, _ = c.refs()
    ws, wsb = c.workspace(lib.veris_evp_auto_workspace_bytes(g_, p_))
    out = c.empty(5)

    def run(stream):
        assert lib.veris_evp_auto_solver_f64(*c.refs(), n, *[t.data_ptr() for t in out], ws, wsb, stream) == 0

    run(c.stream)
    torch.cuda.synchronize()
    eager = [t.clone() for t in out]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        run(torch.cuda.current_stream().cuda_stream)
    for _ in range(2):
        for t in out:
            t.fill_(-1.0)
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(out, eager))
