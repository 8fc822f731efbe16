"""Builds that do not find the memory of their fastest form: without the sorted copy of the base, then
without the tensor-core prune and the stored distances, the graph, the projection and the evaluation
count stay the same; once memory is free again the next build takes the fastest form."""
import ctypes

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

N, D, DEGREE, BEAM = 60_000, 200, 32, 64


@pytest.fixture(scope="module")
def pg():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import paragraph_gb300
    paragraph_gb300.lib()
    return paragraph_gb300


def _free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def _leave(nbytes):
    """Takes all device memory but nbytes."""
    torch.cuda.empty_cache()
    return torch.empty(_free() - nbytes, dtype=torch.uint8, device="cuda")


def _ids(*shape):
    return torch.full(shape, -1, dtype=torch.int32, device="cuda")


def _data():
    from paragraph_gb300 import datagen
    return datagen.make_dataset_cuda(N, D, N, seed=41)


def _bytes_per_point():
    """Every point's words in the lists of a build that stores no distances: the least it needs."""
    lists = 2 * DEGREE + 111 + BEAM + 16 + 32
    return 4 * (lists + DEGREE + 8)


# what is left free, in units of the smallest form: 1.1 leaves room for that only, 2.3 for the form on
# the caller's rows but not for the sorted copy
@pytest.mark.parametrize("graph_flag", [False, True])
@pytest.mark.parametrize("room", [1.1, 2.3])
def test_same_result_with_less_memory(pg, room, graph_flag):
    base, gt = _data()
    graph, proj = _ids(N, DEGREE), _ids(N, 16)
    params = pg.default_params(DEGREE, BEAM, screen=pg.SCREEN_FP16,
                               flags=pg.FLAG_CUDA_GRAPH if graph_flag else 0)
    small = N * _bytes_per_point()
    need = ctypes.c_uint64(0)
    assert pg.lib().pg_workspace_bytes(ctypes.byref(params), N, D, N, ctypes.byref(need)) == 0
    assert need.value > 1.1 * room * small  # the fastest form does not fit
    torch.cuda.synchronize()
    stream = torch.cuda.Stream()
    with pg.Handle(0, stream=stream) as h:
        want = h.build_device(base, gt, graph, proj, params).evals_total
        want_graph, want_proj = graph.clone(), proj.clone()
    with pg.Handle(0, stream=stream) as h:
        for screen in (pg.SCREEN_NONE, pg.SCREEN_FP16):  # kernels loaded while there is room
            few = pg.default_params(DEGREE, BEAM, screen=screen, flags=params.flags)
            h.build_device(base[:2000].contiguous(), gt[:2000] % 2000, _ids(2000, DEGREE),
                           _ids(2000, 16), few)
        taken = _leave(int(room * small))
        for _ in range(2):
            graph.fill_(-1)
            proj.fill_(-1)
            torch.cuda.synchronize()
            st = h.build_device(base, gt, graph, proj, params)
            assert st.evals_total == want
            assert torch.equal(graph, want_graph) and torch.equal(proj, want_proj)
        del taken
        torch.cuda.empty_cache()
        graph.fill_(-1)
        torch.cuda.synchronize()
        assert h.build_device(base, gt, graph, proj, params).evals_total == want
        assert torch.equal(graph, want_graph)
        before = _free()
        h.close()
        # memory free again: the last build took the workspace of the fastest form (up to the
        # projection's place, which was the caller's here)
        assert _free() - before >= need.value - N * 16 * 4


def test_workspace_makes_room_for_host_inputs(pg):
    """A handle that holds a build's workspace and then needs the inputs' device copies."""
    base, gt = _data()
    graph, proj = _ids(N, DEGREE), _ids(N, 16)
    params = pg.default_params(DEGREE, BEAM, screen=pg.SCREEN_FP16)
    hb, hg = base.cpu().numpy(), gt.cpu().numpy()
    with pg.Handle(0, stream=0) as h:
        torch.cuda.synchronize()
        h.build_device(base, gt, graph, proj, params)
        h.build_host(hb[:2000], hg[:2000] % 2000, params)
        want, want_proj = graph.cpu().numpy().view("uint32"), proj.cpu().numpy().view("uint32")
        # less than the inputs and outputs of the host call; with the workspace given back, enough
        # for them and the smallest form
        taken = _leave(N * (D + 128) * 4 // 2)
        got, got_proj, _ = h.build_host(hb, hg, params)
        del taken
        torch.cuda.empty_cache()
    assert (got == want).all() and (got_proj == want_proj).all()
