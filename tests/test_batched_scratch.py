"""The batched path's fp32 rows: a block that a captured graph may hold is never given back while its container lives."""
import numpy as np
import pytest

import lutgemm_b200 as L
from lutgemm_b200 import synth
from oracle import oracle

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

# several k-ranges for 16, 128 and 256 rows, so that each of these calls reduces into the rows
N, K, Q, G = 1024, 4096, 4, 128


def _container():
    bW, alpha, _ = synth.bcq_layer(N, K, Q, G, seed=11)
    return L.nQWeight_fp16(bW, alpha, K, N, Q, False, K // G), bW, alpha.astype(np.float16)


def _device(x):
    return torch.from_numpy(x.view(np.int16)).cuda().view(torch.float16)


def _close(y, x, bW, alpha):
    ref = oracle.bcq_matmul_f64(x, bW, alpha, None, G)
    assert np.linalg.norm(y - ref) <= 8e-4 * np.linalg.norm(ref)      # the rounding to fp16, as in perf/cases.py


def _capture(w, x, m):
    """The graph of one call, its output and its input (which has to live as long as the graph)."""
    xd = _device(x)
    y = torch.zeros((m, N), dtype=torch.float16, device="cuda")
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        L.matmul(y, xd, w, m)
    return graph, y, xd


def _eager(w, bW, alpha, m, seed):
    x = synth.activations(m, K, seed=seed)
    y = torch.empty((m, N), dtype=torch.float16, device="cuda")
    L.matmul(y, _device(x), w, m)
    _close(y.cpu().numpy(), x, bW, alpha)


@pytest.mark.parametrize("m", [16, 128])
def test_a_larger_call_leaves_the_rows_of_a_captured_one(m):
    w, bW, alpha = _container()
    w.reserve_batch(128)
    before = w.scratch()
    x = synth.activations(m, K, seed=m)
    graph, y, xd = _capture(w, x, m)
    for rows in (256, 300):
        _eager(w, bW, alpha, rows, rows)
        assert w.scratch() == before
        y.zero_()
        graph.replay()
        torch.cuda.synchronize()
        _close(y.cpu().numpy(), x, bW, alpha)
    del graph
    w.close()


def test_growth_keeps_the_earlier_rows():
    """Calls on a container that nothing was reserved for, and a later reservation: more rows, the earlier ones kept."""
    w, bW, alpha = _container()
    assert w.scratch() == (0, 0, 0)
    graphs, blocks = [], set()
    for m in (16, 40, 128):
        _eager(w, bW, alpha, m, m)
        x = synth.activations(m, K, seed=m + 1)
        graphs.append((*_capture(w, x, m), x))
        blocks.add(w.scratch()[:2])
    w.reserve_batch(1024)
    address, size, kept = w.scratch()
    assert size >= max(b for _, b in blocks) and kept <= size
    assert kept == sum(b for a, b in blocks if a != address)
    assert len({a for a, _ in blocks}) >= 2               # the sizes above do make it grow
    _eager(w, bW, alpha, 512, 7)
    for graph, y, xd, x in graphs:
        y.zero_()
        graph.replay()
        torch.cuda.synchronize()
        _close(y.cpu().numpy(), x, bW, alpha)
    del graphs, graph
    w.close()


def test_host_call_replays_after_larger_calls_and_reservations():
    """matmul_host keeps the last call as a graph: it stays right when other calls and reservations come between."""
    w, bW, alpha = _container()
    x = synth.activations(128, K, seed=3)
    out = np.empty((128, N), np.float16)                  # the same buffers each time: the recorded graph is what runs
    _close(L.matmul_host(out, x, w, 128), x, bW, alpha)
    before = w.scratch()
    _eager(w, bW, alpha, 256, 5)
    assert w.scratch() == before
    out.fill(0)
    _close(L.matmul_host(out, x, w, 128), x, bW, alpha)
    w.reserve_batch(512)
    assert w.scratch()[2] == before[1]
    out.fill(0)
    _close(L.matmul_host(out, x, w, 128), x, bW, alpha)
    w.close()


def test_rising_batches_do_not_allocate_once_128_rows_are_there():
    w, bW, alpha = _container()
    _eager(w, bW, alpha, 128, 1)
    before = w.scratch()
    for m in (129, 300, 301, 1100):
        _eager(w, bW, alpha, m, m)
        assert w.scratch() == before
    w.close()


@pytest.mark.parametrize("m", [16, 130, 256, 512])
@pytest.mark.parametrize("max_n", [N, 5 * N])
def test_explicit_workspace_runs_the_plan_of_the_containers_own(m, max_n):
    """A workspace of the same batch has the rows for the same k-ranges, for its own width and for narrower containers."""
    w, bW, alpha = _container()
    w.reserve_batch(m)
    x = synth.activations(m, K, seed=m)
    y = torch.empty((m, N), dtype=torch.float16, device="cuda")
    L.matmul(y, _device(x), w, m)
    own = L.last_launch()
    assert own[2] > 1                                     # k-ranges: the shape is one that needs the rows
    ws = L.Workspace(max_n, K, m)
    for _ in range(2):                                    # the second call finds the workspace as the first one left it
        y.zero_()
        L.matmul(y, _device(x), w, m, workspace=ws)
        assert L.last_launch() == own
        _close(y.cpu().numpy(), x, bW, alpha)
    assert ws.status() == 0
    ws.close()
    w.close()


@pytest.mark.parametrize("q,m", [(1, 256), (2, 130), (4, 300), (4, 129), (1, 513)])
def test_captured_call_above_the_reserved_rows(q, m):
    """Fewer rows than the call's: some rows at a time or no k-ranges, the outputs the same, and nothing allocated."""
    bW, alpha, _ = synth.bcq_layer(N, K, q, G, seed=q)
    w = L.nQWeight_fp16(bW, alpha, K, N, q, False, K // G).reserve_batch(128)
    before = w.scratch()
    x = synth.activations(m, K, seed=m)
    graph, y, xd = _capture(w, x, m)
    for _ in range(2):
        y.zero_()
        graph.replay()
        torch.cuda.synchronize()
        _close(y.cpu().numpy(), x, bW, alpha.astype(np.float16))
    assert w.scratch() == before
    del graph
    w.close()


@pytest.mark.parametrize("n,k,q,rows", [(24576, 512, 1, 128), (24576, 512, 4, 128), (1000, 1024, 5, 128), (1004, 1024, 3, 128),
                                        (8192, 8192, 4, 512)])
def test_reserved_rows_are_bounded_by_what_a_plan_can_ask_for(n, k, q, rows):
    """Wide outputs never split beyond 128 rows, five planes and containers without a tensor-core kernel neither."""
    bW, alpha, _ = synth.bcq_layer(n, k, q, 128, seed=q)
    w = L.nQWeight_fp16(bW, alpha, k, n, q, False, k // 128).reserve_batch(2048)
    assert w.scratch()[1] <= rows * n * 4
    w.close()


@pytest.mark.parametrize("q", [1, 3])
def test_reserved_rows_are_enough_for_every_plan(q):
    """Every batch up to the reserved one runs the plan that it has with far more rows than any call can use."""
    n, k = 2048, 2048
    bW, alpha, _ = synth.bcq_layer(n, k, q, 128, seed=q)
    w = L.nQWeight_fp16(bW, alpha, k, n, q, False, k // 128).reserve_batch(2048)
    plenty = L.Workspace(64 * n, k, 2048)
    x = _device(synth.activations(2048, k, seed=1))
    y = torch.empty((2048, n), dtype=torch.float16, device="cuda")
    split = 0
    for m in [*range(100, 700, 37), 256, 512, 768, 1024, 1500, 2048]:
        L.matmul(y, x, w, m, workspace=plenty)
        free = L.last_launch()
        L.matmul(y, x, w, m)
        assert L.last_launch() == free, m
        split += m > 128 and free[2] > 1
    assert split > 0
    plenty.close()
    w.close()


def test_captured_wx_call_outlives_a_larger_one():
    """The transposed copies of the (output, nqW, input, n) form: a larger call leaves those of a captured one in place."""
    w, bW, alpha = _container()
    w.reserve_batch(5)
    x = synth.activations(5, K, seed=5)
    xd = _device(np.ascontiguousarray(x.T))
    y = torch.zeros((N, 5), dtype=torch.float16, device="cuda")
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        L.matmul_wx(y, w, xd, 5)
    for n in (6, 40):
        xl = synth.activations(n, K, seed=n)
        yl = torch.empty((N, n), dtype=torch.float16, device="cuda")
        L.matmul_wx(yl, w, _device(np.ascontiguousarray(xl.T)), n)
        _close(yl.cpu().numpy().T, xl, bW, alpha)
        w.reserve_batch(2 * n)
        y.zero_()
        graph.replay()
        torch.cuda.synchronize()
        _close(y.cpu().numpy().T, x, bW, alpha)
    del graph
    w.close()
