"""The device grammar compressor against the host compressor of this package: the two must return the
same arrays (the reference's tests/test_batch_compression.py:36-48 asks exactly that of its CPU and
CUDA back ends), and every vertex row must expand to its input row in order."""
import numpy as np
import pytest
import torch

from compressgnn_b200 import offline as off
from compressgnn_b200.loader import CompressgnnData, compress_graph_csr, resolve_backend

pytestmark = pytest.mark.gpu


def expand(v, e, node, n):
    stack = list(reversed(e[v[node]:v[node + 1]].tolist()))
    out = []
    while stack:
        child = stack.pop()
        if child < n:
            out.append(child)
        else:
            children = e[v[child]:v[child + 1]]
            assert np.all(children < child)
            stack.extend(reversed(children.tolist()))
    return out


def csr_of(rows):
    v = np.array([0] + list(np.cumsum([len(x) for x in rows])), dtype=np.int64)
    e = np.array([j for row in rows for j in row], dtype=np.int64)
    return v, e


def same(a, b):
    assert a[0].dtype == np.int32 and a[1].dtype == np.int32
    assert a[2] == b[2] and a[3] == b[3]
    np.testing.assert_array_equal(a[0], b[0])
    np.testing.assert_array_equal(a[1], b[1])


def test_backend_resolution_on_a_gpu():
    assert resolve_backend('auto') == 'cuda' and resolve_backend('cuda') == 'cuda' and resolve_backend('cpu') == 'cpu'


def test_fixtures_of_the_reference_test():
    rng = np.random.default_rng(17)
    fixtures = [[], [[]], [[0] * 50], [list(range(32)) for _ in range(64)]]
    fixtures += [[rng.integers(32, size=20).tolist() for _ in range(32)] for _ in range(4)]
    fixtures += [[[] for _ in range(5)], [[i] for i in range(7)], [[0, 1], [], [0, 1], [0, 1], [], [0, 1, 0, 1, 0, 1]]]
    for rows in fixtures:
        v, e = csr_of(rows)
        for frequency in [3, 16, 256]:
            host = compress_graph_csr(v, e, frequency, backend='cpu')
            device = compress_graph_csr(v, e, frequency, backend='cuda')
            same(device, host)
            dv, de, n, _ = device
            for node, row in enumerate(rows):
                assert expand(dv, de, node, n) == row


@pytest.mark.parametrize("rounds", [1, 2, 12])
@pytest.mark.parametrize("frequency", [3, 4, 16])
def test_web_graph_rows(rounds, frequency):
    """Rows with long shared runs and a few hubs (the copying-model generator of the benchmark), so that
    several rounds nest rules inside rules and the parse meets overlapping candidates."""
    v, e = off.generate_copy_graph(6000, alpha=2.1, x_min=5.3, max_degree=2000, copy_prob=0.7, window=64,
                                   candidates=8, seed=rounds + frequency)
    v, e = off.add_self_loop_csr(v, e)
    host = compress_graph_csr(v, e, frequency, backend='cpu', rounds=rounds)
    device = compress_graph_csr(v, e, frequency, backend='cuda', rounds=rounds)
    same(device, host)
    assert host[3] > 0
    dv, de, n, _ = device
    for node in range(0, n, 97):
        assert expand(dv, de, node, n) == e[v[node]:v[node + 1]].tolist()


def test_runs_of_the_left_to_right_step():
    """Rows of one repeated symbol (every pair weighs the same, the whole row is one run), of two in turn, runs begun
    behind a pair the first step took, and lengths around them, against the host's row-by-row walk."""
    rng = np.random.default_rng(2)
    rows = [[1] * k for k in range(1, 45)] + [[2, 3] * k for k in range(1, 20)] + [[4] * 3000]
    rows += [[7, 8] * 2 + [1] * k + [7, 8] for k in range(12)]
    rows += [rng.integers(0, 3, rng.integers(0, 40)).tolist() for _ in range(400)]
    v, e = csr_of(rows)
    for frequency in (3, 5, 40):
        same(compress_graph_csr(v, e, frequency, backend='cuda'), compress_graph_csr(v, e, frequency, backend='cpu'))


def test_with_and_without_a_workspace():
    """The entry point that allocates for itself and the one that is given a workspace."""
    import ctypes
    from compressgnn_b200 import runtime as rt
    from compressgnn_b200._lib import check, lib
    v, e = off.generate_copy_graph(2000, alpha=2.1, x_min=5.3, max_degree=500, copy_prob=0.7, window=64, candidates=8, seed=1)
    dv, de = torch.from_numpy(v).cuda(), torch.from_numpy(e).cuda()
    want = rt.compress_csr_batch(dv, de, 12, 4)
    handle, info = ctypes.c_void_p(0), (ctypes.c_int64 * 3)()
    check(lib().cgnn_compress_csr_batch(dv.data_ptr(), de.data_ptr(), v.size - 1, 12, 4, ctypes.byref(handle), 0))
    check(lib().cgnn_compressed_info(handle, info))
    assert list(info) == [want[2], want[3], want[1].numel()]
    got = torch.empty_like(want[0]), torch.empty_like(want[1])
    check(lib().cgnn_compressed_copy(handle, got[0].data_ptr(), got[1].data_ptr(), 0))
    torch.cuda.synchronize()
    lib().cgnn_compressed_destroy(handle)
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    room = lib().cgnn_compress_workspace_bytes(v.size - 1, e.size, 4)
    small = torch.empty(room, dtype=torch.uint8, device="cuda")
    with pytest.raises(RuntimeError, match="workspace"):
        check(lib().cgnn_compress_csr_batch_in(dv.data_ptr(), de.data_ptr(), v.size - 1, 12, 4, small.data_ptr(), room - 256,
                                               ctypes.byref(handle), 0))


def test_a_large_workspace_goes_back_to_the_driver(monkeypatch):
    """Beyond the bound nothing of the work stays in torch's cache, and the arrays are the same."""
    from compressgnn_b200 import runtime as rt
    v, e = off.generate_copy_graph(20000, alpha=2.1, x_min=5.3, max_degree=500, copy_prob=0.7, window=64, candidates=8, seed=1)
    dv, de = torch.from_numpy(v).cuda(), torch.from_numpy(e).cuda()
    room = rt.lib().cgnn_compress_workspace_bytes(v.size - 1, e.size, 4)
    want = rt.compress_csr_batch(dv, de, 12, 4)
    torch.cuda.empty_cache()
    monkeypatch.setattr(rt, "KEPT_WORKSPACE", room - 1)
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.max_memory_reserved()
    got = rt.compress_csr_batch(dv, de, 12, 4)
    assert torch.cuda.max_memory_reserved() - before < room // 2  # the result only
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1]) and got[2:] == want[2:]


def test_row_pointers_beyond_the_edges_are_refused():
    """Nothing is read behind the edge array, by however little the last row pointer passes its end."""
    from compressgnn_b200 import runtime as rt
    for beyond in (1, 2, 300):
        vlist, elist = np.array([0, 2, 2 + beyond], np.int64), np.array([0, 1], np.int64)
        with pytest.raises(RuntimeError, match="row pointers"):
            compress_graph_csr(vlist, elist, 3, backend='cuda')
        with pytest.raises(RuntimeError, match="row pointers"):
            rt.compress_csr_batch(torch.from_numpy(vlist).cuda(), torch.from_numpy(elist).cuda())
    with pytest.raises(RuntimeError, match="row pointers"):
        rt.compress_csr_batch(torch.tensor([0, 1], device="cuda"), torch.empty(0, dtype=torch.int64, device="cuda"))


def test_argument_errors():
    v, e = csr_of([[0, 1], [1, 5]])
    with pytest.raises(RuntimeError):
        compress_graph_csr(v, e, 3, backend='cuda')          # a value outside [0, n)
    with pytest.raises(ValueError):
        compress_graph_csr(*csr_of([[0]]), 2, backend='cuda')
    with pytest.raises(ValueError):
        compress_graph_csr(np.array([0, 1], np.int64), np.array([2**32], np.uint64), backend='cuda')
    with pytest.raises(ValueError):
        compress_graph_csr(np.array([0, 1]), np.array([0.5]), backend='cuda')
    from compressgnn_b200 import runtime as rt
    with pytest.raises(RuntimeError):
        rt.compress_csr_batch(torch.tensor([0, 2, 1], device="cuda"), torch.tensor([0, 0], device="cuda"))


def test_loader_builds_the_same_graph_with_either_back_end():
    n = 64
    v = np.arange(n + 1, dtype=np.int32) * 32
    e = np.tile(np.arange(32, dtype=np.int32), n)
    coo = np.vstack([np.repeat(np.arange(n, dtype=np.int32), 32), e])
    x = np.random.default_rng(3).standard_normal((n, 8)).astype(np.float32)
    mask = np.ones(n, dtype=bool)
    for graph_type, edge in [('coo', coo), ('csr', (v, e))]:
        for normalize in [False, True]:
            pieces = {}
            for backend in ['cpu', 'cuda']:
                data = CompressgnnData(x, edge, np.zeros(n, np.int64), mask, mask, mask, add_self_loop=False,
                                       normalize=normalize, graph_type=graph_type, compression_backend=backend)
                assert data.compression_backend == backend
                if graph_type == 'coo':
                    pieces[backend] = list(data.edge_index) + list(data.edge_weight)
                else:
                    g = data.edge_index
                    pieces[backend] = [part for blk in g.blocks() for part in blk.csr()]
            assert len(pieces['cpu']) == len(pieces['cuda'])
            assert all(torch.equal(a, b) for a, b in zip(pieces['cpu'], pieces['cuda']))


@pytest.mark.parametrize("dtype", [torch.int64, torch.int32])
def test_staged_copies(dtype, monkeypatch):
    """Arrays of less than a stage, whole stages, one element more or less, and enough parts to use each stage again; then
    from several threads at once, each with a stream of its own."""
    from concurrent.futures import ThreadPoolExecutor
    from compressgnn_b200.loader import compression_backend as backend
    monkeypatch.setattr(backend, "STAGE_BYTES", 1 << 16)
    step = (1 << 16) // torch.empty((), dtype=dtype).element_size()

    def both_ways(size):
        host = torch.randint(-2**31, 2**31 - 1, (size,), dtype=dtype)
        with torch.cuda.stream(torch.cuda.Stream()):
            there = backend._to_device(host)
            back = backend._to_host(there)
        return there.is_cuda and torch.equal(back, host)

    sizes = [0, 1, step - 1, step, step + 1, 2 * step, 2 * step + 1, 7 * step - 1, 8 * step]
    assert all(both_ways(size) for size in sizes)
    with ThreadPoolExecutor(4) as pool:
        assert all(pool.map(both_ways, sizes * 4))


def test_staged_copies_with_a_default_device(monkeypatch):
    """The stages and the result lie in host memory whatever torch's default device is."""
    from compressgnn_b200.loader import compression_backend as backend
    vlist = np.arange(0, 40001, 4)
    elist = np.random.default_rng(3).integers(0, 1000, 40000)
    want = backend.compress_graph_csr(vlist, elist, 4, backend="cuda")
    monkeypatch.setattr(backend, "STAGE_BYTES", 1 << 14)
    with torch.device("cuda"):
        got = backend.compress_graph_csr(vlist, elist, 4, backend="cuda")
    assert got[2:] == want[2:] and all(np.array_equal(g, w) for g, w in zip(got[:2], want[:2]))


def test_copies_without_page_locked_memory(monkeypatch):
    """Where the system has no page-locked memory to give, the arrays are copied without stages."""
    from compressgnn_b200.loader import compression_backend as backend
    vlist = np.arange(0, 40001, 4)
    elist = np.random.default_rng(4).integers(0, 1000, 40000)
    want = backend.compress_graph_csr(vlist, elist, 4, backend="cuda")
    empty = torch.empty

    def refuses(*args, **kwargs):
        if kwargs.get("pin_memory"):
            raise RuntimeError("CUDA error: out of memory")
        return empty(*args, **kwargs)

    monkeypatch.setattr(backend, "STAGE_BYTES", 1 << 14)
    monkeypatch.setattr(torch, "empty", refuses)
    got = backend.compress_graph_csr(vlist, elist, 4, backend="cuda")
    assert got[2:] == want[2:] and all(np.array_equal(g, w) for g, w in zip(got[:2], want[:2]))
