"""Parity of the CUDA cluster / reconstruct operators (through the C ABI) with the CPU
oracle, the golden vectors, and the closed-form expectations of the reference's
tests/test_transformation.py (same grids of widths, sizes and bit counts)."""
import numpy as np
import pytest
import torch

from conftest import assert_close_rel
from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def rt():
    from compressgnn_b200 import runtime
    return runtime


def cu(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def assign(rt, x, w, bits):
    return rt.cluster_assign(x, w, bits, rt.cluster_workspace(x, bits))


@pytest.mark.parametrize("tag", ["a", "b", "c", "f"])
def test_golden_lsh_ids_are_bit_exact(rt, golden, tag):
    x, w = cu(golden[f"lsh_{tag}_x"]), cu(golden[f"lsh_{tag}_planes"])
    ids, counts, active = assign(rt, x, w, w.size(1))
    assert active == int(golden[f"lsh_{tag}_active"])
    assert ids.dtype == torch.int64 and counts.dtype == torch.int32
    np.testing.assert_array_equal(ids.cpu().numpy(), golden[f"lsh_{tag}_ids"].astype(np.int64))
    np.testing.assert_array_equal(counts.cpu().numpy(),
                                  np.bincount(golden[f"lsh_{tag}_ids"], minlength=active + 1))
    legacy_ids, legacy_active = rt.cluster_forward(x, w, w.size(1))
    assert legacy_ids.dtype == torch.int32 and legacy_active == active
    np.testing.assert_array_equal(legacy_ids.cpu().numpy(), golden[f"lsh_{tag}_ids"])


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("width", [0, 1, 31, 33, 128, 602])
@pytest.mark.parametrize("n,bits", [(0, 8), (1, 0), (67, 8), (257, 16), (1500, 24)])
def test_assign_mean_grid_is_bit_exact_against_the_oracle(rt, dtype, width, n, bits):
    """Grid of reference tests/test_transformation.py:21-29; N(0,1) inputs, so the ids depend
    on the documented fma order, which the oracle restates exactly."""
    rng = np.random.default_rng(1000 * width + n + bits)
    x = rng.standard_normal((n, width)).astype(dtype)
    w = rng.standard_normal((width, bits)).astype(dtype)
    ids, counts, active = assign(rt, cu(x), cu(w), bits)
    rids, rcounts, ractive = oracle.cluster_assign(x, w)
    assert active == ractive
    np.testing.assert_array_equal(ids.cpu().numpy(), rids)
    np.testing.assert_array_equal(counts.cpu().numpy(), rcounts)
    y = rt.cluster_mean(cu(x), ids, counts)
    assert y.shape == (active + 1, width)
    assert_close_rel(y.cpu().numpy(), oracle.cluster_mean(x, rids, rcounts), what="mean")
    grad = rng.standard_normal((active + 1, width)).astype(dtype)
    dx = rt.cluster_mean_backward(cu(grad), ids, counts)
    assert_close_rel(dx.cpu().numpy(), oracle.cluster_mean_backward(grad, rids, rcounts),
                     rel=1e-6, what="mean backward")


def test_projection_matches_the_oracle_bit_for_bit(rt):
    rng = np.random.default_rng(77)
    for n, width, bits in [(1000, 128, 16), (333, 130, 7), (129, 96, 30), (64, 5, 1)]:
        x = rng.standard_normal((n, width)).astype(np.float32)
        w = rng.standard_normal((width, bits)).astype(np.float32)
        got = rt.project(cu(x), cu(w)).cpu().numpy()
        np.testing.assert_array_equal(got, oracle.project(x, w))
        ids, counts, active = rt.cluster_assign_from_projection(cu(got), rt.cluster_workspace(cu(x), bits))
        rids, rcounts, ractive = oracle.cluster_assign(x, w)
        assert active == ractive
        np.testing.assert_array_equal(ids.cpu().numpy(), rids)


@pytest.mark.parametrize("bits", [4, 8, 12, 16, 20, 24, 28])
@pytest.mark.parametrize("width", [16, 48, 128, 256])
def test_tile_copy_projection_is_bit_exact(rt, bits, width):
    """fp32, a width that is a multiple of 16 and a multiple of four planes take the kernel whose row
    tiles arrive by TMA: every tile-boundary case against the oracle, and against the cp.async kernel
    (reached through a feature matrix that starts 4 bytes off a 16-byte boundary)."""
    rng = np.random.default_rng(31 * bits + width)
    w = rng.standard_normal((width, bits)).astype(np.float32)
    for n in (1, 255, 512, 513, 1024 + 77, 5000):
        x = rng.standard_normal((n, width)).astype(np.float32)
        want = oracle.project(x, w)
        got = rt.project(cu(x), cu(w))
        np.testing.assert_array_equal(got.cpu().numpy(), want)
        ids, counts, active = assign(rt, cu(x), cu(w), bits)
        rids, rcounts, ractive = oracle.cluster_assign(x, w)
        assert active == ractive
        np.testing.assert_array_equal(ids.cpu().numpy(), rids)
        np.testing.assert_array_equal(counts.cpu().numpy(), rcounts)
        shifted = torch.empty(n * width + 1, dtype=torch.float32, device="cuda")[1:].view(n, width)
        shifted.copy_(cu(x))
        assert shifted.data_ptr() % 16 == 4
        assert torch.equal(rt.project(shifted, cu(w)), got)
    rt.raise_on_device_status()


def test_non_default_stream(rt):
    x = torch.randn(67, 33, device="cuda")
    w = torch.randn(33, 8, device="cuda")
    ids, counts, active = assign(rt, x, w, 8)
    ref = rt.cluster_mean(x, ids, counts)
    stream = torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        ii, cc, aa = assign(rt, x, w, 8)
        yy = rt.cluster_mean(x, ii, cc)
    stream.synchronize()
    assert aa == active and torch.equal(ii, ids) and torch.equal(yy, ref)


@pytest.mark.parametrize("bits", [0, 8, 24])
def test_all_rows_collide(rt, bits):
    x = torch.ones(513, 33, device="cuda")
    w = torch.ones(33, bits, device="cuda")
    ids, counts, active = assign(rt, x, w, bits)
    assert active == 1 and counts.tolist() == [0, 513] and bool((ids == 1).all())


def test_large_mean_is_deterministic_with_long_segments(rt):
    """Config-3 shape in small: Gaussian mixture, buckets collapse, segments far longer than
    the plan's split."""
    rng = np.random.default_rng(4)
    n, width, bits = 60000, 128, 16
    cent = rng.standard_normal((64, width)).astype(np.float32)
    x = (cent[rng.integers(0, 64, n)] + 0.1 * rng.standard_normal((n, width))).astype(np.float32)
    w = rng.standard_normal((width, bits)).astype(np.float32)
    dx = cu(x)
    ids, counts, active = assign(rt, dx, cu(w), bits)
    rids, rcounts, ractive = oracle.cluster_assign(x, w)
    assert active == ractive
    np.testing.assert_array_equal(ids.cpu().numpy(), rids)
    plan = rt.index_plan(ids, active + 1)
    assert plan.long_rows > 0
    reps = rng.standard_normal((active + 1, 64)).astype(np.float32)
    bias = rng.standard_normal(64).astype(np.float32)
    fwd = rt.cluster_reconstruct(cu(reps), ids, cu(bias), True)
    go = cu(rng.standard_normal((n, 64)).astype(np.float32))
    exact = rt.cluster_reconstruct_backward(go, ids, fwd, active + 1, True)
    fast = rt.cluster_reconstruct_backward(go, ids, fwd, active + 1, True, output_is_forward_result=True)
    assert torch.equal(exact, fast)
    assert_close_rel(exact.cpu().numpy(),
                     oracle.reconstruct_backward(go.cpu().numpy(), rids, fwd.cpu().numpy(), active + 1, True)[0],
                     what="long reconstruct backward")
    y1 = rt.cluster_mean(dx, ids, counts)
    y2 = rt.cluster_mean(dx, ids, counts)
    assert torch.equal(y1, y2)
    assert_close_rel(y1.cpu().numpy(), oracle.cluster_mean(x, rids, rcounts), what="long mean")
    # an index tensor the library has never seen: the plan is rebuilt from the index alone
    fresh = ids.clone()
    y3 = rt.cluster_mean(dx, fresh, counts)
    assert torch.equal(y1, y3)


def test_golden_mean_and_reconstruct(rt, golden):
    g = golden
    idx, cnt = cu(g["mean_index"]), cu(g["mean_counts"])
    assert_close_rel(rt.cluster_mean(cu(g["mean_x"]), idx, cnt).cpu().numpy(), g["mean_out"],
                     what="golden mean")
    assert_close_rel(rt.cluster_mean_backward(cu(g["mean_grad_out"]), idx, cnt).cpu().numpy(),
                     g["mean_grad_in"], rel=1e-6, what="golden mean backward")
    for tag, relu in (("lin", False), ("relu", True)):
        y = rt.cluster_reconstruct(cu(g["rec_reps"]), idx, cu(g["rec_bias"]), relu)
        np.testing.assert_array_equal(y.cpu().numpy(), g[f"rec_{tag}_out"])
        dr, db = rt.cluster_reconstruct_backward(cu(g["rec_grad_out"]), idx, y, cnt.numel(), relu,
                                                 return_bias_grad=True)
        assert_close_rel(dr.cpu().numpy(), g[f"rec_{tag}_dreps"], what="golden d_reps")
        assert_close_rel(db.cpu().numpy(), g[f"rec_{tag}_dbias"], what="golden d_bias")


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("width", [1, 31, 33, 128, 256, 520, 602])
@pytest.mark.parametrize("relu", [False, True])
def test_reconstruct_grid(rt, dtype, width, relu):
    """Grid of reference tests/test_transformation.py:44-54, including unused groups."""
    rng = np.random.default_rng(width)
    idx = np.array([1, 1, 3, 1, 3, 3] * 50, np.int64)
    reps = rng.standard_normal((5, width)).astype(dtype)
    bias = rng.standard_normal(width).astype(dtype)
    go = rng.standard_normal((idx.size, width)).astype(dtype)
    y = rt.cluster_reconstruct(cu(reps), cu(idx), cu(bias), relu)
    ref = oracle.reconstruct(reps, idx, bias, relu)
    np.testing.assert_array_equal(y.cpu().numpy(), ref)
    y_nobias = rt.cluster_reconstruct(cu(reps), cu(idx), None, relu)
    np.testing.assert_array_equal(y_nobias.cpu().numpy(), oracle.reconstruct(reps, idx, None, relu))
    dr, db = rt.cluster_reconstruct_backward(cu(go), cu(idx), y, 5, relu, return_bias_grad=True)
    rdr, rdb = oracle.reconstruct_backward(go, idx, ref, 5, relu)
    assert_close_rel(dr.cpu().numpy(), rdr, what="d_reps")
    assert_close_rel(db.cpu().numpy(), rdb, what="d_bias")
    assert not dr[0].any() and not dr[2].any() and not dr[4].any()
    # one mask row per group instead of the whole forward output: same bits
    dr2 = rt.cluster_reconstruct_backward(cu(go), cu(idx), y, 5, relu, output_is_forward_result=True)
    assert torch.equal(dr, dr2)


def test_argument_errors_raise_runtime_error(rt):
    x = torch.randn(10, 7, device="cuda")
    with pytest.raises(RuntimeError):  # bad plane shape (reference test :105-107)
        rt.cluster_assign(x, torch.randn(7, 3, device="cuda"), 4, rt.cluster_workspace(x, 4))
    with pytest.raises(RuntimeError):
        rt.cluster_workspace(x, 31)
    with pytest.raises(RuntimeError):  # workspace made for fewer rows
        small = rt.cluster_workspace(x[:2].contiguous(), 4)
        rt.cluster_assign(torch.randn(5000, 7, device="cuda"), torch.randn(7, 4, device="cuda"), 4, small)
    idx = torch.tensor([0, 1, 7], device="cuda")
    cnt = torch.tensor([1, 1], dtype=torch.int32, device="cuda")
    with pytest.raises(RuntimeError, match="outside"):  # index beyond the groups: reported, not trapped
        rt.cluster_mean(torch.randn(3, 4, device="cuda"), idx, cnt)
    out = rt.cluster_reconstruct(torch.randn(2, 4, device="cuda"), idx, None, False)
    assert rt.device_status() & 1 and not out[2].any()
    assert rt.device_status() == 0


@pytest.mark.parametrize("groups", [1, 7, 255, 256, 257, 2049, 70001])
def test_bias_gradient_sums(groups):
    """Column sums of the group gradients around the row blocks of the two stages, against 64 bits: a sum is a
    chain of at most 32 + 8 and then 35 + 8 additions here, each within half an ulp of the sum of magnitudes."""
    from compressgnn_b200 import runtime as rt
    gen = torch.Generator(device="cuda").manual_seed(groups)
    index = torch.arange(groups, device="cuda")
    for width in (1, 31, 33, 47, 128):
        grad = torch.randn(groups, width, device="cuda", generator=gen)
        d_reps, d_bias = rt.cluster_reconstruct_backward(grad, index, grad, groups, False, return_bias_grad=True)
        assert torch.equal(d_reps, grad)
        bound = 96 * 2.0 ** -24 * grad.double().abs().sum(0)
        assert bool(((d_bias.double() - grad.double().sum(0)).abs() <= bound).all())


@pytest.mark.parametrize("n, bits, shape", [
    (1, 4, "one"), (900, 4, "spread"), (1024, 16, "distinct"), (1500, 11, "spread"), (5000, 16, "distinct"),
    (70000, 1, "spread"), (70000, 16, "two giants"), (70000, 12, "power"), (300000, 16, "power"),
    (300000, 16, "two giants"), (1500000, 21, "distinct"), (1500000, 21, "power"), (9000, 0, "one")])
def test_bucket_plan_of_the_device_equals_the_host_one(rt, n, bits, shape):
    """An assignment's plan (statistics, lists and entries by kernels) against the plan the host cuts for the same
    index: figures, degrees and every bit of a mean (the summation order is the plan's), over one row, rows
    below, at and beyond a tile of rows, lengths beyond the histogram, and more than 2^20 buckets."""
    gen = torch.Generator(device="cuda").manual_seed(n + bits)
    if shape == "distinct":
        codes = torch.randperm(n, device="cuda", generator=gen)
    elif shape == "two giants":
        codes = torch.randint(0, 2 ** bits, (n,), device="cuda", generator=gen)
        codes[: n // 2] = 5
        codes[n // 2: n - 3000] = 2 ** bits - 1
    elif shape == "power":
        codes = (torch.rand(n, device="cuda", generator=gen) ** 6 * 2 ** bits).long()
    else:
        codes = torch.randint(0, 2 ** bits, (n,), device="cuda", generator=gen) * (shape != "one")
    codes = (codes % 2 ** bits).int()
    workspace = rt.cluster_workspace(torch.empty(n, 1, device="cuda"), bits)
    ids, counts, active = rt._assign_from_codes(codes, n, bits, workspace, codes.device)
    mine, host = rt.index_plan(ids, active + 1), rt.SegmentPlan.from_index(ids, active + 1)
    for name in ("rows", "nnz", "split", "long_rows", "chunks", "direct_units", "compact_rows", "source_rows",
                 "degree_p50", "degree_p99", "degree_max"):
        assert getattr(mine, name) == getattr(host, name), name
    x = torch.randn(n, 12, device="cuda", generator=gen)
    assert torch.equal(rt.cluster_mean(x, ids, counts, plan=mine), rt.cluster_mean(x, ids, counts, plan=host))


def test_bias_gradients_of_two_threads(rt):
    """Two threads, one plan, one stream: the column sums meet in the plan's scratch, each thread gets its own."""
    from concurrent.futures import ThreadPoolExecutor
    ids = torch.arange(9000, device="cuda") % 3000
    grads = [torch.randn(9000, 48, device="cuda") for _ in range(2)]

    def sums(which):
        return rt.cluster_reconstruct_backward(grads[which], ids, grads[which], 3000, False, return_bias_grad=True)[1]

    alone = [sums(which) for which in range(2)]
    with ThreadPoolExecutor(2) as pool:
        assert all(pool.map(lambda which: all(torch.equal(sums(which), alone[which]) for _ in range(200)), range(2)))


@pytest.mark.parametrize("width", [16, 47, 66, 128, 256])
def test_buckets_of_many_chunks(rt, width):
    """A bucket of several hundred chunks, one just above 32, one of 32 and many small ones: the mean (also from a captured
    graph), and the reconstruct backward without a mask, with a mask row per node and with one per bucket (the last two
    bit for bit alike), through a plan built on the device, against float64 sums; the bound is that of any order of a
    bucket's additions."""
    gen = torch.Generator(device="cuda").manual_seed(width)
    n, bits = 60000, 12
    codes = torch.randint(0, 2 ** bits, (n,), device="cuda", generator=gen).int()
    codes[: 48000] = 5
    codes[48000: 48000 + 32 * 64 + 1] = 9
    codes[51000: 51000 + 32 * 64 - 20] = 7
    workspace = rt.cluster_workspace(torch.empty(n, 1, device="cuda"), bits)
    ids, counts, active = rt._assign_from_codes(codes, n, bits, workspace, codes.device)
    groups = active + 1
    assert rt.index_plan(ids, groups).degree_max > 64 * 128
    eps = 0.5 * torch.finfo(torch.float32).eps * (1 + 1e-3)

    def sums(rows):
        return torch.zeros(groups, width, device="cuda", dtype=torch.float64).index_add_(0, ids, rows.double())

    x = torch.randn(n, width, device="cuda", generator=gen)
    members = counts.double().clamp(min=1)[:, None]
    mean = rt.cluster_mean(x, ids, counts)
    bound = (members + 1) * eps * sums(x.abs()) / members
    assert bool(((mean.double() - sums(x) / members).abs() <= bound).all())
    output = torch.randn(groups, width, device="cuda", generator=gen)[ids]
    plain, exact, fast = (rt.cluster_reconstruct_backward(x, ids, output, groups, relu, output_is_forward_result=per_bucket)
                          for relu, per_bucket in ((False, False), (True, False), (True, True)))
    assert torch.equal(exact, fast)
    captured = torch.cuda.CUDAGraph()
    with torch.cuda.graph(captured):
        again = rt.cluster_mean(x, ids, counts)
    captured.replay()
    assert torch.equal(again, mean)
    for got, kept in ((plain, x), (exact, x * (output > 0))):
        assert bool(((got.double() - sums(kept)).abs() <= members * eps * sums(kept.abs())).all())


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_expanded_rows_of_no_whole_vectors(rt, dtype):
    """The row-block form of the reconstruction: widths whose vectors cross rows at every offset, on both sides of the
    256 positions a block holds, row counts with every remainder; bit for bit the oracle's, dropped and kept
    elements those of the whole-vector kernels (a mask is a function of the element's position)."""
    rng = np.random.default_rng(11)
    for width in (5, 6, 7, 9, 47, 127, 129, 254, 255, 257, 258, 602):
        for n in (1, 2, 3, 5, 8, 1026, 4099):
            idx = rng.integers(0, 9, n)
            reps, bias = rng.standard_normal((9, width)).astype(dtype), rng.standard_normal(width).astype(dtype)
            for relu in (False, True):
                got = rt.cluster_reconstruct(cu(reps), cu(idx), cu(bias), relu)
                np.testing.assert_array_equal(got.cpu().numpy(), oracle.reconstruct(reps, idx, bias, relu))
            dropped = rt.cluster_reconstruct(cu(reps), cu(idx), cu(bias), True, 0.4, 77).flatten()
            # the same element positions through rows of one 16-byte vector
            flat = torch.nn.functional.pad(got.flatten(), (0, -got.numel() % 4)).view(-1, 4)
            mask = rt.cluster_reconstruct(torch.ones_like(flat), torch.arange(flat.size(0), device="cuda"), None, True, 0.4, 77)
            want = got.flatten() * (mask.flatten()[:got.numel()] != 0) * dtype(1.0 / 0.6)
            np.testing.assert_allclose(dropped.cpu().numpy(), want.cpu().numpy(), rtol=1e-6)
    bad = torch.tensor([0, 9, 2, -1, 3], device="cuda")
    out = rt.cluster_reconstruct(cu(reps), bad, None, False)
    assert not out[1].any() and not out[3].any() and torch.equal(out[4], cu(reps)[3])
    with pytest.raises(RuntimeError):
        rt.raise_on_device_status()


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_expanded_rows_few_and_wide(rt, dtype):
    """Few rows whose columns are shared among the blocks, and rows behind the last whole block of rows: bit for bit
    the oracle's."""
    rng = np.random.default_rng(12)
    for width in (511, 513, 10007, 227329):  # 888 slices of 256 positions and one more
        for n in (1, 2, 3, 5, 9, 103):
            if n * width > 3_000_000:
                continue
            idx = rng.integers(0, 4, n)
            reps, bias = rng.standard_normal((4, width)).astype(dtype), rng.standard_normal(width).astype(dtype)
            got = rt.cluster_reconstruct(cu(reps), cu(idx), cu(bias), True)
            np.testing.assert_array_equal(got.cpu().numpy(), oracle.reconstruct(reps, idx, bias, True))
