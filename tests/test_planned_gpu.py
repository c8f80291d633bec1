"""GPU parity tests of the one-launch SpMM (plans and groups), called through the C ABI, against the CPU
oracle (fp32 restatement of the reference's host loop, SSpMM/sspmm_test.cpp:75-95).  Tolerances are the
ones of test_spmm_gpu.py."""
import numpy as np
import pytest
import torch

from oracle import spmm_oracle
from sspmm_b200 import ops, synthetic
from tests.test_spmm_gpu import assert_close, compress, random_cvse

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def dev(*arrays):
    return [torch.from_numpy(np.ascontiguousarray(a)).to(DEV) for a in arrays]


def planned(ptr, col, vals, rhs, V, out_dtype):
    d_ptr, d_col, d_val, d_rhs = dev(ptr, col, vals, rhs)
    plan = ops.Plan(d_ptr, d_col, V, rhs.shape[0])
    out = ops.sspmm_planned(plan, d_val, d_rhs, out_dtype=out_dtype)
    torch.cuda.synchronize()
    assert ops.device_status() == 0
    return plan, out.float().cpu().numpy()


@pytest.mark.parametrize("out_dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("V", [8, 16])
def test_config1_planned(lib, V, out_dtype):
    a, rhs = synthetic.config1()
    ptr, col, vals = compress(a, V)
    ref = spmm_oracle.sspmm_host(V, ptr, col, vals, rhs)
    plan, got = planned(ptr, col, vals, rhs, V, out_dtype)
    assert plan.one_launch and plan.ascending and plan.nvec == col.size
    assert_close(got, ref, fp32=out_dtype == torch.float32)


@pytest.mark.parametrize("shape_id", [0, 1])
@pytest.mark.parametrize("sparsity_id", [0, 1, 2, 3, 4, 5])
def test_ffn_v16_planned_and_grouped(lib, shape_id, sparsity_id):
    """All twelve FFN cases: the planned call (static tiles) and a group of one (queue, K cut into parts)."""
    a, rhs = synthetic.ffn(shape_id, sparsity_id)
    ptr, col, vals = compress(a, 16)
    ref = spmm_oracle.sspmm_host(16, ptr, col, vals, rhs, threads=8)
    plan, got = planned(ptr, col, vals, rhs, 16, torch.float16)
    if not plan.one_launch:
        assert col.size < ptr.size * a.K / 16          # only very sparse structures are left to the gather kernels
    assert_close(got, ref)
    if plan.one_launch:
        d_val, d_rhs = dev(vals, rhs)
        for dt, mode in ((torch.float16, ops.Group.COMPRESSED), (torch.float32, ops.Group.COMPRESSED), (torch.float16, ops.Group.EXPANDED),
                         (torch.float16, ops.Group.PAIRS), (torch.float32, ops.Group.PAIRS)):
            out = torch.full((a.M, rhs.shape[1]), float("nan"), dtype=dt, device=DEV)
            g = ops.Group([(plan, d_val, d_rhs, out)], mode=mode)
            assert g.launches == 1
            for _ in range(3):                         # the queue and the arrival counters reset themselves
                out.fill_(float("nan"))
                g.run()
            torch.cuda.synchronize()
            assert ops.device_status() == 0
            assert_close(out.float().cpu().numpy(), ref, fp32=dt == torch.float32)


@pytest.mark.parametrize("V", [8, 16])
@pytest.mark.parametrize("N", [8, 64, 72, 136, 200, 256, 520])
def test_ragged_unsorted_rows_and_tails(lib, V, N):
    """Unsorted column lists (the permutation path), empty rows, a partial last row tile, K and N tails."""
    rng = np.random.default_rng(300 + N + V)
    lens = [0, 1, 2, 3, 15, 16, 17, 31, 33, 63, 64, 65, 0, 127, 129, 200, 0, 70, 5]
    K = 300
    ptr, col, vals = random_cvse(rng, len(lens), K, V, lens)
    rhs = rng.normal(0, 1, (K, N)).astype(np.float16)
    ref = spmm_oracle.sspmm_host(V, ptr, col, vals, rhs)
    for dt in (torch.float32, torch.float16):
        plan, got = planned(ptr, col, vals, rhs, V, dt)
        assert plan.one_launch and not plan.ascending
        assert_close(got, ref, fp32=dt == torch.float32)


def test_irregular_structure_falls_back(lib):
    """A column listed twice in a vector row: the plan carries no metadata and the call still gives the
    reference's answer (both vectors count), through the regular entry point."""
    ptr = np.array([0, 3, 5], dtype=np.int32)
    col = np.array([4, 9, 4, 0, 63], dtype=np.int32)
    rng = np.random.default_rng(5)
    vals = rng.uniform(-1, 1, 5 * 8).astype(np.float16)
    rhs = rng.normal(0, 1, (64, 64)).astype(np.float16)
    ref = spmm_oracle.sspmm_host(8, ptr, col, vals, rhs)
    plan, got = planned(ptr, col, vals, rhs, 8, torch.float32)
    assert not plan.one_launch
    assert_close(got, ref, fp32=True)
    d_val, d_rhs = dev(vals, rhs)
    with pytest.raises(Exception):
        ops.Group([(plan, d_val, d_rhs, torch.empty((16, 64), dtype=torch.float16, device=DEV))])


@pytest.mark.parametrize("mode", [ops.Group.COMPRESSED, ops.Group.EXPANDED, ops.Group.PAIRS])
def test_group_of_mixed_products(lib, mode):
    """Products of different shapes, V = 8 and 16, K from 64 to 2304, column counts with partial tiles, in one
    group (A tiles built in the kernel, or fetched from dense copies written at every run); every product against
    the oracle; replays give bit-identical results."""
    rng = np.random.default_rng(77)
    shapes = [(256, 2304, 16, 0.9, 1000), (64, 576, 8, 0.8, 1000), (512, 128, 16, 0.8, 1000), (256, 64, 8, 0.9, 1000),
              (1024, 256, 8, 0.9, 328), (128, 1152, 16, 0.8, 328)]
    prods, refs = [], []
    for (M, K, V, s, N) in shapes:
        a = synthetic.magnitude_pruned(M, K, s, rng)
        ptr, col, vals = compress(a, V)
        rhs = rng.normal(0, 1, (K, N)).astype(np.float16)
        d_ptr, d_col, d_val, d_rhs = dev(ptr, col, vals, rhs)
        plan = ops.Plan(d_ptr, d_col, V, K)
        assert plan.one_launch
        out = torch.full((M, N), float("nan"), dtype=torch.float16, device=DEV)
        prods.append((plan, d_val, d_rhs, out))
        refs.append(spmm_oracle.sspmm_host(V, ptr, col, vals, rhs, threads=8))
    g = ops.Group(prods, mode=mode)
    g.run()
    torch.cuda.synchronize()
    assert ops.device_status() == 0
    first = [p[3].clone() for p in prods]
    for (plan, _, _, out), ref in zip(prods, refs):
        assert_close(out.float().cpu().numpy(), ref)
    for _ in range(2):
        for p in prods:
            p[3].fill_(float("nan"))
        g.run()
        torch.cuda.synchronize()
        for p, f in zip(prods, first):
            assert torch.equal(p[3], f)
    assert ops.device_status() == 0


@pytest.mark.parametrize("N", [3136, 25088])
def test_conv_layer_planned_wide(lib, N):
    """Conv layer (512, 4608) at the 8-GPU shard width and at full width: planned call and group against the
    oracle on sampled vector rows, and against each other everywhere."""
    a = synthetic.conv_weight(3, 1)
    V = 16
    ptr, col, vals = compress(a, V)
    rng = np.random.default_rng(15)
    rhs = rng.normal(0, 1, (a.K, N)).astype(np.float16)
    d_ptr, d_col, d_val, d_rhs = dev(ptr, col, vals, rhs)
    plan = ops.Plan(d_ptr, d_col, V, a.K)
    assert plan.one_launch
    got = ops.sspmm_planned(plan, d_val, d_rhs)
    out = torch.full_like(got, float("nan"))
    out2 = torch.full_like(got, float("nan"))
    g = ops.Group([(plan, d_val, d_rhs, out)], mode=ops.Group.COMPRESSED)
    g2 = ops.Group([(plan, d_val, d_rhs, out2)], mode=ops.Group.EXPANDED)
    out3 = torch.full_like(got, float("nan"))
    g3 = ops.Group([(plan, d_val, d_rhs, out3)], mode=ops.Group.PAIRS)
    g.run()
    g2.run()
    g3.run()
    torch.cuda.synchronize()
    assert ops.device_status() == 0
    a_np, b_np = got.float().cpu().numpy(), out.float().cpu().numpy()
    assert_close(b_np, a_np)
    assert_close(out2.float().cpu().numpy(), a_np)
    assert_close(out3.float().cpu().numpy(), a_np)
    for rows in ((0, 2), (15, 17), (a.M // V - 2, a.M // V)):
        ref = spmm_oracle.sspmm_host(V, ptr, col, vals, rhs, rows=rows, threads=8)
        assert_close(a_np[rows[0] * V: rows[1] * V], ref)
        assert_close(b_np[rows[0] * V: rows[1] * V], ref)


@pytest.mark.parametrize("out_dtype", [torch.float16, torch.float32])
@pytest.mark.parametrize("shapes,rows", [
    ([(24, 64, 8)], True), ([(256, 256, 128)] * 3, True), ([(256, 1024, 128)], True), ([(8, 100, 72), (1000, 300, 8), (64, 64, 200)], True),
    ([(40, 130, 64)] * 8, True),                                                # as many products as one launch takes
    ([(40, 130, 64)] * 9, False),
    ([(128, 4608, 1000), (64, 576, 512)], False),                              # deep tiles are cut, shallow ones are not
    ([(768, 3072, 1000)], False), ([(384, 2048, 2048)], False), ([(1024, 768, 4104)], False)])      # few wide tiles, many, copies of A
def test_automatic_group(lib, shapes, rows, out_dtype):
    """Automatic groups on both sides of the lines between the row-gather kernel, cut tiles, whole tiles and dense copies."""
    rng = np.random.default_rng(len(shapes))
    prods, refs = [], []
    for (M, K, N) in shapes:
        a = synthetic.magnitude_pruned(M, K, 0.8, rng)
        ptr, col, vals = compress(a, 8)
        rhs = rng.normal(0, 1, (K, N)).astype(np.float16)
        d_ptr, d_col, d_val, d_rhs = dev(ptr, col, vals, rhs)
        plan = ops.Plan(d_ptr, d_col, 8, K)
        prods.append((plan, d_val, d_rhs, torch.full((plan.m_vec * 8, N), float("nan"), dtype=out_dtype, device=DEV)))
        refs.append((spmm_oracle.sspmm_host(8, ptr, col, vals, rhs, threads=8)))
    g = ops.Group(prods)
    assert g.launches == 1 and (g.work_items == sum((p[0].m_vec * -(-p[2].shape[1] // 64)) for p in prods)) == rows
    for _ in range(2):
        for p in prods:
            p[3].fill_(float("nan"))
        g.run()
        torch.cuda.synchronize()
        assert ops.device_status() == 0
        for p, ref in zip(prods, refs):
            assert_close(p[3].float().cpu().numpy(), ref, fp32=out_dtype == torch.float32)


def test_automatic_group_of_both_vector_lengths(lib):
    rng = np.random.default_rng(3)
    prods, refs = [], []
    for V in (8, 16):
        ptr, col, vals = compress(synthetic.magnitude_pruned(64, 200, 0.7, rng), V)
        rhs = rng.normal(0, 1, (200, 72)).astype(np.float16)
        d_ptr, d_col, d_val, d_rhs = dev(ptr, col, vals, rhs)
        prods.append((ops.Plan(d_ptr, d_col, V, 200), d_val, d_rhs, torch.empty((64, 72), dtype=torch.float16, device=DEV)))
        refs.append(spmm_oracle.sspmm_host(V, ptr, col, vals, rhs))
    g = ops.Group(prods)
    g.run()
    g.run()
    for p, ref in zip(prods, refs):
        assert_close(p[3].float().cpu().numpy(), ref)


def test_group_biases(lib):
    """A group of the row-gather kernel adds biases from the run after they were given, a tile group says that it does not."""
    rng = np.random.default_rng(12)
    ptr, col, vals = compress(synthetic.magnitude_pruned(100, 200, 0.7, rng), 8)
    for N, taken in ((72, True), (20000, False)):
        rhs = rng.normal(0, 1, (200, N)).astype(np.float16)
        d_ptr, d_col, d_val, d_rhs = dev(ptr, col, vals, rhs)
        out = torch.empty((104, N), dtype=torch.float32, device=DEV)
        g = ops.Group([(ops.Plan(d_ptr, d_col, 8, 200), d_val, d_rhs, out)])
        g.run()
        plain = out.clone()
        bias = torch.randn(104, device=DEV).half()
        assert g.bias(0, bias) == taken
        g.run()
        assert torch.equal(out, plain + bias.float()[:, None] if taken else plain)
        assert g.bias(0, None) == taken
        g.run()
        assert torch.equal(out, plain)
        with pytest.raises(ValueError):
            g.bias(0, bias[:100])
        with pytest.raises(IndexError):
            g.bias(1, bias)


@pytest.mark.parametrize("longest,rows", [(300, True), (2000, False)])
def test_automatic_group_with_a_long_row(lib, longest, rows):
    rng = np.random.default_rng(longest)
    ptr, col, vals = random_cvse(rng, 40, 2048, 8, [140] * 39 + [longest])
    rhs = rng.normal(0, 1, (2048, 64)).astype(np.float16)
    d_ptr, d_col, d_val, d_rhs = dev(ptr, col, vals, rhs)
    out = torch.empty((320, 64), dtype=torch.float32, device=DEV)
    plan = ops.Plan(d_ptr, d_col, 8, 2048)
    g = ops.Group([(plan, d_val, d_rhs, out)])
    assert plan.one_launch and (g.work_items == 40) == rows
    g.run()
    assert_close(out.cpu().numpy(), spmm_oracle.sspmm_host(8, ptr, col, vals, rhs), fp32=True)


@pytest.mark.parametrize("mode", [ops.Group.AUTO, ops.Group.COMPRESSED, ops.Group.EXPANDED])
def test_fp32_groups_keep_their_sums_short(lib, mode):
    """Eight products of 512 x 4608 at N = 200: parts of at most 18 steps of 64 columns, which the tensor unit adds in 72 additions that
    truncate.  One loses 0.72 * 2^-24 of the sum so far on average (half a unit in the last place, over all mantissas), and the sum of
    products of random sign after j of n additions is sqrt(j / n) of the last one, 2/3 on average; the parts are added in
    round-to-nearest.  Parts of 36 steps lose twice as much."""
    rng = np.random.default_rng(31)
    K, g = 4608, torch.Generator(device=DEV).manual_seed(31)
    d_ptr, d_col, d_val = dev(*random_cvse(rng, 32, K, 16, [3700] * 32))
    d_val = torch.randn(d_val.numel(), device=DEV, generator=g).half()
    dense = torch.zeros((32, 16, K), dtype=torch.float64, device=DEV)
    dense[torch.arange(32, device=DEV).repeat_interleave(3700), :, d_col.long()] = d_val.double().view(-1, 16)
    dense = dense.view(512, K)
    plan = ops.Plan(d_ptr, d_col, 16, K)
    prods = [(plan, d_val, torch.randn(K, 200, device=DEV, generator=g).half(), torch.empty((512, 200), device=DEV)) for _ in range(8)]
    ops.Group(prods, mode=mode).run()
    for _, _, rhs, out in prods:
        ref = dense @ rhs.double()
        assert (out.double() - ref).norm() <= 2 / 3 * 0.72 * 72 * 2.0 ** -24 * ref.norm()
    assert ops.device_status() == 0


@pytest.mark.parametrize("N,tiles", [(9984, 4 * 39), (19200, 4 * 75)])
@pytest.mark.parametrize("mode", [ops.Group.AUTO, ops.Group.COMPRESSED])
def test_deep_tiles_of_several_rounds_stay_whole(lib, mode, N, tiles):
    """512 x 4608 at just over one and two rounds of tiles: whole tiles of 256 columns; in parts every round of tiles has its round of
    sums (N = 19200: 258 us in three parts, 125 whole)."""
    rng = np.random.default_rng(N)
    d_ptr, d_col, d_val = dev(*random_cvse(rng, 32, 4608, 16, [3700] * 32))
    rhs, out = torch.zeros((4608, N), dtype=torch.float16, device=DEV), torch.full((512, N), float("nan"), dtype=torch.float16, device=DEV)
    g = ops.Group([(ops.Plan(d_ptr, d_col, 16, 4608), d_val, rhs, out)], mode=mode)
    assert torch.cuda.get_device_properties(0).multi_processor_count != 148 or (g.tile_columns, g.work_items) == (256, tiles)
    g.run()
    assert not out.any() and ops.device_status() == 0


def test_automatic_group_with_a_deep_product_of_few_rows(lib):
    """A warp would walk 230 steps of the deep product's rows while the others are done after eight: a tile group (row-gather groups
    add biases, the others say that they do not)."""
    rng = np.random.default_rng(9)
    prods, refs = [], []
    for (m_vec, K, n, N) in ((8, 4608, 3700, 64), (256, 300, 120, 256), (256, 300, 120, 256)):
        ptr, col, vals = random_cvse(rng, m_vec, K, 8, [n] * m_vec)
        rhs = rng.normal(0, 1, (K, N)).astype(np.float16)
        d_ptr, d_col, d_val, d_rhs = dev(ptr, col, vals, rhs)
        prods.append((ops.Plan(d_ptr, d_col, 8, K), d_val, d_rhs, torch.empty((m_vec * 8, N), device=DEV)))
        refs.append(spmm_oracle.sspmm_host(8, ptr, col, vals, rhs, threads=8))
    g, shallow = ops.Group(prods), ops.Group(prods[1:2])
    assert not g.bias(0, None) and shallow.bias(0, None)
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:        # 256 rows x 2 tiles, two items of four warps in a CTA
        assert (shallow.tile_columns, shallow.work_items, shallow.ctas) == (128, 512, 256)
    g.run()
    for p, ref in zip(prods, refs):
        assert_close(p[3].cpu().numpy(), ref, fp32=True)
    shallow.run()
    assert_close(prods[1][3].cpu().numpy(), refs[1], fp32=True)


def test_no_copies_where_the_loaders_keep_up(lib):
    """512 x 1024 at N = 25088: 392 equal tiles, 47.7 steps per SM of 148."""
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the figures are those of 148 SMs")
    d_ptr, d_col, d_val = dev(*random_cvse(np.random.default_rng(2), 32, 1024, 16, [830] * 32))
    rhs, out = torch.zeros((1024, 25088), dtype=torch.float16, device=DEV), torch.full((512, 25088), float("nan"), device=DEV)
    g = ops.Group([(ops.Plan(d_ptr, d_col, 16, 1024), d_val, rhs, out)])
    assert (g.tile_columns, g.work_items, g.scratch_bytes) == (256, 392, 0)
    g.run()
    assert not out.any() and ops.device_status() == 0
