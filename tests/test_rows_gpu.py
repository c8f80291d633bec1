"""GPU parity tests of the row-gather kernel and of the choice between it, the block kernel and the aligned copy of B, at
the sizes where they can go wrong: one vector, one step and one more, rows of one CTA and of a cluster, partial column
tiles, unaligned dense operands, row orders, rows that are cut.

Tolerance: a sum of n products of fp16 numbers in fp32 in any order is within n * 2^-23 * sum|a||b| of the exact one (the
tensor cores truncate, hence 2^-23 and not 2^-24); fp16 output adds half a unit of the result, 2^-11 |c|."""
import numpy as np
import pytest
import torch

from sspmm_b200 import ops
from sspmm_b200.sptrans.spmm import bspmm

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def operands(lens, K, V, N, seed, offset=0):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    ptr = torch.zeros(len(lens) + 1, dtype=torch.int32, device=DEV)
    ptr[1:] = torch.cumsum(torch.tensor(lens, device=DEV), 0)
    nvec = int(ptr[-1])
    col = torch.cat([torch.randperm(K, device=DEV, generator=g)[:n] for n in lens]).int()
    val = (torch.rand(nvec * V, device=DEV, generator=g) * 2 - 1).half()
    flat = torch.randn(K * N + offset, device=DEV, generator=g).half()
    return ptr, col, val, flat[offset:].view(K, N)


def exact(ptr, col, val, rhs, V):
    """The product and the sums of magnitudes, in 64 bits."""
    m = ptr.numel() - 1
    rows = torch.repeat_interleave(torch.arange(m, device=DEV), (ptr[1:] - ptr[:-1]).long())
    a = torch.zeros(m * V, rhs.shape[0], dtype=torch.float64, device=DEV)
    v = val.double().view(-1, V)
    for r in range(V):
        a[rows * V + r, col.long()] = v[:, r]
    return a @ rhs.double(), a.abs() @ rhs.double().abs()


def check(got, ptr, col, val, rhs, V):
    ref, mag = exact(ptr, col, val, rhs, V)
    n = int((ptr[1:] - ptr[:-1]).max())
    bound = max(n, 1) * 2.0 ** -23 * mag + 1e-30
    if got.dtype == torch.float16:
        bound = bound + 2.0 ** -11 * ref.abs() + 2.0 ** -24
    assert (got.double() - ref).abs().le(bound).all()
    assert ops.device_status() == 0


@pytest.mark.parametrize("V", [8, 16])
@pytest.mark.parametrize("lens,K,N", [
    ([1], 64, 8), ([16, 17, 0, 15, 33], 64, 72), ([300] * 3, 512, 64), ([2600, 1, 0], 4608, 136), ([700] * 300, 1024, 128),
    ([40] * 3000, 300, 200)])
@pytest.mark.parametrize("kernel", [ops.KERNEL_AUTO, ops.KERNEL_GATHER_LSU])
def test_tile_edges_teams_and_clusters(lib, V, lens, K, N, kernel):
    ptr, col, val, rhs = operands(lens, K, V, N, 3)
    ops.set_kernel(kernel)
    try:
        for dt in (torch.float16, torch.float32):
            check(ops.sspmm(ptr, col, val, rhs, V, out_dtype=dt), ptr, col, val, rhs, V)
    finally:
        ops.set_kernel(ops.KERNEL_AUTO)


@pytest.mark.parametrize("V", [8, 16])
@pytest.mark.parametrize("rows,len_,N", [(74, 560, 64), (75, 560, 64), (75, 1780, 64), (75, 1800, 64), (37, 640, 64), (38, 640, 64), (37, 630, 64), (9, 640, 200)])
def test_edges_of_the_division_into_clusters(lib, V, rows, len_, N):
    """148 SMs: items that get an SM each in clusters of two or not, and of four, rows of 112 steps and more, of 40 and fewer; a row that
    is longer than the mean and an empty one."""
    ptr, col, val, rhs = operands([len_] * (rows - 2) + [0, min(2 * len_, 2000)], 2000, V, N, rows)
    for dt in (torch.float16, torch.float32):
        check(ops.sspmm(ptr, col, val, rhs, V, out_dtype=dt), ptr, col, val, rhs, V)


@pytest.mark.parametrize("V", [8, 16])
@pytest.mark.parametrize("lens,K,N,offset", [([5, 0, 40], 64, 1, 0), ([900] * 4, 1000, 49, 0), ([40] * 20, 64, 50, 0), ([40] * 20, 64, 64, 3),
                                             ([1000] * 64, 1024, 1001, 1)])
def test_unaligned_dense_operand(lib, V, lens, K, N, offset):
    """N not a multiple of 8, rhs off its 16-byte boundary; the last one runs the block kernel on the aligned copy."""
    ptr, col, val, rhs = operands(lens, K, V, N, 4, offset)
    for kernel in (ops.KERNEL_AUTO, ops.KERNEL_GATHER_LSU, ops.KERNEL_BLOCK, ops.KERNEL_SIMT):
        ops.set_kernel(kernel)
        try:
            for dt in (torch.float16, torch.float32):
                check(ops.sspmm(ptr, col, val, rhs, V, out_dtype=dt), ptr, col, val, rhs, V)
        finally:
            ops.set_kernel(ops.KERNEL_AUTO)


@pytest.mark.parametrize("V,N", [(8, 40), (8, 200), (16, 136)])
def test_cut_rows_any_order(lib, V, N):
    """One row of two parts, one of many, rows at both sides of what a warp does alone; any order gives the same numbers."""
    lens = [257, 256, 0, 1, 600, 2900] + [20] * 200
    ptr, col, val, rhs = operands(lens, 3000, V, N, 5)
    base = ops.sspmm(ptr, col, val, rhs, V, out_dtype=torch.float32)
    check(base, ptr, col, val, rhs, V)
    order = torch.randperm(len(lens), device=DEV).int()
    assert torch.equal(base, ops.sspmm(ptr, col, val, rhs, V, row_indices=order, out_dtype=torch.float32))
    check(ops.sspmm(ptr, col, val, rhs, V), ptr, col, val, rhs, V)


@pytest.mark.parametrize("V,N", [(8, 64), (16, 49)])
def test_batches(lib, V, N):
    lens = [51, 0, 70, 16]
    ptr, col, val, _ = operands(lens, 80, V, 8, 6)
    rhs = torch.randn(5, 80, N, device=DEV).half()
    vals = torch.stack([val * s for s in (1.0, -1.0, 0.5, 2.0, 0.25)])
    order = torch.arange(len(lens), dtype=torch.int32, device=DEV)
    got = bspmm(order, ptr, col, vals, rhs, V)
    for b in range(5):
        check(got[b], ptr, col, vals[b], rhs[b], V)


@pytest.mark.parametrize("V,M,K,N", [(8, 512, 2048, 200), (16, 64, 64, 8), (16, 1500, 3000, 72)])
def test_planned_small_products(lib, V, M, K, N):
    lens = [int(x) for x in np.random.default_rng(7).integers(K // 2, K, -(-M // V))]
    ptr, col, val, rhs = operands(lens, K, V, N, 8)
    plan = ops.Plan(ptr, col, V, K)
    assert plan.one_launch
    for dt in (torch.float16, torch.float32):
        check(ops.sspmm_planned(plan, val, rhs, out_dtype=dt), ptr, col, val, rhs, V)


@pytest.mark.parametrize("V", [8, 16])
@pytest.mark.parametrize("lens,K,N", [([40, 0, 17], 64, 8), ([900] * 40, 1000, 49), ([700] * 40, 1024, 1024), ([400] * 80, 512, 8192),
                                      ([600] + [5] * 300, 3000, 40)])
def test_bias_in_every_epilogue(lib, V, lens, K, N):
    """Per-row bias: row-gather (teams, cut rows, aligned copy), block kernel with and without split K, CTA pairs, CUDA cores."""
    ptr, col, val, rhs = operands(lens, K, V, N, 9)
    bias = torch.randn(len(lens) * V, device=DEV).half()
    ref, mag = exact(ptr, col, val, rhs, V)
    ref, mag = ref + bias.double()[:, None], mag + bias.double().abs()[:, None]
    for kernel in (ops.KERNEL_AUTO, ops.KERNEL_GATHER_LSU, ops.KERNEL_BLOCK, ops.KERNEL_BLOCK_SINGLE, ops.KERNEL_SIMT):
        ops.set_kernel(kernel)
        try:
            for dt in (torch.float16, torch.float32):
                got = ops.sspmm_bias(ptr, col, val, rhs, V, bias, out_dtype=dt).double()
                bound = (max(lens) + 1) * 2.0 ** -23 * mag + (2.0 ** -11 * ref.abs() + 2.0 ** -24 if dt == torch.float16 else 0)
                assert (got - ref).abs().le(bound).all(), kernel
        finally:
            ops.set_kernel(ops.KERNEL_AUTO)
    assert ops.device_status() == 0


@pytest.mark.parametrize("V,N", [(8, 1000), (16, 4096)])
def test_cut_rows_of_wide_products(lib, V, N):
    """Parts grow with the number of column tiles: rows of several parts, of one, and short ones, over many tiles."""
    lens = [2900, 513, 512, 257, 256, 0, 2900, 600] + [20] * 200
    ptr, col, val, rhs = operands(lens, 3000, V, N, 10)
    assert ops.workspace_bytes(len(lens), V, N, 3000, sum(lens)) > 0
    for dt in (torch.float16, torch.float32):
        check(ops.sspmm(ptr, col, val, rhs, V, out_dtype=dt), ptr, col, val, rhs, V)


@pytest.mark.parametrize("V,N", [(8, 136), (16, 64)])
def test_cut_rows_listed_by_many_ctas(lib, V, N):
    """More than 16384 vector rows: the list comes from several CTAs."""
    lens = [3] * 9000 + [2500, 0, 300, 900] + [2] * 11000 + [1100]
    ptr, col, val, rhs = operands(lens, 2600, V, N, 11)
    assert ops.workspace_bytes(len(lens), V, N, 2600, sum(lens)) > 0
    got = ops.sspmm(ptr, col, val, rhs, V, out_dtype=torch.float32)
    for a, b in ((0, 40), (8990, 9020), (20000, len(lens))):
        part = (ptr[a:b + 1] - ptr[a]).int()
        s = slice(int(ptr[a]), int(ptr[b]))
        check(got[a * V:b * V], part, col[s], val.view(-1, V)[s].reshape(-1), rhs, V)
    assert torch.equal(got, ops.sspmm(ptr, col, val, rhs, V, row_indices=ops.sorted_row_swizzle(ptr), out_dtype=torch.float32))


@pytest.mark.parametrize("stated", [300, 4000, 20000])
def test_a_count_that_is_too_small_cuts_nothing(lib, stated):
    """The list is sized from the count; when the matrix holds more long rows than that, the result is the same."""
    from sspmm_b200 import capi
    V, N, K = 8, 72, 3000
    lens = [2800] * 40 + [300] * 300 + [10] * 60
    ptr, col, val, rhs = operands(lens, K, V, N, 12)
    assert ops.workspace_bytes(len(lens), V, N, K, stated) > 0
    out = torch.full((len(lens) * V, N), float("nan"), device=DEV)
    for kernel in (ops.KERNEL_AUTO, ops.KERNEL_GATHER_LSU):
        ops.set_kernel(kernel)
        try:
            capi.check(capi.lib().sspmm_counted(len(lens), V, N, K, 1, stated, None, ptr.data_ptr(), col.data_ptr(), val.data_ptr(), 0,
                                                rhs.data_ptr(), 0, None, out.data_ptr(), 0, 0, torch.cuda.current_stream().cuda_stream))
            check(out, ptr, col, val, rhs, V)
        finally:
            ops.set_kernel(ops.KERNEL_AUTO)


@pytest.mark.parametrize("V", [8, 16])
@pytest.mark.parametrize("lens,K,N", [
    ([1500] + [30] * 4000, 1600, 128), ([20] * 2403 + [257, 256, 700, 1, 1600], 1600, 136), ([1600] * 9 + [0] * 700 + [512, 513], 1600, 64),
    ([30] * 300 + [1025, 1024, 1600], 1600, 200), ([300] * 600 + [2000] * 3, 2000, 1000)])
def test_long_rows_below_2048_columns(lib, V, lens, K, N):
    """Long rows among short ones, cut (all but the last) and not; any order gives the same numbers."""
    ptr, col, val, rhs = operands(lens, K, V, N, 15)
    ops.set_kernel(ops.KERNEL_GATHER_LSU)
    try:
        base = ops.sspmm(ptr, col, val, rhs, V, out_dtype=torch.float32)
        check(base, ptr, col, val, rhs, V)
        for order in (ops.sorted_row_swizzle(ptr), torch.randperm(len(lens), device=DEV).int()):
            assert torch.equal(base, ops.sspmm(ptr, col, val, rhs, V, row_indices=order, out_dtype=torch.float32))
        check(ops.sspmm(ptr, col, val, rhs, V), ptr, col, val, rhs, V)
    finally:
        ops.set_kernel(ops.KERNEL_AUTO)


def test_long_rows_of_a_batch(lib):
    V, K, N, lens = 8, 1024, 72, [1024, 1024] + [40] * 70 + [600]
    ptr, col, val, _ = operands(lens, K, V, 8, 16)
    rhs = torch.randn(30, K, N, device=DEV).half()
    vals = torch.stack([val * (1 - b / 64) for b in range(30)])
    got = bspmm(ops.sorted_row_swizzle(ptr), ptr, col, vals, rhs, V)
    for b in (0, 1, 17, 29):
        check(got[b], ptr, col, vals[b], rhs[b], V)


def test_more_than_two_to_the_28_items(lib):
    """Vector rows times column tiles are counted in 32 bits: up to 2^31 - 1 of them, less what the counter may run over."""
    V, N, K, m_vec = 8, 8, 64, (1 << 28) + 3
    if torch.cuda.mem_get_info()[0] < 60 << 30:
        pytest.skip("needs 36 GB")
    ptr = torch.zeros(m_vec + 1, dtype=torch.int32, device=DEV)
    ptr[5:] = 2
    ptr[m_vec] = 5
    col = torch.tensor([3, 60, 1, 2, 63], dtype=torch.int32, device=DEV)
    val = torch.randn(5 * V, device=DEV).half()
    rhs = torch.randn(K, N, device=DEV).half()
    out = torch.full((m_vec * V, N), float("nan"), dtype=torch.float16, device=DEV)
    ops.sspmm(ptr, col, val, rhs, V, out=out)
    v = val.double().view(5, V, 1)
    for row, s in ((4, slice(0, 2)), (m_vec - 1, slice(2, 5))):
        ref = (v[s] * rhs[col[s].long()].double()[:, None, :]).sum(0)
        assert (out[row * V:row * V + V].double() - ref).abs().max() <= 2.0 ** -9 * ref.abs().max()
    # everything else was written, with zeros
    assert sum(int(torch.count_nonzero(part)) for part in out.view(-1).split(1 << 30)) == 2 * V * N
    assert ops.device_status() == 0


@pytest.mark.parametrize("V,M,K,N,offset", [(8, 64, 1024, 1001, 0), (16, 128, 4608, 601, 0), (8, 128, 2048, 1024, 4)])
def test_unaligned_dense_operand_keeps_fp32_sums(lib, V, M, K, N, offset):
    """Products that the dense-tile path would take if they were aligned: fp32 results are no further from 64 bits than those of
    the CUDA-core kernel, which adds in round-to-nearest."""
    ptr, col, val, rhs = operands([K - 24] * M, K, V, N, 13, offset)
    ref, _ = exact(ptr, col, val, rhs, V)
    error = {}
    for kernel in (ops.KERNEL_AUTO, ops.KERNEL_BLOCK, ops.KERNEL_SIMT):
        ops.set_kernel(kernel)
        try:
            error[kernel] = (ops.sspmm(ptr, col, val, rhs, V, out_dtype=torch.float32).double() - ref).norm()
        finally:
            ops.set_kernel(ops.KERNEL_AUTO)
    assert error[ops.KERNEL_AUTO] <= error[ops.KERNEL_SIMT] and error[ops.KERNEL_BLOCK] <= error[ops.KERNEL_SIMT]


@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
@pytest.mark.parametrize("N,offset", [(1001, 0), (1024, 3)])
def test_unaligned_dense_operand_with_infinities(lib, N, offset, dtype):
    """An infinity or NaN of B reaches the vector rows that name its row, and no others."""
    K, V, lens = 1024, 8, [900] * 64
    ptr, col, val, rhs = operands(lens, K, V, N, 14, offset)
    rhs[5, 7], rhs[900, N - 1], rhs[17, 30] = float("inf"), float("-inf"), float("nan")
    got = ops.sspmm(ptr, col, val, rhs, V, out_dtype=dtype)
    names = lambda k: torch.stack([(col[a:b] == k).any() for a, b in zip(ptr[:-1].tolist(), ptr[1:].tolist())])
    want = torch.zeros(len(lens) * V, N, dtype=torch.bool, device=DEV)
    for k, n in ((5, 7), (900, N - 1), (17, 30)):
        hit = names(k).repeat_interleave(V)
        assert hit.any() and not hit.all()
        want[:, n] = hit
    assert torch.equal(~got.isfinite(), want)


@pytest.mark.parametrize("m,longest,K,N", [(2369, 40, 300, 64), (2400, 150, 160, 72), (800, 200, 256, 264), (37888, 3, 64, 128), (76032, 2, 64, 40)])
def test_more_items_than_warps(lib, m, longest, K, N):
    """One warp per item: a few more items than warps, empty rows and long ones among short ones, row orders, partial column tiles, as
    many rounds of CTAs as a table of look-ups holds (37888 items of 128 columns: 128; 76032: 257, one more than fit)."""
    rng = np.random.default_rng(m)
    lens = np.where(rng.random(m) < 0.05, longest, rng.integers(0, min(longest, 6), m))
    ptr, col, val, rhs = operands_fast(lens, K, 8, N, m)
    ops.set_kernel(ops.KERNEL_GATHER_LSU)
    try:
        for order in (None, ops.sorted_row_swizzle(ptr)):
            for dt in (torch.float16, torch.float32):
                check(ops.sspmm(ptr, col, val, rhs, 8, row_indices=order, out_dtype=dt), ptr, col, val, rhs, 8)
    finally:
        ops.set_kernel(ops.KERNEL_AUTO)


def operands_fast(lens, K, V, N, seed):
    """operands() for many rows: columns at a random place, one after another (wrapped)."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    n = torch.as_tensor(lens, device=DEV)
    ptr = torch.zeros(n.numel() + 1, dtype=torch.int32, device=DEV)
    ptr[1:] = torch.cumsum(n, 0)
    at = torch.arange(int(ptr[-1]), device=DEV) - torch.repeat_interleave(ptr[:-1].long(), n)
    col = ((at + torch.repeat_interleave(torch.randint(K, (n.numel(),), device=DEV, generator=g), n)) % K).int()
    return ptr, col, (torch.rand(col.numel() * V, device=DEV, generator=g) * 2 - 1).half(), torch.randn(K, N, device=DEV, generator=g).half()


def test_batch_of_more_items_than_warps(lib):
    """The longest row of every batch entry would fall to one warp if items were dealt out in turn: 64 rows, 2368 warps."""
    lens = [512] + [7] * 62 + [0]
    ptr, col, _, _ = operands_fast(lens, 512, 8, 64, 1)
    g = torch.Generator(device=DEV).manual_seed(2)
    val = torch.rand(96, col.numel() * 8, device=DEV, generator=g).half()
    rhs = torch.randn(96, 512, 72, device=DEV, generator=g).half()
    out = bspmm(ops.sorted_row_swizzle(ptr), ptr, col, val, rhs, 8)
    for b in (0, 1, 37, 95):
        check(out[b], ptr, col, val[b], rhs[b], 8)


# Rows that may be many times the mean: more warps for every item, warps by length (one round and several, empty rows, one item and
# several per cluster, 512 items and one more, 20 steps per warp of a full row and more), cut rows.
@pytest.mark.parametrize("V", [8, 16])
@pytest.mark.parametrize("lens,K,N", [
    ([230] * 128, 4608, 72), ([230] * 128, 4608, 49), ([0] * 127 + [2304], 2304, 48), ([2304] * 3 + [20] * 29, 2304, 800), ([4608] + [400] * 63, 4608, 56),
    ([115, 0, 17, 1, 33, 32, 600] * 20, 2304, 200), ([25] * 512, 2048, 64), ([25] * 513, 2048, 64), ([1000] * 8, 20480, 24), ([1000] * 8, 20496, 24),
    ([1], 2048, 8), ([1900] * 10 + [30] * 500, 2000, 64)])
def test_rows_that_may_be_long(lib, V, lens, K, N):
    ptr, col, val, rhs = operands(lens, K, V, N, 11)
    order = torch.randperm(len(lens), device=DEV).int()
    for dt in (torch.float16, torch.float32):
        got = ops.sspmm(ptr, col, val, rhs, V, out_dtype=dt)
        check(got, ptr, col, val, rhs, V)
        assert torch.equal(got, ops.sspmm(ptr, col, val, rhs, V, row_indices=order, out_dtype=dt))
    bias = torch.randn(len(lens) * V, device=DEV).half()
    assert torch.equal(ops.sspmm_bias(ptr, col, val, rhs, V, bias, out_dtype=torch.float32), got + bias.float()[:, None])


# Rows of B read where they lie: every offset from a 16-byte boundary, one element, row ends at the last column of a tile and of B, steps
# that do not fill a warp's share, clusters.  The same numbers in the same order as from an aligned copy of B.
@pytest.mark.parametrize("V", [8, 16])
@pytest.mark.parametrize("lens,K,N", [
    ([1], 1, 1), ([1], 1, 3), ([1, 1], 2, 3), ([3, 0, 5], 7, 5), ([17, 32, 0, 33], 40, 49), ([33] * 5, 33, 63), ([60] * 64, 60, 65), ([460] * 64, 600, 49),
    ([300] * 3, 301, 127)])
def test_rows_of_an_unaligned_operand(lib, V, lens, K, N):
    for offset in range(8):
        ptr, col, val, rhs = operands(lens, K, V, N, 7, offset)
        for dt in (torch.float16, torch.float32):
            got = ops.sspmm(ptr, col, val, rhs, V, out_dtype=dt)
            check(got, ptr, col, val, rhs, V)
            ops.set_kernel(ops.KERNEL_GATHER_LSU)
            try:
                want = ops.sspmm(ptr, col, val, rhs, V, out_dtype=dt)
            finally:
                ops.set_kernel(ops.KERNEL_AUTO)
            assert torch.equal(got, want)
        bias = torch.randn(len(lens) * V, device=DEV).half()
        assert torch.equal(ops.sspmm_bias(ptr, col, val, rhs, V, bias, out_dtype=torch.float32), got + bias.float()[:, None])
