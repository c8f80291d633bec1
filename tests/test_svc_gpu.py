"""GPU parity tests of sparse vector compression: the CUDA path, called through
the C ABI, against the golden vectors of the unmodified reference module and
against the CPU oracle on seeded inputs.  Integer outputs must be bit-exact."""
import numpy as np
import pytest
import torch

from oracle import svc_oracle
from sspmm_b200 import ops, synthetic
from tests.golden_cases import golden_cases, load_golden

pytestmark = pytest.mark.gpu

CASES = golden_cases()
GOLD = load_golden()


def run_gpu(a, V, with_values=True):
    dev = torch.device("cuda:0")
    ptr = torch.from_numpy(a.row_ptr).to(dev)
    col = torch.from_numpy(a.col_idx).to(dev)
    val = torch.from_numpy(a.values).to(dev) if with_values else None
    vec_ptr, vec_col, vec_val, replayed = ops.svc(ptr, col, val, a.M, a.K, V)
    torch.cuda.synchronize()
    return (vec_ptr.cpu().numpy(), vec_col.cpu().numpy(), None if vec_val is None else vec_val.cpu().numpy(), replayed)


def check_against_oracle(a, V):
    r = svc_oracle.cvse(a.M, a.K, a.nnz, a.row_lists(), V)
    ptr, col, val, _ = run_gpu(a, V)
    assert np.array_equal(ptr, np.asarray(r.vec_row_ptr, dtype=np.int32))
    assert np.array_equal(col, np.asarray(r.vec_colInd_list, dtype=np.int32))
    exp = svc_oracle.pack_values(a.M, V, a.row_ptr, a.col_idx, a.values, r)
    assert np.array_equal(val.view(np.uint16), exp.view(np.uint16))
    return r


@pytest.mark.parametrize("name", sorted(CASES))
def test_svc_matches_reference_golden(lib, name):
    a, V = CASES[name]
    ptr, col, val, replayed = run_gpu(a, V)
    assert np.array_equal(ptr, GOLD[name + "/vec_row_ptr"])
    assert np.array_equal(col, GOLD[name + "/vec_colInd_list"])
    # value vectors: densifying the compressed form gives back A
    dense = svc_oracle.densify(ptr.size - 1, V, a.K, ptr.tolist(), col.tolist(), val)
    assert np.array_equal(dense[: a.M].view(np.uint16), a.dense().view(np.uint16))
    assert not dense[a.M:].any()
    if name.startswith("powerlaw"):
        assert replayed > 0          # the hash-order replay really ran


@pytest.mark.parametrize("name", sorted(CASES))
def test_python_entry_point_matches_reference_golden(lib, name):
    from sspmm_b200 import sparse_matrix_format as smf
    a, V = CASES[name]
    c = smf.CVSE(a.M, a.K, a.nnz, a.row_lists(), V)
    assert c.vec_row_ptr == GOLD[name + "/vec_row_ptr"].tolist()
    assert c.vec_colInd_list == GOLD[name + "/vec_colInd_list"].tolist()
    assert c.tile_num == GOLD[name + "/tile_num"].tolist()
    assert [c.return_CSR_storage(), c.return_CVSE_storage(), c.return_TCF_storage(),
            c.return_SRBCSR_storage()] == GOLD[name + "/storage"].tolist()
    assert c.num_vec == len(c.vec_colInd_list) and len(c.vec_colInd_list_array) == c.num_vec_row


@pytest.mark.parametrize("V", [8, 16])
@pytest.mark.parametrize("shape_id,sparsity_id", [(0, 0), (0, 5), (1, 2), (1, 4)])
def test_svc_ffn_configs(lib, V, shape_id, sparsity_id):
    a, _ = synthetic.ffn(shape_id, sparsity_id)
    check_against_oracle(a, V)


def test_svc_power_law_with_giant_rows(lib):
    a = synthetic.power_law(16384, np.random.default_rng(123))
    r = check_against_oracle(a, 8)
    assert max(len(l) for l in r.vec_colInd_list_array) > 1229     # a table of 8192 slots or more was replayed


@pytest.mark.parametrize("V", [8, 16])
def test_svc_edge_cases(lib, V):
    rng = np.random.default_rng(V)
    cases = []
    # empty matrix rows everywhere
    cases.append(synthetic.CSR(40, 100, np.zeros(41, dtype=np.int32), np.zeros(0, dtype=np.int32), np.zeros(0, dtype=np.float16)))
    # single row, single entry, last column
    cases.append(synthetic.CSR(1, 70000, np.array([0, 1], dtype=np.int32), np.array([69999], dtype=np.int32), np.array([1.5], dtype=np.float16)))
    # M = 0
    cases.append(synthetic.CSR(0, 10, np.zeros(1, dtype=np.int32), np.zeros(0, dtype=np.int32), np.zeros(0, dtype=np.float16)))
    # dense rows (every column), M not a multiple of V
    M, K = 19, 96
    ptr = (np.arange(M + 1) * K).astype(np.int32)
    cases.append(synthetic.CSR(M, K, ptr, np.tile(np.arange(K, dtype=np.int32), M), rng.uniform(-1, 1, M * K).astype(np.float16)))
    # exactly at the growth thresholds of the hash table: 4, 5, 18, 19, 76, 77, 306, 307 distinct keys, wide key range
    for u in (4, 5, 18, 19, 76, 77, 306, 307, 1228, 1229):
        cols = rng.permutation(200000)[:u].astype(np.int32)
        cases.append(synthetic.CSR(1, 200000, np.array([0, u], dtype=np.int32), cols, rng.uniform(-1, 1, u).astype(np.float16)))
    # colliding keys: all congruent modulo every small table length
    cols = (np.arange(30, dtype=np.int32) * 8192 + 5)
    lens = [10, 0, 8, 12] + [0] * (V - 4)
    ptr = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    cases.append(synthetic.CSR(V, 30 * 8192, ptr, rng.permutation(cols).astype(np.int32), rng.uniform(-1, 1, 30).astype(np.float16)))
    for a in cases:
        check_against_oracle(a, V)


def test_svc_rejects_bad_column(lib):
    a = synthetic.CSR(2, 10, np.array([0, 1, 2], dtype=np.int32), np.array([3, 10], dtype=np.int32), np.ones(2, dtype=np.float16))
    from sspmm_b200 import capi
    with pytest.raises(capi.SspmmError):
        run_gpu(a, 8)
    # the library stays usable afterwards
    ok = synthetic.CSR(2, 10, np.array([0, 1, 2], dtype=np.int32), np.array([3, 9], dtype=np.int32), np.ones(2, dtype=np.float16))
    check_against_oracle(ok, 8)


def test_all_zero_vector_count_entry_point(lib):
    from sspmm_b200 import sparse_matrix_format as smf
    a, V = CASES["config1_v8"]
    om = smf.OriginMatrix(a.M, a.K, a.row_ptr, a.col_idx)
    assert smf.return_all_zero_vec(V, a.M, a.K, om) == int(GOLD["config1_v8/all_zero_vec_cnt"][0])


def test_sorted_row_swizzle(lib):
    a = synthetic.power_law(4096, np.random.default_rng(5))
    r = svc_oracle.cvse(a.M, a.K, a.nnz, a.row_lists(), 8)
    d = torch.tensor(r.vec_row_ptr, dtype=torch.int32, device="cuda:0")
    got = ops.sorted_row_swizzle(d).cpu().numpy()
    assert np.array_equal(got, svc_oracle.sorted_row_swizzle(r.vec_row_ptr))


@pytest.mark.parametrize("m_vec", [8192, 8193, 100_000, 262_144])
def test_sorted_row_swizzle_many_rows(lib, m_vec):
    """Around and far above the row count where the rank loop gives way to the sort: order = length descending, row id
    ascending among equal lengths (many ties: lengths are drawn from 0..40), a permutation of all rows."""
    rng = np.random.default_rng(m_vec)
    lens = rng.integers(0, 41, m_vec)
    lens[rng.integers(0, m_vec, 5)] = rng.integers(1000, 100000, 5)
    ptr = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    got = ops.sorted_row_swizzle(torch.from_numpy(ptr).to("cuda:0")).cpu().numpy()
    want = np.lexsort((np.arange(m_vec), -lens))
    assert np.array_equal(got, want)


def test_svc_full_size_properties(lib):
    """n = 65536 power-law matrix (largest sweep size): checked through
    size-independent properties instead of the slow CPU oracle."""
    a = synthetic.power_law(65536, np.random.default_rng(2024))
    V = 8
    ptr, col, val, _ = run_gpu(a, V)
    m_vec = a.M // V
    assert ptr[0] == 0 and np.all(np.diff(ptr) >= 0) and ptr[-1] == col.size
    # each vector row holds exactly the distinct columns of its V rows
    grp = np.repeat(np.arange(a.M) // V, np.diff(a.row_ptr)).astype(np.int64)
    key_in = np.unique(grp * a.K + a.col_idx)
    key_out = np.repeat(np.arange(m_vec, dtype=np.int64), np.diff(ptr)) * a.K + col
    assert key_out.size == key_in.size and np.array_equal(np.sort(key_out), key_in)
    # value vectors carry every original value once and zeros elsewhere
    assert np.isclose(val.astype(np.float64).sum(), a.values.astype(np.float64).sum(), atol=1e-6)
    assert np.count_nonzero(val) == np.count_nonzero(a.values)
    # spot-check a slice of vector rows against the oracle, including order
    sub = synthetic.CSR(512, a.K, (a.row_ptr[:513] - a.row_ptr[0]).astype(np.int32), a.col_idx[a.row_ptr[0]:a.row_ptr[512]], a.values[a.row_ptr[0]:a.row_ptr[512]])
    r = svc_oracle.cvse(sub.M, sub.K, sub.nnz, sub.row_lists(), V)
    assert np.array_equal(col[: ptr[64]], np.asarray(r.vec_colInd_list, dtype=np.int32))


def test_generate_cvse_file_batch_driver(lib, tmp_path):
    """The batch entry point row_merge.py calls (reference :190-250): files in, files + CSV rows out."""
    import csv
    from sspmm_b200 import sparse_matrix_format as smf
    names = ["config1_v8", "ffn_512x2048_s98_v8"]
    src, dest = tmp_path / "dlmc", tmp_path / "dlmc-v8"
    (src / "sub").mkdir(parents=True)
    listing = []
    for n in names:
        a, _ = CASES[n]
        rel = f"sub/{n}.smtx"
        svc_oracle.write_smtx(str(src / rel), a.M, a.K, a.nnz, a.row_ptr.tolist(), a.col_idx.tolist())
        listing.append(rel)
    (tmp_path / "paths.txt").write_text("\n".join(listing) + "\n")
    smf.generate_CVSE_file(str(src) + "/", str(dest) + "/", str(tmp_path / "paths.txt"), 8, csv_dir=str(tmp_path / "csv_data"))
    rows = list(csv.reader(open(tmp_path / "csv_data" / "RowMerge_V8.csv")))
    assert len(rows) == len(names)
    for i, n in enumerate(names):
        a, V = CASES[n]
        m, k, nnz, ptr, col = svc_oracle.read_smtx(str(dest / listing[i]))
        assert (m, k, nnz) == ((a.M + 7) // 8, a.K, a.nnz)
        assert ptr == GOLD[n + "/vec_row_ptr"].tolist() and col == GOLD[n + "/vec_colInd_list"].tolist()
        zero = int(GOLD[n + "/all_zero_vec_cnt"][0])
        exp = [str(i), str(a.M), str(a.K), str(a.nnz), str(svc_oracle.new_sparsity(8, a.M, a.K, a.nnz, zero)), str(zero)] + \
              [str(x) for x in GOLD[n + "/storage"].tolist()]
        assert rows[i] == exp


def test_svc_batch_equals_one_by_one(lib):
    """Several matrices of different shapes compressed in one stacked pass give exactly what separate
    calls give (and therefore what the reference gives)."""
    dev = torch.device("cuda:0")
    names = ["ragged_unsorted_v8", "powerlaw_4096_v8", "config1_v8", "ffn_512x2048_s98_v8"]
    mats = []
    for n in names:
        a, _ = CASES[n]
        mats.append((torch.from_numpy(a.row_ptr).to(dev), torch.from_numpy(a.col_idx).to(dev),
                     torch.from_numpy(a.values).to(dev), a.M, a.K))
    res, replayed = ops.svc_batch(mats, 8)
    assert replayed > 0
    for n, (p, c, v) in zip(names, res):
        a, _ = CASES[n]
        assert np.array_equal(p.cpu().numpy(), GOLD[n + "/vec_row_ptr"])
        assert np.array_equal(c.cpu().numpy(), GOLD[n + "/vec_colInd_list"])
        dense = svc_oracle.densify(p.numel() - 1, 8, a.K, p.cpu().tolist(), c.cpu().tolist(), v.cpu().numpy())
        assert np.array_equal(dense[: a.M].view(np.uint16), a.dense().view(np.uint16))


def test_reader_rows_take_the_array_path_through_the_python_entry_point(lib, tmp_path):
    """CVSE fed with the reader's row sequence (CSR arrays handed over without list conversion) equals CVSE fed
    with plain lists of lists, and both equal the oracle."""
    from sspmm_b200 import sparse_matrix_format as smf
    a = synthetic.power_law(3000, np.random.default_rng(77))
    p = str(tmp_path / "p.smtx")
    smf.write_smtx(p, a.M, a.K, a.nnz, a.row_ptr, a.col_idx)
    m = smf.sparse_matrix(p)
    fast = smf.CVSE(m.M, m.N, m.nnz, m.colInd_list_array(), 8)
    slow = smf.CVSE(a.M, a.K, a.nnz, a.row_lists(), 8)
    r = svc_oracle.cvse(a.M, a.K, a.nnz, a.row_lists(), 8)
    assert fast.vec_row_ptr == slow.vec_row_ptr == r.vec_row_ptr
    assert fast.vec_colInd_list == slow.vec_colInd_list == r.vec_colInd_list
    assert fast.tile_num == r.tile_num and fast.vec_colInd_list_array == r.vec_colInd_list_array
    assert fast.return_TCF_storage() == r.return_TCF_storage() and fast.return_SRBCSR_storage() == r.return_SRBCSR_storage()


def _one_group(K, lens, seed, repeat=0, order="ascending"):
    """A matrix of one vector row whose matrix rows have these lengths; `repeat`: so many columns of the longest row twice."""
    rng = np.random.default_rng(seed)
    rows = [rng.permutation(K)[:n] for n in lens]
    if order == "ascending":
        rows = [np.sort(r) for r in rows]
    if repeat:
        at = int(np.argmax(lens))
        rows[at] = rng.permutation(np.concatenate([rows[at], rows[at][:repeat]]))
    ptr = np.concatenate([[0], np.cumsum([r.size for r in rows])]).astype(np.int32)
    col = np.concatenate(rows).astype(np.int32)
    val = rng.uniform(-1, 1, K).astype(np.float16)[col]        # by column: which of two equal entries is kept makes no difference
    return synthetic.CSR(len(lens), K, ptr, col, val)


@pytest.mark.parametrize("order", ["ascending", "any"])
@pytest.mark.parametrize("K,big", [
    (140, 70), (600, 150), (600, 300), (2100, 400), (2100, 1220), (8300, 1300), (9000, 4900),            # tables of 128 to 8192 slots, wrapped a little
    (33000, 5000), (33903, 17900), (32900, 19600), (65536, 15000), (131072, 19650),                      # 32768 slots
    (131073, 19600), (140000, 9000), (262144, 19655),                                                    # 32768 slots, columns of 18 bits
    (140000, 21000), (200000, 78600)])                                                                   # tables in global memory
def test_replay_of_every_table_length(lib, K, big, order):
    """The long row first, in the middle and last: the sets of the rows after it are rebuilt from nearly the same sequence, and
    later rows bring nothing, few and many new columns."""
    for at, others in ((0, [1, 0, 3, 9, 2, 40, 5]), (3, [2, 7, 1, 60, 0, 2, 5]), (7, [3] * 7), (2, [30, big // 3, 8, big // 2, 0, 1, 4])):
        lens = others[:at] + [big] + others[at:]
        check_against_oracle(_one_group(K, lens, K + at, order=order), 8)
    check_against_oracle(_one_group(K, [big // 20] * 16, K + 1, order=order), 16)


@pytest.mark.parametrize("K,big", [(140, 60), (2100, 300), (2100, 1100), (9000, 4800), (33000, 17000), (140000, 18000), (140000, 21000)])
def test_replay_of_rows_that_repeat_columns(lib, K, big):
    for repeat in (1, 5):
        check_against_oracle(_one_group(K, [4, big, 3, 0, 6, 1, 2, 9], K + repeat, repeat=repeat), 8)
        check_against_oracle(_one_group(K, [4, 9, 3, big, 6], K + repeat, repeat=repeat), 8)


@pytest.mark.parametrize("u", [5, 19, 31, 32, 33, 64, 65, 76, 77, 97, 256, 257, 306, 307, 512, 513, 1228, 1229, 2600])
def test_replay_at_the_edges_of_batches(lib, u):
    """Sets around the sizes of a batch (32, 256 and 512 elements) and of the classes, ascending and not, without and with a column
    that its row repeats."""
    for order, repeat in (("ascending", 0), ("any", 0), ("any", 1)):
        for lens in ([u, 0, 1, 2], [2, 1, u - 3], [u // 2, u - u // 2, 0, 3]):
            check_against_oracle(_one_group(200000, lens, u, repeat=repeat, order=order), 8)


@pytest.mark.parametrize("count", [1, 60, 61])
def test_batches_around_the_table_of_a_launch(lib, count):
    """Up to 60 matrices travel with the launch, more are copied; with matrices of no rows and no entries, and without values."""
    dev, rng = torch.device("cuda:0"), np.random.default_rng(count)
    mats = []
    for i in range(count):
        m, k = (0 if i == 7 else 8 * int(rng.integers(1, 8))), int(rng.integers(50, 400))
        n = np.zeros(m, dtype=np.int64) if i == 9 else rng.integers(0, 30, m)
        ptr = np.concatenate([[0], np.cumsum(n)]).astype(np.int32)
        col = np.concatenate([np.sort(rng.permutation(k)[:x]) for x in n] + [np.zeros(0, dtype=np.int64)]).astype(np.int32)
        mats.append(tuple(torch.from_numpy(x).to(dev) for x in (ptr, col, rng.uniform(-1, 1, col.size).astype(np.float16))) + (m, k))
    for with_values in (True, False):
        given = [x if with_values else x[:2] + (None,) + x[3:] for x in mats]
        res, replayed = ops.svc_batch(given, 8)
        single = [ops.svc(*x, 8) for x in given]
        assert replayed == sum(x[3] for x in single)
        for got, want in zip(res, single):
            assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
            assert got[2] is None and want[2] is None if not with_values else torch.equal(got[2], want[2])


def test_value_vectors_off_their_boundary(lib):
    """The caller's value array need not start on a 16-byte boundary; nothing before or after it is written."""
    import ctypes as C
    a = _one_group(9000, [4, 2000, 3, 0, 60, 1, 2, 9] * 3, 5)
    dev = torch.device("cuda:0")
    d = [torch.from_numpy(x).to(dev) for x in (a.row_ptr, a.col_idx, a.values)]
    want = ops.svc(*d, a.M, a.K, 8)
    job, nvec, st = C.c_void_p(), C.c_int64(), torch.cuda.current_stream().cuda_stream
    assert lib.svc_begin(a.M, a.K, 8, d[0].data_ptr(), d[1].data_ptr(), d[2].data_ptr(), st, C.byref(job), C.byref(nvec)) == 0
    ptr, col = torch.empty(4, dtype=torch.int32, device=dev), torch.empty(nvec.value, dtype=torch.int32, device=dev)
    room = torch.full((nvec.value * 8 + 16,), 7.0, dtype=torch.float16, device=dev)
    assert lib.svc_finish(job, ptr.data_ptr(), col.data_ptr(), room.data_ptr() + 6, st) == 0
    lib.svc_free(job)
    assert torch.equal(ptr, want[0]) and torch.equal(col, want[1]) and torch.equal(room[3: 3 + want[2].numel()], want[2])
    assert (room[:3] == 7).all() and (room[3 + want[2].numel():] == 7).all()


@pytest.mark.parametrize("V", [8, 16])
@pytest.mark.parametrize("groups,K,most", [(296, 200, 150), (297, 200, 150), (300, 3000, 900), (2368, 40, 9), (2369, 40, 9)])
def test_svc_with_few_and_many_groups(lib, V, groups, K, most):
    """Both team sizes of the launches with a CTA per group, on 148 SMs: 296 groups and one more, 2368 and one more; a last group of
    one row, empty rows, ascending and replayed groups."""
    rng = np.random.default_rng(groups)
    rows = [np.sort(rng.permutation(K)[:n]) for n in rng.integers(0, most + 1, (groups - 1) * V + 1)]
    rows[3:7] = [r[:0] for r in rows[3:7]]
    ptr = np.concatenate([[0], np.cumsum([r.size for r in rows])]).astype(np.int32)
    col = np.concatenate(rows).astype(np.int32)
    check_against_oracle(synthetic.CSR(len(rows), K, ptr, col, rng.uniform(-1, 1, col.size).astype(np.float16)), V)


def test_svc_with_almost_two_to_the_31_entries(lib):
    """Entry numbers are 32-bit: the last group ends a hundred entries before 2^31, closer than one step of a team's loop."""
    if torch.cuda.mem_get_info()[0] < 48 << 30:
        pytest.skip("needs 30 GB on the device")
    K, rows, short = 16384, 131072, 100
    nnz = rows * K - short
    col = torch.arange(K, dtype=torch.int32, device="cuda:0").repeat(rows)[:nnz]
    val = torch.ones(nnz, dtype=torch.float16, device="cuda:0")
    ptr = torch.arange(0, rows, device="cuda:0") * K
    ptr = torch.cat([ptr, ptr.new_tensor([nnz])]).int()
    vec_ptr, vec_col, vec_val, _ = ops.svc(ptr, col, val, rows, K, 8)
    assert torch.equal(vec_ptr, torch.arange(0, rows // 8 + 1, device="cuda:0", dtype=torch.int32) * K)
    assert torch.equal(vec_col, col[: K].repeat(rows // 8))
    assert (vec_val[: -8 * K] == 1).all()
    last = vec_val[-8 * K:].view(K, 8)
    assert (last[:, :7] == 1).all() and (last[: K - short, 7] == 1).all() and not last[K - short:, 7].any()
