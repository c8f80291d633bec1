"""Encoder layer with pruned, SVC-compressed weights against the same layer evaluated with dense
matrices (torch.matmul on the densified pruned weights)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_sparse_encoder_layer_matches_dense_evaluation(lib):
    from sspmm_b200.encoder import SparseEncoderLayer
    torch.manual_seed(0)
    layer = SparseEncoderLayer(hidden=256, ffn=1024, heads=4, sparsity=0.9, vec_length=16)
    batch, seq = 4, 128
    x = torch.randn(256, batch * seq, device="cuda:0", dtype=torch.float16)
    y_sparse = layer.forward(x, batch, seq)
    y_dense = layer.forward(x, batch, seq, dense=True)
    torch.cuda.synchronize()
    assert y_sparse.shape == (256, batch * seq) and torch.isfinite(y_sparse).all()
    err = (y_sparse.float() - y_dense.float()).abs().max().item()
    scale = y_dense.float().abs().max().item()
    assert err <= 2e-2 * scale, (err, scale)
    rms = ((y_sparse.float() - y_dense.float()).pow(2).mean().sqrt() / y_dense.float().pow(2).mean().sqrt()).item()
    assert rms < 5e-3


@pytest.mark.parametrize("hidden,tokens", [(64, 8), (3072, 40), (256, 4768), (100, 9600)])
def test_layer_norm_feature_major(lib, hidden, tokens):
    """Both tile widths, a partial tile, the largest and an odd number of features; the bound is the rounding of the result
    (2^-11 of it) and of the fp32 statistics (a few 2^-22 of the spread)."""
    from sspmm_b200 import ops
    g = torch.Generator(device="cuda:0").manual_seed(hidden + tokens)
    r = lambda *s: torch.randn(s, device="cuda:0", generator=g).half()
    x, add, gamma, beta = r(hidden, tokens) * 3 + 1, r(hidden, tokens), r(hidden), r(hidden)
    for a, bias in ((None, None), (add, None), (add, beta + 1), (None, gamma)):
        out, total = torch.empty_like(x), torch.empty_like(x)
        ops.layer_norm_fm(x, gamma, beta, 1e-5, out, a, total if a is not None else None, bias)
        s = x if bias is None else x + bias[:, None]
        s = s if a is None else s + a
        if a is not None:
            assert torch.equal(total, s)
        d = s.double()
        ref = (d - d.mean(0)) / torch.sqrt(d.var(0, unbiased=False) + 1e-5) * gamma.double()[:, None] + beta.double()[:, None]
        assert ((out.double() - ref).abs() <= 2.0 ** -11 * ref.abs() + 2.0 ** -19 * (1 + gamma.double().abs()[:, None] * 4)).all()


@pytest.mark.parametrize("heads,batch,seq,scale", [(1, 1, 8, 1.0), (2, 3, 64, 1.0), (4, 2, 72, 3.0), (1, 2, 512, 6.0), (3, 1, 200, 0.1)])
def test_attention_feature_major(lib, heads, batch, seq, scale):
    """One key block and several, partial blocks, flat and peaked probabilities.  Bound: rounding of the fp16 result, and the
    fp32 scores (2^-20 of their size, at most 64 * 8 * scale^2 / 8 times, enters a probability relatively)."""
    from sspmm_b200 import ops
    g = torch.Generator(device="cuda:0").manual_seed(seq)
    r = lambda s: (torch.randn((heads * 64, batch * seq), device="cuda:0", generator=g) * s).half()
    q, k, v = r(scale), r(scale), r(1.0)
    bq, bk, bv = (torch.randn(heads * 64, device="cuda:0", generator=g).half() for _ in range(3))
    out, with_bias = torch.full_like(q, float("nan")), torch.full_like(q, float("nan"))
    ops.attention_fm(q, k, v, heads, batch, seq, out)
    ops.attention_fm(q, k, v, heads, batch, seq, with_bias, bq, bv)
    split = lambda t: t.double().view(heads, 64, batch, seq).permute(2, 0, 3, 1)
    # the bias of v is added to the finished sum, so |v| and |bias| enter the bound separately
    for got, dq, dk, dv, mag in ((out, q.double(), k.double(), v.double(), v.double().abs()),
                                 (with_bias, (q + bq[:, None]).double(), k.double() + bk.double()[:, None],
                                  v.double() + bv.double()[:, None], v.double().abs() + bv.double().abs()[:, None])):
        score = split(dq) @ split(dk).transpose(-1, -2) / 8
        p = torch.softmax(score, -1)
        ref = p @ split(dv)
        slack = 2.0 ** -20 * (1 + score.abs().amax()) * (p @ split(mag))
        assert ((split(got) - ref).abs() <= 2.0 ** -11 * ref.abs() + 2.0 ** -24 + slack).all()


def test_bias_and_residual_feature_major(lib):
    from sspmm_b200 import ops
    x, add = (torch.randn(33, 72, device="cuda:0").half() for _ in range(2))
    bias = torch.randn(33, device="cuda:0").half()
    assert torch.equal(ops.add_bias_fm(x, bias, add), x + bias[:, None] + add)


def test_grouped_layer_follows_replaced_bias_and_odd_shapes(lib):
    from sspmm_b200.encoder import SparseEncoderLayer
    layer = SparseEncoderLayer(hidden=256, ffn=1024, heads=4, sparsity=0.9, vec_length=16)
    for batch, seq in ((2, 72), (3, 20), (1, 13)):                # the last two are outside what the fused parts take
        x = torch.randn(256, batch * seq, device="cuda:0", dtype=torch.float16)
        for _ in range(2):
            if (batch * seq) % 8 == 0:
                a, b = layer.forward(x, batch, seq), layer.forward_grouped(x, batch, seq)
                assert (a.float() - b.float()).abs().max() <= 1e-2 * a.float().abs().max()
            c, d = layer.forward(x, batch, seq), layer.forward(x, batch, seq, dense=True)
            assert (c.float() - d.float()).abs().max() <= 2e-2 * d.float().abs().max()
            layer.linears[0].bias = layer.linears[0].bias + 1.0
            layer.linears[4].bias = layer.linears[4].bias + 0.5
            layer.linears[5].bias = layer.linears[5].bias - 2.0


@pytest.mark.parametrize("seq,scale", [(64, 0.0), (64, 1.0), (136, 1.0), (200, 0.5)])
def test_attention_infinities_and_nans(lib, seq, scale):
    """An infinite value times any probability is infinite (all of these are above 2^-60), two of opposite sign and a NaN give
    NaN, other features and sequences keep their numbers; a query whose scores are all -inf has no softmax.  scale 0: every
    probability is a power of two and its low term zero.  Bound of the numbers: see test_attention_feature_major."""
    from sspmm_b200 import ops
    heads, batch = 2, 2
    g = torch.Generator(device="cuda:0").manual_seed(seq)
    r = lambda s: (torch.randn((heads * 64, batch * seq), device="cuda:0", generator=g) * s).half()
    q, k, v = r(scale), r(scale), r(1.0)
    inf = float("inf")
    v[3, 5], v[10, seq - 1], v[70, 0], v[90, 1], v[90, seq - 2], v[127, seq + 7] = inf, -inf, inf, inf, -inf, float("nan")
    q[64, seq + 9], k[64, seq:] = inf, -1.0            # sequence 1, head 1, query 9: every score is -inf
    if scale == 0:
        k[64:, seq:] = -1.0                             # equal scores for the other queries as well
    out = torch.full_like(q, float("nan"))
    ops.attention_fm(q, k, v, heads, batch, seq, out)
    split = lambda t: t.double().view(heads, 64, batch, seq).permute(2, 0, 3, 1)
    score = split(q) @ split(k).transpose(-1, -2) / 8
    p = torch.softmax(score, -1)
    ref, got = p @ split(v), split(out)
    assert torch.equal(ref.isnan(), got.isnan()) and torch.equal(ref.isposinf(), got.isposinf()) and torch.equal(ref.isneginf(), got.isneginf())
    assert ref.isinf().any() and ref.isnan().any()
    fin = ref.isfinite()
    top = score[score.isfinite()].abs().amax()
    slack = 2.0 ** -20 * (1 + top) * (p @ split(v).abs())
    assert ((got - ref).abs()[fin] <= (2.0 ** -11 * ref.abs() + 2.0 ** -24 + slack)[fin]).all()


def test_attention_sums_have_no_drift(lib):
    """Values of one sign: truncated additions would pull every result the same way.  A block of 64 keys adds eight times to
    a sum that starts at zero, each time losing at most 2^-23 of it; over half a million results the rounding to fp16
    (2^-11 / sqrt(12) of a result at most) averages out to 2^-11 / sqrt(12 n), four of which are allowed."""
    from sspmm_b200 import ops
    heads, batch, seq = 2, 2, 2048
    g = torch.Generator(device="cuda:0").manual_seed(0)
    q, k = ((torch.randn(heads * 64, batch * seq, device="cuda:0", generator=g) * 0.5).half() for _ in range(2))
    v = (torch.rand(heads * 64, batch * seq, device="cuda:0", generator=g) + 1).half()
    out = torch.empty_like(q)
    ops.attention_fm(q, k, v, heads, batch, seq, out)
    split = lambda t: t.double().view(heads, 64, batch, seq).permute(2, 0, 3, 1)
    ref = torch.softmax(split(q) @ split(k).transpose(-1, -2) / 8, -1) @ split(v)
    drift = (split(out) / ref - 1).mean().abs().item()
    assert drift <= 8 * 2.0 ** -23 + 4 * 2.0 ** -11 / (12 * out.numel()) ** 0.5


def exact_layer(layer, x, batch, seq):
    """The layer in 64 bits, from its dense weights."""
    lin = [(l.dense.double(), 0 if l.bias is None else l.bias.double()[:, None]) for l in layer.linears]

    def norm(t, wb):
        return (t - t.mean(0)) / torch.sqrt(t.var(0, unbiased=False) + 1e-5) * wb[0].double()[:, None] + wb[1].double()[:, None]
    x = x.double()
    n = norm(x, layer.ln1)
    q, k, v = ((w @ n + b).view(layer.heads, -1, batch, seq).permute(2, 0, 3, 1) for w, b in lin[:3])
    att = torch.softmax(q @ k.transpose(-1, -2) / q.shape[-1] ** 0.5, -1) @ v
    out = lin[3][0] @ att.permute(1, 3, 0, 2).reshape(x.shape) + lin[3][1] + x
    return lin[5][0] @ (lin[4][0] @ norm(out, layer.ln2) + lin[4][1]) + lin[5][1] + out


@pytest.mark.parametrize("hidden,heads,batch,seq", [(256, 4, 3, 72), (128, 2, 1, 200), (128, 4, 2, 64), (256, 4, 2, 20)])
def test_layer_against_64_bits(lib, hidden, heads, batch, seq):
    """Heads, sequences, residuals and biases end up where they belong (head width 32 and sequences that are not a multiple of
    eight take the framework's attention).  An activation is rounded to fp16 at most a dozen times on the way, each time by at
    most 2^-11 of its norm, and the layer's parts pass a relative error on without raising it."""
    from sspmm_b200.encoder import SparseEncoderLayer
    layer = SparseEncoderLayer(hidden=hidden, ffn=4 * hidden, heads=heads, sparsity=0.9, vec_length=16)
    g = torch.Generator(device="cuda:0").manual_seed(hidden + seq)
    r = lambda *s: torch.randn(s, device="cuda:0", generator=g)
    layer.ln1, layer.ln2 = ((r(hidden) * 0.3 + 1).half(), r(hidden).half()), ((r(hidden) * 0.3 - 1).half(), r(hidden).half())
    for l in layer.linears:
        l.bias = r(l.out_features).half()
    x = (r(hidden, batch * seq) * 2 + 0.5).half()
    ref = exact_layer(layer, x, batch, seq)
    for got in (layer.forward(x, batch, seq), layer.forward_grouped(x, batch, seq), layer.forward(x, batch, seq, dense=True)):
        assert got.shape == x.shape and (got.double() - ref).norm() <= 12 * 2.0 ** -11 * ref.norm()


def test_layer_under_autograd_takes_framework_operations(lib):
    """With a bias that wants a gradient the sums, LayerNorm and attention are recorded, and the numbers are the same."""
    from sspmm_b200.encoder import SparseEncoderLayer
    layer = SparseEncoderLayer(hidden=128, ffn=512, heads=2, sparsity=0.9, vec_length=16)
    x = torch.randn(128, 144, device="cuda:0", dtype=torch.float16)
    plain = layer.forward(x, 2, 72)
    layer.linears[5].bias.requires_grad_()
    y = layer.forward(x, 2, 72)
    assert (y - plain).norm() <= 12 * 2.0 ** -11 * plain.norm()
    y.sum().backward()
    assert torch.equal(layer.linears[5].bias.grad, torch.full((128,), 144.0, device="cuda:0").half())


def test_grouped_layer_refuses_other_token_counts(lib):
    from sspmm_b200.encoder import SparseEncoderLayer
    layer = SparseEncoderLayer(hidden=128, ffn=512, heads=2, sparsity=0.9, vec_length=16)
    x = torch.randn(128, 144, device="cuda:0", dtype=torch.float16)
    y = layer.forward_grouped(x, 2, 72).clone()
    before = {n: t.clone() for n, t in layer.buf.items()}
    for other in (x[:, :136].contiguous(), torch.cat([x, x], 1)):
        with pytest.raises(RuntimeError):
            layer.forward_grouped(other, 2, 72)
    assert all(torch.equal(before[n].view(torch.int16), t.view(torch.int16)) for n, t in layer.buf.items())
    assert torch.equal(y, layer.forward_grouped(x, 2, 72))


def test_layer_norm_wide_tile_with_most_features(lib):
    """32 tokens per CTA and 3072 features: all of the shared memory it may ask for; bound as in test_layer_norm_feature_major."""
    from sspmm_b200 import ops
    x = torch.randn(3072, 32 * 148 + 8, device="cuda:0").half()
    w, b, out = torch.randn(3072, device="cuda:0").half(), torch.randn(3072, device="cuda:0").half(), torch.empty_like(x)
    ops.layer_norm_fm(x, w, b, 1e-5, out)
    d = x.double()
    ref = (d - d.mean(0)) / torch.sqrt(d.var(0, unbiased=False) + 1e-5) * w.double()[:, None] + b.double()[:, None]
    assert ((out.double() - ref).abs() <= 2.0 ** -11 * ref.abs() + 2.0 ** -19 * (1 + w.double().abs()[:, None] * 4)).all()


@pytest.mark.parametrize("tokens", [40, 16 * 148 + 8, 32 * 148 + 8])
@pytest.mark.parametrize("hidden", [1, 127, 129, 256, 257, 512, 513, 768, 1000, 1024, 1025, 3072])
def test_layer_norm_with_features_in_registers(lib, hidden, tokens):
    """8, 16 and 32 tokens per CTA on 148 SMs: every number of features per thread, its edges, the first that goes through shared memory,
    and a partly filled tile; then the result in place of the operand.  Bound as in test_layer_norm_feature_major."""
    from sspmm_b200 import ops
    test_layer_norm_feature_major(lib, hidden, tokens)
    x, w = torch.randn(hidden, tokens, device="cuda:0").half(), torch.ones(hidden, device="cuda:0").half()
    out = torch.empty_like(x)
    ops.layer_norm_fm(x, w, w, 1e-5, out)
    ops.layer_norm_fm(x, w, w, 1e-5, x)
    assert torch.equal(out, x)


@pytest.mark.parametrize("M,K,N,V,sparsity,kernel", [
    (64, 64, 8, 8, 0.5, 0), (256, 1024, 128, 16, 0.9, 0), (200, 300, 72, 8, 0.9, 0), (768, 3072, 200, 16, 0.95, 0),     # rows by warps
    (256, 512, 128, 8, 0.9, 3), (136, 520, 264, 8, 0.5, 3), (768, 3072, 128, 16, 0.9, 3),                             # tiles, K cut or not
    (768, 3072, 8192, 16, 0.9, 0), (272, 640, 19000, 16, 0.9, 3)])                                                    # CTA pairs, a half empty one
def test_product_plus_a_matrix(lib, M, K, N, V, sparsity, kernel):
    """Against the same product with fp32 results: the sum is rounded once, and the fp32 sums of two launches differ by 1e-5 of the
    operands' sizes at most (order of the parts, truncation of the tensor unit over K <= 3072)."""
    from sspmm_b200 import ops, synthetic
    w = synthetic.magnitude_pruned(M, K, sparsity, np.random.default_rng(M + N))
    d = lambda a: torch.from_numpy(a).to("cuda:0")
    ptr, col, val, _ = ops.svc(d(w.row_ptr), d(w.col_idx), d(w.values), M, K, V)
    rows = (ptr.numel() - 1) * V
    g = torch.Generator(device="cuda:0").manual_seed(N)
    r = lambda *s: torch.randn(s, device="cuda:0", generator=g).half()
    rhs, add, bias, order = r(K, N), r(rows, N) * 4, r(rows), ops.sorted_row_swizzle(ptr)
    ops.set_kernel(kernel)
    try:
        got = ops.sspmm_sum(ptr, col, val, rhs, V, bias, order, add)
        want = ops.sspmm_bias(ptr, col, val, rhs, V, bias, row_indices=order, out_dtype=torch.float32).double() + add.double()
    finally:
        ops.set_kernel(0)
    assert got is not None and got.dtype == torch.float16
    assert ((got.double() - want).abs() <= 2.0 ** -11 * want.abs() + 1e-5 * (1 + want.abs().max())).all()
    if kernel == 0 and K <= 1024:
        plan = ops.Plan(ptr, col, V, K)
        group = ops.Group([(plan, val, rhs, torch.full((rows, N), 7.0, device="cuda:0", dtype=torch.float16))])
        if plan.one_launch and group.run_sum(None, add) is not None:
            assert torch.equal(group.run_sum(bias, add), got) or N % 64            # the same division, or another tile width
            assert (group._keep[0][3] == 7).all()
    assert ops.sspmm_sum(ptr, col, val, rhs, V, bias, order, add[:, : N - 8]) is None
    assert ops.sspmm_sum(ptr, col, val, rhs, V, bias, order, add.float()) is None


@pytest.mark.parametrize("V,N,shapes", [(8, 264, [(64, 64), (136, 1300), (512, 100)]), (16, 136, [(768, 3072), (48, 1024), (16, 8), (3072, 768)]),
                                        (16, 8192, [(768, 3072), (256, 1040)])])
def test_products_of_copies_made_by_one_launch(lib, V, N, shapes):
    """Rows and chunks of several operands in one launch, one of them three pieces: bit by bit the product that makes its own copy."""
    from sspmm_b200 import ops, synthetic
    d = lambda a: torch.from_numpy(a).to("cuda:0")
    g = torch.Generator(device="cuda:0").manual_seed(N)
    r = lambda *s: torch.randn(s, device="cuda:0", generator=g).half()
    operands, products = [], []
    for i, (M, K) in enumerate(shapes):
        pieces = [ops.svc(d(w.row_ptr), d(w.col_idx), d(w.values), M, K, V)
                  for w in (synthetic.magnitude_pruned(M, K, 0.8, np.random.default_rng(M + K + x)) for x in range(3 if i == 0 else 1))]
        ends = torch.cumsum(torch.tensor([p[1].numel() for p in pieces]), 0).tolist()
        col, val = torch.cat([p[1] for p in pieces]), torch.cat([p[2] for p in pieces])
        operands.append(([p[0] for p in pieces], ends, col, val, V, K))
        products.append((pieces, r(K, N), r(len(pieces) * (pieces[0][0].numel() - 1) * V)))
    ops.set_kernel(3)
    try:
        copies = ops.dense_copies(operands, N)
        assert all(c is not None and c.data_ptr() % 256 == 0 for c in copies)
        for copy, (pieces, rhs, bias) in zip(copies, products):
            rows = bias.numel() // len(pieces)
            got = ops.of_copy(copy, rhs, V, bias)
            for i, (ptr, col, val, _) in enumerate(pieces):
                dense = copy[:, i * rows: (i + 1) * rows].contiguous()
                own = ops.sspmm_bias(ptr, col, val, rhs, V, bias[i * rows: (i + 1) * rows].contiguous())
                one = ops.of_copy(dense, rhs, V, bias[i * rows: (i + 1) * rows].contiguous())
                assert torch.equal(one, own)
                assert (got[i * rows: (i + 1) * rows].double() - own.double()).norm() <= 2 * 2.0 ** -11 * own.double().norm()
                if len(pieces) == 1:
                    assert torch.equal(got, own)
    finally:
        ops.set_kernel(0)
    assert ops.dense_copies([([torch.tensor([0, 1], device="cuda:0", dtype=torch.int32)], [1], *[t[:n].contiguous() for t, n in
                            ((products[0][0][0][1], 1), (products[0][0][0][2], V))], V, 64)], 512) == [None]


@pytest.mark.parametrize("hidden,tokens", [(256, 640), (512, 2400), (768, 2408), (768, 4744), (1088, 4744)])
def test_layer_norm_beside_copies(lib, hidden, tokens):
    """One launch for both, at every tile width, and two where the tile goes through shared memory: bit by bit the launches of their own."""
    from sspmm_b200 import ops, synthetic
    d = lambda a: torch.from_numpy(a).to("cuda:0")
    w = synthetic.magnitude_pruned(512, 1500, 0.8, np.random.default_rng(hidden))
    ptr, col, val, _ = ops.svc(d(w.row_ptr), d(w.col_idx), d(w.values), 512, 1500, 16)
    operands = [([ptr], [col.numel()], col, val, 16, 1500)] * 2
    x, g, b = torch.randn(hidden, tokens, device="cuda:0").half(), torch.randn(hidden, device="cuda:0").half(), torch.randn(hidden, device="cuda:0").half()
    want = torch.empty_like(x)
    ops.layer_norm_fm(x, g, b, 1e-5, want)
    ops.set_kernel(3)
    try:
        one, two, norm = ops.dense_copies(operands, tokens, (x, g, b, 1e-5))
        alone, _ = ops.dense_copies(operands, tokens)
    finally:
        ops.set_kernel(0)
    assert torch.equal(norm, want) and torch.equal(one, alone) and torch.equal(two, alone)


def test_layer_of_copies_is_the_layer(lib, monkeypatch):
    """The same layer with every product making its own copy, and one whose linears were replaced."""
    from sspmm_b200.encoder import SparseEncoderLayer
    layer = SparseEncoderLayer(hidden=512, ffn=2048, heads=8, sparsity=0.9, vec_length=16)
    x = torch.randn(512, 4096, device="cuda:0", dtype=torch.float16)
    copies, norm = layer._copies(x)
    assert all(c is not None for c in copies) and layer._copies(x[:, :64].contiguous()) == ([None] * 4, None)
    assert torch.equal(norm, layer._norm(x, layer.ln1)[1])
    y = layer.forward(x, 8, 512)
    layer.linears[4].values.mul_(2)
    scaled = layer.forward(x, 8, 512)
    layer.linears[4].values.div_(2)
    monkeypatch.setattr(layer, "_copies", lambda x: ([None] * 4, None))
    assert torch.equal(y, layer.forward(x, 8, 512)) and not torch.equal(y, scaled)
    monkeypatch.undo()
    own = layer.linears[5]
    layer.linears[5] = lambda a: own(a)
    assert layer._copies(x) == ([None] * 4, None)
    assert (layer.forward(x, 8, 512).double() - y.double()).norm() <= 4 * 2.0 ** -11 * y.double().norm()


def test_stacked_linears_follow_their_tensors(lib):
    """Q, K and V as one product: values and biases changed in place count, and so do tensors put in their place."""
    from sspmm_b200.encoder import SparseEncoderLayer
    layer = SparseEncoderLayer(hidden=128, ffn=512, heads=2, sparsity=0.9, vec_length=16)
    x = torch.randn(128, 144, device="cuda:0", dtype=torch.float16)
    L = layer.linears[:3]

    def check(taken):
        got = layer.qkv(L, x)
        assert (got is not None) == taken
        for y, l in zip(got or [], L):
            assert (y.double() - l(x).double()).norm() <= 2 * 2.0 ** -11 * y.double().norm() and y.is_contiguous()
        y = layer.forward(x, 2, 72)
        qkv, layer.qkv = layer.qkv, None
        want = layer.forward(x, 2, 72)
        layer.qkv = qkv
        assert (y.double() - want.double()).norm() <= 12 * 2.0 ** -11 * want.double().norm()
    check(True)
    L[1].values.mul_(2.0)
    L[2].bias.add_(1.0)
    check(True)
    L[0].bias = L[0].bias + 1.0
    check(False)
    L[0].bias = layer.qkv.bias[:128]
    check(True)
    L[2].values = L[2].values * 0.5
    check(False)
    L[2].values = layer.qkv.values[-L[2].values.numel():]
    L[1].bias.requires_grad_()
    check(False)


@pytest.mark.parametrize("hidden,tokens", [(128, 144), (256, 16384)])
def test_stacked_linears_follow_row_pointers_changed_in_place(lib, hidden, tokens):
    """The first row loses its last vector to the second, once with and once without torch noticing; row-gather and block kernel.
    The stacked product and the linear's own round the same sums, taken in another order, to fp16."""
    from sspmm_b200.encoder import SparseEncoderLayer
    layer = SparseEncoderLayer(hidden=hidden, ffn=4 * hidden, heads=hidden // 64, sparsity=0.9, vec_length=16)
    x = torch.randn(hidden, tokens, device="cuda:0", dtype=torch.float16)
    L = layer.linears[:3]
    l, end = L[0], int(L[0].row_offsets[1])
    free = sorted(set(range(hidden)) - set(l.col[: int(l.row_offsets[2])].tolist()))
    l.col[end - 2: end] = torch.tensor(free[:2], dtype=torch.int32, device="cuda:0")       # columns that neither row names
    before = layer.qkv(L, x)[0].clone()
    for change in (lambda t: t[1].sub_(1), lambda t: t.data[1].sub_(1)):
        change(l.row_offsets)
        got = layer.qkv(L, x)
        for y, own in zip(got, L):
            want = own(x).double()
            assert (y.double() - want).norm() <= 2 * 2.0 ** -11 * want.norm()
        assert (before[:32].double() - got[0][:32].double()).norm() > 0.05 * before[:32].double().norm()


def test_plans_of_stacked_linears_read_the_stacked_columns(lib):
    from sspmm_b200.encoder import SparseEncoderLayer
    layer = SparseEncoderLayer(hidden=128, ffn=512, heads=2, sparsity=0.9, vec_length=16)
    for l in layer.linears:
        assert l.plan.column_indices.data_ptr() == l.col.data_ptr() and l.plan.row_offsets is l.row_offsets and l.plan.one_launch


@pytest.mark.parametrize("tokens", [512, 768, 1024, 1536, 2048, 2560, 3072, 4096])
def test_stacked_linears_keep_infinities_where_their_rows_name_them(lib, tokens):
    """Token counts around the one from which the dense-tile kernel, which multiplies an infinity by zeros that are in no list, is the
    faster one for three products, and the one from which it is for one: NaN and infinity come out as from the products one by one."""
    from sspmm_b200.encoder import SparseEncoderLayer
    layer = SparseEncoderLayer(hidden=512, ffn=512, heads=8, sparsity=0.9, vec_length=16)
    x = torch.randn(512, tokens, device="cuda:0", dtype=torch.float16)
    x[3, 5], x[100, tokens - 1] = float("inf"), -float("inf")
    got = layer.qkv(layer.linears[:3], x)
    for y, l in zip(got or [], layer.linears):
        want = l(x)
        assert torch.equal(y.isnan(), want.isnan()) and torch.equal(y.isposinf(), want.isposinf()) and torch.equal(y.isneginf(), want.isneginf())
    assert got is not None


@pytest.mark.parametrize("heads,batch,seq,scale", [(3, 75, 72, 3.0), (2, 112, 120, 1.0), (4, 56, 128, 1.0), (2, 40, 136, 0.1), (1, 80, 200, 1.0),
                                                   (3, 3, 512, 6.0), (1, 10, 1928, 1.0), (8, 40, 64, 1.0)])
def test_attention_with_many_tiles(lib, heads, batch, seq, scale):
    """Enough tiles of 128 queries and blocks of keys for the tcgen05 kernel: two blocks, three stages and more, half tiles, sequences
    that end inside a block; one block, however many tiles, stays with the other kernel."""
    test_attention_feature_major(lib, heads, batch, seq, scale)


@pytest.mark.parametrize("seq,scale", [(72, 0.0), (136, 1.0), (200, 0.5)])
def test_attention_infinities_and_nans_with_many_tiles(lib, seq, scale):
    """As test_attention_infinities_and_nans, in some of the tiles of the tcgen05 kernel."""
    from sspmm_b200 import ops
    heads, batch, inf = 2, 112, float("inf")
    g = torch.Generator(device="cuda:0").manual_seed(seq)
    r = lambda s: (torch.randn((heads * 64, batch * seq), device="cuda:0", generator=g) * s).half()
    q, k, v = r(scale), r(scale), r(1.0)
    v[3, 5], v[10, seq - 1], v[70, 0], v[90, 1], v[90, seq - 2], v[127, seq + 7] = inf, -inf, inf, inf, -inf, float("nan")
    q[64, seq + 9], k[64, seq: 2 * seq] = inf, -1.0
    out = torch.full_like(q, float("nan"))
    ops.attention_fm(q, k, v, heads, batch, seq, out)
    split = lambda t: t.double().view(heads, 64, batch, seq).permute(2, 0, 3, 1)
    score = split(q) @ split(k).transpose(-1, -2) / 8
    p = torch.softmax(score, -1)
    ref, got = p @ split(v), split(out)
    assert torch.equal(ref.isnan(), got.isnan()) and torch.equal(ref.isposinf(), got.isposinf()) and torch.equal(ref.isneginf(), got.isneginf())
    assert ref.isinf().any() and ref.isnan().any()
    fin = ref.isfinite()
    slack = 2.0 ** -20 * (1 + score[score.isfinite()].abs().amax()) * (p @ split(v).abs())
    assert ((got - ref).abs()[fin] <= (2.0 ** -11 * ref.abs() + 2.0 ** -24 + slack)[fin]).all()


@pytest.mark.parametrize("batch,seq", [(2, 72), (112, 136)])
@pytest.mark.parametrize("finite", [True, False])
def test_attention_into_its_queries(lib, batch, seq, finite):
    """The result may take the queries' place, also where a tile is done twice because something infinite or NaN went in."""
    from sspmm_b200 import ops
    g = torch.Generator(device="cuda:0").manual_seed(seq)
    q, k, v = (torch.randn(128, batch * seq, device="cuda:0", generator=g).half() for _ in range(3))
    if not finite:
        v[3, 5], v[70, seq - 1], v[90, 1] = float("inf"), -float("inf"), float("nan")
    out = torch.empty_like(q)
    ops.attention_fm(q, k, v, 2, batch, seq, out)
    ops.attention_fm(q, k, v, 2, batch, seq, q)
    assert torch.equal(q.view(torch.int16), out.view(torch.int16))


def attend_by(lib, kernel, q, k, v, heads, batch, seq, biases=(None, None)):
    import ctypes as C
    out, taken = torch.full_like(q, float("nan")), C.c_int()
    rc = lib.sspmm_attention_fm_as(kernel, heads, 64, batch, seq, q.data_ptr(), k.data_ptr(), v.data_ptr(),
                                   *(None if b is None else b.data_ptr() for b in biases), out.data_ptr(),
                                   torch.cuda.current_stream().cuda_stream, C.byref(taken))
    assert rc == 0
    return out, taken.value


@pytest.mark.parametrize("heads,batch,seq,tc", [(8, 40, 64, False), (1, 1, 512, False), (3, 75, 72, True), (2, 120, 120, True), (4, 60, 128, True),
                                                (1, 80, 200, True), (3, 3, 512, None), (1, 10, 1928, True)])
def test_attention_takes_the_kernel_of_its_size(lib, heads, batch, seq, tc):
    """Two thirds of the SMs times the blocks of keys after the first decide; the sizes are 3 % or more from the line of 148 SMs."""
    q, k, v = (torch.randn(heads * 64, batch * seq, device="cuda:0").half() for _ in range(3))
    out, taken = attend_by(lib, 0, q, k, v, heads, batch, seq)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert taken == (2 if 2 * -(-seq // 128) * heads * batch * ((seq - 1) // 64) >= 3 * sms else 1)
    assert tc is None or sms != 148 or taken == (2 if tc else 1)
    assert torch.equal(out, attend_by(lib, taken, q, k, v, heads, batch, seq)[0])


@pytest.mark.parametrize("kernel", [1, 2])
@pytest.mark.parametrize("heads,batch,seq,scale,finite", [(1, 1, 8, 1.0, True), (2, 3, 64, 1.0, True), (4, 2, 72, 3.0, True), (1, 2, 136, 6.0, True),
                                                          (3, 1, 200, 0.1, True), (2, 1, 520, 1.0, True), (2, 2, 72, 1.0, False), (2, 3, 328, 0.5, False)])
def test_attention_by_either_kernel(lib, kernel, heads, batch, seq, scale, finite):
    """The same operands through both kernels, at sizes that the choice gives to one of them only; infinities and NaNs come out as in
    the plain formula.  Bound: see test_attention_feature_major."""
    g = torch.Generator(device="cuda:0").manual_seed(seq)
    r = lambda s: (torch.randn((heads * 64, batch * seq), device="cuda:0", generator=g) * s).half()
    q, k, v = r(scale), r(scale), r(1.0)
    bq, bv = (torch.randn(heads * 64, device="cuda:0", generator=g).half() for _ in range(2))
    if not finite:
        inf = float("inf")
        v[3, 5], v[10, seq - 1], v[70, 0], v[90, 1], v[90, seq - 2], v[127, seq + 7] = inf, -inf, inf, inf, -inf, float("nan")
    out, taken = attend_by(lib, kernel, q, k, v, heads, batch, seq, (bq, bv))
    assert taken == kernel
    split = lambda t: t.double().view(heads, 64, batch, seq).permute(2, 0, 3, 1)
    score = split(q + bq[:, None]) @ split(k).transpose(-1, -2) / 8
    p = torch.softmax(score, -1)
    ref, got = p @ split(v) + bv.double().view(heads, 64)[None, :, None, :], split(out)
    assert torch.equal(ref.isnan(), got.isnan()) and torch.equal(ref.isposinf(), got.isposinf()) and torch.equal(ref.isneginf(), got.isneginf())
    fin = ref.isfinite()
    slack = 2.0 ** -20 * (1 + score.abs().amax()) * (p @ split(v).abs() + bv.double().abs().view(heads, 64)[None, :, None, :])
    assert ((got - ref).abs()[fin] <= (2.0 ** -11 * ref.abs() + 2.0 ** -24 + slack)[fin]).all()
