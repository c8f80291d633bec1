"""Host-side checks of the encoder layer that launch nothing: which tensors its kernels are given at all."""
import pytest
import torch

from sspmm_b200 import encoder


@pytest.fixture
def launches(monkeypatch):
    """Every tensor counts as one the kernels can take, and launches are only counted."""
    made = []
    monkeypatch.setattr(encoder, "_plain", lambda *t: True)
    monkeypatch.setattr(encoder.ops, "launch_layer_norm_fm", lambda *a, **k: made.append(a))
    return made


def layer(hidden=8):
    L = encoder.SparseEncoderLayer.__new__(encoder.SparseEncoderLayer)
    L.hidden, L.ffn, L.heads, L.dev, L.linears = hidden, hidden, 1, torch.device("cpu"), []
    L.ln1 = L.ln2 = (torch.ones(hidden).half(), torch.zeros(hidden).half())
    return L


@pytest.mark.parametrize("tokens,room", [(16, 8), (8, 16), (64, 8)])
def test_norm_does_not_write_results_of_another_shape(launches, tokens, room):
    L, x, out = layer(), torch.randn(8, tokens).half(), torch.zeros(8, room).half()
    with pytest.raises(RuntimeError):
        L._norm(x, L.ln1, out=out)
    assert not launches and not out.any()


def test_norm_does_not_write_sums_of_another_shape(launches):
    L, x = layer(), torch.randn(8, 16).half()
    total, out = torch.zeros(8, 8).half(), torch.zeros(8, 16).half()
    L._norm(x, L.ln1, add=x, out=out, sum_out=total)
    assert not launches and not total.any() and out.any()
    L._norm(x, L.ln1, add=x, out=out, sum_out=torch.zeros(8, 16).half())
    assert len(launches) == 1


def test_norm_broadcasts_one_column_as_before(launches):
    L, x, out = layer(), torch.randn(8, 1).half(), torch.zeros(8, 8).half()
    L._norm(x, L.ln1, out=out)
    assert not launches and torch.equal(out, L._layer_norm_fm(x, L.ln1).expand(8, 8))


def test_norm_returns_what_was_normalised(launches):
    L, x, bias = layer(), torch.randn(8, 8).half(), torch.randn(8).half()
    was, _ = L._norm(x, L.ln1, bias=bias)
    assert torch.equal(was, x + bias[:, None])


def fm(*shape, dtype=torch.float16):
    return torch.zeros(shape, dtype=dtype)


@pytest.mark.parametrize("change,message", [
    ({"gamma": fm(7)}, "gamma has shape"), ({"beta": fm(8, 1)}, "beta has shape"), ({"out": fm(8, 8)}, "out has shape"),
    ({"add": fm(8, 8), "sum_out": fm(8, 16)}, "add has shape"), ({"add": fm(8, 16)}, "add needs sum_out"),
    ({"add": fm(8, 16), "sum_out": fm(16, 8)}, "sum_out has shape"), ({"bias": fm(9)}, "bias has shape"),
    ({"gamma": torch.empty(8, device="meta").half()}, "gamma is on")])
def test_layer_norm_rejects_operands_of_other_shapes(change, message):
    args = {"x": fm(8, 16), "gamma": fm(8), "beta": fm(8), "eps": 1e-5, "out": fm(8, 16), **change}
    # x itself is looked at first and is on the host here: give the others a chance
    with pytest.MonkeyPatch.context() as m:
        m.setattr(encoder.ops, "_require", lambda *a: None)
        m.setattr(encoder.ops.capi, "lib", lambda: pytest.fail("launched"))
        with pytest.raises(ValueError, match=message):
            encoder.ops.layer_norm_fm(**args)


@pytest.mark.parametrize("change,message", [
    ({"q": fm(128, 24)}, "q has shape"), ({"k": fm(64, 24)}, "k has shape"), ({"v": fm(128, 16)}, "v has shape"),
    ({"out": fm(128, 32)}, "out has shape"), ({"bias_q": fm(64)}, "bias_q has shape"), ({"bias_v": fm(128, 1)}, "bias_v has shape"),
    ({"heads": 1}, "q has shape"), ({"seq": 8}, "q has shape")])
def test_attention_rejects_operands_of_other_shapes(change, message):
    args = {"q": fm(128, 48), "k": fm(128, 48), "v": fm(128, 48), "heads": 2, "batch": 3, "seq": 16, "out": fm(128, 48), **change}
    with pytest.MonkeyPatch.context() as m:
        m.setattr(encoder.ops, "_require", lambda *a: None)
        m.setattr(encoder.ops.capi, "lib", lambda: pytest.fail("launched"))
        with pytest.raises(ValueError, match=message):
            encoder.ops.attention_fm(**args)


def test_feature_major_operators_reject_types_and_layouts():
    ops, x, w = encoder.ops, fm(8, 16), fm(8)
    with pytest.MonkeyPatch.context() as m:
        m.setattr(torch.Tensor, "is_cuda", True)
        m.setattr(ops.capi, "lib", lambda: pytest.fail("launched"))
        for bad, error in ((x.float(), TypeError), (fm(16, 8).t(), ValueError), (fm(8, 8), ValueError)):
            with pytest.raises(error):
                ops.add_bias_fm(x, w, bad)
            with pytest.raises(error):
                ops.layer_norm_fm(x, w, w, 1e-5, bad)
        for bad, error in ((w.float(), TypeError), (fm(16)[::2], ValueError), (fm(7), ValueError)):
            with pytest.raises(error):
                ops.add_bias_fm(x, bad, x)
            with pytest.raises(error):
                ops.layer_norm_fm(x, w, bad, 1e-5, x)
        q = fm(64, 16)
        for bad in (q.float(), fm(16, 64).t()):
            with pytest.raises((TypeError, ValueError)):
                ops.attention_fm(q, q, bad, 1, 1, 16, q)


def test_transformed_tensors_take_the_general_path(monkeypatch):
    """Products, LayerNorm and attention as framework operations carry tangents and batch dimensions; kernels drop them."""
    monkeypatch.setattr(torch.Tensor, "get_device", lambda t: 0)
    monkeypatch.setattr(encoder.ops, "launch_layer_norm_fm", lambda *a, **k: pytest.fail("launched"))
    monkeypatch.setattr(encoder.ops, "sspmm_bias", lambda *a, **k: pytest.fail("launched"))
    monkeypatch.setattr(encoder.ops, "sspmm", lambda *a, **k: torch.zeros(8, 16).half())
    L, x, t = layer(), torch.randn(8, 16).half(), torch.randn(8, 16).half()
    assert encoder._plain(x, t)
    general = lambda a: L._layer_norm_fm(a, L.ln1)
    assert torch.equal(torch.func.jvp(lambda a: L._norm(a, L.ln1)[1], (x,), (t,))[1], torch.func.jvp(general, (x,), (t,))[1])
    with torch.autograd.forward_ad.dual_level():
        y = L._norm(torch.autograd.forward_ad.make_dual(x, t), L.ln1)[1]
        assert torch.autograd.forward_ad.unpack_dual(y).tangent.any()
    xs = torch.stack([x, t])
    assert torch.equal(torch.vmap(lambda a: L._norm(a, L.ln1)[1])(xs), torch.vmap(general)(xs))
    lin = encoder.SparseLinear.__new__(encoder.SparseLinear)
    lin.out_features, lin.V = 8, 8
    lin.row_offsets = lin.col = lin.values = lin.row_indices = None

    def with_bias(b):
        lin.bias = b
        return lin(x)
    b, db = torch.randn(8).half(), torch.randn(8).half()
    assert torch.equal(torch.func.jvp(with_bias, (b,), (db,))[1], db[:, None].expand(8, 16))


def test_dense_evaluation_uses_none_of_the_kernels(monkeypatch):
    monkeypatch.setattr(encoder, "_plain", lambda *t: True)
    for name in ("launch_layer_norm_fm", "launch_attention_fm", "launch_add_bias_fm", "sspmm", "sspmm_bias"):
        monkeypatch.setattr(encoder.ops, name, lambda *a, **k: pytest.fail("launched"))
    L = layer(64)
    for _ in range(6):
        lin = encoder.SparseLinear.__new__(encoder.SparseLinear)
        lin.dense, lin.bias = torch.randn(64, 64).half() / 8, torch.randn(64).half()
        L.linears.append(lin)
    x = torch.randn(64, 48).half().requires_grad_()
    y = L.forward(x, 3, 16, dense=True)
    d = [(l.dense.double(), l.bias.double()[:, None]) for l in L.linears]
    norm = lambda t: (t - t.mean(0)) / torch.sqrt(t.var(0, unbiased=False) + 1e-5)
    n = norm(x.double())
    q, k, v = ((w @ n + b).view(64, 3, 16).permute(1, 2, 0) for w, b in d[:3])
    att = (torch.softmax(q @ k.transpose(1, 2) / 8, -1) @ v).permute(2, 0, 1).reshape(64, 48)
    out = d[3][0] @ att + d[3][1] + x.double()
    ref = d[5][0] @ (d[4][0] @ norm(out) + d[4][1]) + d[5][1] + out
    assert (y.double() - ref).norm() <= 4e-3 * ref.norm()            # eight roundings to fp16 of at most 2^-11 each
    y.sum().backward()
    assert x.grad is not None and x.grad.any()


class Linear:
    def __init__(self, plan):
        self.plan, self.values, self.bias = plan, torch.zeros(4).half(), None
        self.V, self.out_features = 8, 8


def test_groups_are_made_again_for_other_values_and_plans(monkeypatch):
    class Plan:
        one_launch = True
    made = []
    monkeypatch.setattr(encoder.ops, "Group", lambda products: made.append([p[1].data_ptr() for p in products]) or made[-1])
    L = layer()
    L.linears = [Linear(Plan()) for _ in range(6)]

    def bound():
        L._groups_for(8)
        return [a for g in L.groups for a in g]
    first = bound()
    assert bound() == first and len(made) == 4
    L.linears[3].values = torch.ones(4).half()
    assert bound() == [l.values.data_ptr() for l in L.linears] and len(made) == 8
    keep, L.linears[0].values.data = L.linears[0].values.data, torch.ones(4).half()
    assert bound() == [l.values.data_ptr() for l in L.linears] and len(made) == 12 and keep is not None
    L.linears[5].plan = Plan()
    bound()
    assert len(made) == 16
    L.linears[1].values.mul_(2)
    bound()
    assert len(made) == 16


def test_stacked_linears_leave_other_callables_alone():
    class Scaled(encoder.SparseLinear):
        def __call__(self, x):
            return 2 * super().__call__(x)
    stack = encoder.StackedLinears.__new__(encoder.StackedLinears)
    for other in (lambda x: x, Scaled.__new__(Scaled)):
        assert stack([other] * 3, fm(8, 8)) is None
