"""Host-side checks of the encoder layer that launch nothing: which tensors its kernels are given at all."""
import pytest
import torch

from sspmm_b200 import encoder


@pytest.fixture
def launches(monkeypatch):
    """Every tensor counts as one the kernels can take, and launches are only counted."""
    made = []
    monkeypatch.setattr(encoder, "_plain", lambda *t: True)
    monkeypatch.setattr(encoder.ops, "layer_norm_fm", lambda *a, **k: made.append(a))
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
