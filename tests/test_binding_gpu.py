"""The extension calls behind ops: which operands they take, and that the calls they leave to the checks in Python are
answered, or refused, as by those."""
import numpy as np
import pytest
import torch

from sspmm_b200 import capi, ops, synthetic
from sspmm_b200.sptrans.spmm import bspmm

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture(scope="module")
def product(lib):
    g = torch.Generator(device=DEV).manual_seed(1)
    mask = torch.rand((9, 40), device=DEV, generator=g) < 0.5
    ptr = torch.zeros(10, dtype=torch.int32, device=DEV)
    ptr[1:] = torch.cumsum(mask.sum(1), 0)
    col = mask.nonzero()[:, 1].int().contiguous()
    val = torch.randn(col.numel() * 8, device=DEV, generator=g).half()
    rhs = torch.randn(40, 24, device=DEV, generator=g).half()
    return ptr, col, val, rhs


def no_extension(m):
    """Every call goes through the checks in Python."""
    class Nothing:
        def __getattr__(self, name):
            return lambda *a: (capi.lib().sspmm_group_run(a[0], None) if name == "group_run" else False if name == "same_plain" else None)
    m.setattr(capi, "native", lambda: Nothing())


def test_plain_operands_are_taken_and_give_the_same(product, monkeypatch):
    ptr, col, val, rhs = product
    order = ops.sorted_row_swizzle(ptr)
    bias = torch.randn(72, device=DEV).half()
    plan = ops.Plan(ptr, col, 8, 40)
    n = capi.native()
    assert n.sspmm(ptr, col, val, rhs, 8, None, None, torch.float16) is not None
    assert n.same_plain(rhs, val) and not n.same_plain(rhs, rhs.t()) and not n.same_plain(rhs.cpu()) and not n.same_plain(rhs.view(-1)[1:])
    batch, vals = torch.stack([rhs, rhs + 1]), torch.stack([val, val * 2])
    csr = synthetic.power_law_device(300, 5, torch.device(DEV))
    calls = [lambda: ops.sspmm(ptr, col, val, rhs, 8), lambda: ops.sspmm(ptr, col, val, rhs, 8, row_indices=order, out_dtype=torch.float32),
             lambda: ops.sspmm_bias(ptr, col, val, rhs, 8, bias, order), lambda: ops.sspmm_planned(plan, val, rhs),
             lambda: ops.sspmm_planned(plan, val, rhs, out_dtype=torch.float32), lambda: bspmm(order, ptr, col, vals, batch, 8),
             lambda: bspmm(order, ptr, col, val, batch, 8), lambda: ops.sorted_row_swizzle(ptr),
             lambda: ops.svc(*csr, 300, 300, 8), lambda: ops.svc(csr[0], csr[1], None, 300, 300, 16)]
    got = [f() for f in calls]
    no_extension(monkeypatch)
    for f, g in zip(calls, got):
        want = f()
        for a, b in zip(g if isinstance(g, tuple) else (g,), want if isinstance(want, tuple) else (want,)):
            assert type(a) is type(b)
            if isinstance(a, torch.Tensor):
                assert a.dtype == b.dtype and a.device == b.device and not a.requires_grad and torch.equal(a, b)
            else:
                assert a == b


def test_what_was_refused_is_refused(product):
    ptr, col, val, rhs = product
    n = capi.native()
    bad = [((ptr.long(), col, val, rhs), TypeError), ((ptr, col, val.float(), rhs), TypeError), ((ptr, col, val, rhs.t()), ValueError),
           ((ptr.cpu(), col, val, rhs), ValueError), ((ptr, col, val, rhs.cpu()), ValueError), ((ptr, col[::2], val, rhs), ValueError)]
    for args, error in bad:
        assert n.sspmm(*args, 8, None, None, torch.float16) is None
        with pytest.raises(error):
            ops.sspmm(*args, 8)
    with pytest.raises(ValueError):
        ops.sspmm_bias(ptr, col, val, rhs, 8, torch.zeros(5, device=DEV).half())
    with pytest.raises(capi.SspmmError, match="vec_length"):
        ops.sspmm(ptr, col, val, rhs, 4)
    plan = ops.Plan(ptr, col, 8, 40)
    with pytest.raises(ValueError):
        ops.sspmm_planned(plan, val, rhs[:39])
    with pytest.raises(capi.SspmmError):
        ops.svc(ptr, col + 100, None, 9, 40, 8)
    out = torch.empty(72, 24, device=DEV).half()
    g = ops.Group([(plan, val, rhs, out)])
    g.close()
    with pytest.raises(capi.SspmmError, match="null group"):
        g.run()


def test_wrapped_tensors_and_modes_are_left_to_python(product):
    ptr, col, val, rhs = product
    want = ops.sspmm(ptr, col, val, rhs, 8)
    n, seen = capi.native(), []

    def inside(x):
        seen.append(n.sspmm(ptr, col, val, x, 8, None, None, torch.float16))
        return x
    torch.vmap(inside)(torch.stack([rhs, rhs]))
    torch.func.jvp(inside, (rhs,), (rhs,))
    with torch.device("cpu"):
        seen.append(n.sspmm(ptr, col, val, rhs, 8, None, None, torch.float16))
        assert torch.equal(ops.sspmm(ptr, col, val, rhs, 8), want)
    assert seen == [None] * 3
    s = torch.cuda.Stream()
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        got = ops.sspmm(ptr, col, val, torch.nn.Parameter(rhs), 8)
    s.synchronize()
    assert torch.equal(got, want) and not got.requires_grad


def test_stacked_operands(product):
    """Two operands one below the other against their products one by one, row orders included; what is not such a call is left alone."""
    ptr, col, val, rhs = product
    order, n = ops.sorted_row_swizzle(ptr), col.numel()
    ptr2 = torch.cat([ptr[:1], ptr[1:-1] - (ptr[1:-1] > 0).int(), ptr[-1:]])              # other row ends, the same columns
    cols, vals, bias = torch.cat([col, col]), torch.cat([val, val * 2]), torch.randn(144, device=DEV).half()
    call = lambda ptrs=(ptr, ptr2), orders=(order, order), ends=(n, 2 * n), c=cols, v=vals, r=rhs, V=8, b=bias: \
        ops.sspmm_stacked(list(ptrs), list(orders), list(ends), c, v, r, V, b)
    want = torch.cat([ops.sspmm_bias(ptr, col, val, rhs, 8, bias[:72], order), ops.sspmm_bias(ptr2, col, val * 2, rhs, 8, bias[72:], order)])
    assert torch.equal(call(), want)
    five = [ptr] * 5
    for other in (dict(ends=(n, 2 * n - 1)), dict(ends=(n + 1, n)), dict(ptrs=(ptr, ptr[:-1])), dict(orders=(order, order[:-1])), dict(c=cols[:-1]), dict(v=vals[8:]),
                  dict(r=rhs.float()), dict(r=rhs.t()), dict(r=rhs.cpu()), dict(b=bias[:-1]), dict(b=None), dict(ptrs=(ptr, ptr.long())), dict(r=rhs[:, :20].contiguous()),
                  dict(ptrs=five, orders=[order] * 5, ends=[n * i for i in range(1, 6)], c=col.repeat(5), v=val.repeat(5), b=bias[:72].repeat(5)), dict(ptrs=(), orders=(), ends=())):
        assert call(**other) is None
