"""Device-side operators on torch CUDA tensors.  torch is used for device
memory and streams only; every computation is a call into libsspmm_b200.so."""
from __future__ import annotations

from typing import Optional, Tuple

import torch

from . import capi

# KERNEL_GATHER: TMA row gather; KERNEL_GATHER_LSU: the row-gather kernel whose warps gather by themselves
KERNEL_AUTO, KERNEL_GATHER, KERNEL_SIMT, KERNEL_BLOCK, KERNEL_GATHER_LSU, KERNEL_BLOCK_SINGLE = 0, 1, 2, 3, 4, 5


def _stream_ptr() -> int:
    return torch.cuda.current_stream().cuda_stream


def _ptr(t: Optional[torch.Tensor]) -> Optional[int]:
    return None if t is None else t.data_ptr()


def _launch(fn, like: torch.Tensor, *args) -> None:
    """fn(*args, stream) on the device of ``like``; switching devices costs more than asking for the current one."""
    if torch.cuda.current_device() == like.get_device():
        capi.check(fn(*args, _stream_ptr()))
    else:
        with torch.cuda.device(like.device):
            capi.check(fn(*args, _stream_ptr()))


def _require(t: torch.Tensor, dtype, name: str) -> None:
    if not t.is_cuda:
        raise ValueError(f"{name} must be a CUDA tensor (there is no CPU path)")
    if t.dtype != dtype:
        raise TypeError(f"{name} must be {dtype}, got {t.dtype}")
    if not t.is_contiguous():
        raise ValueError(f"{name} must be contiguous")


def set_kernel(which: int) -> None:
    capi.check(capi.lib().sspmm_set_kernel(which))


def device_status() -> int:
    import ctypes as C
    s = C.c_int(0)
    capi.check(capi.lib().sspmm_device_status(C.byref(s)))
    return s.value


def sspmm(row_offsets: torch.Tensor, column_indices: torch.Tensor, values: torch.Tensor, rhs: torch.Tensor,
          vec_length: int, row_indices: Optional[torch.Tensor] = None, out_dtype=torch.float16,
          out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """C[m_vec*V, N] = A_vs @ rhs[K, N] (the call made at SSpMM/sspmm_test.cpp:189)."""
    return sspmm_bias(row_offsets, column_indices, values, rhs, vec_length, None, row_indices, out_dtype, out)


def _made(got):
    """What an extension call returned: a tensor, or an error code of the library."""
    if type(got) is int:
        capi.check(got)
    return got


def sspmm_bias(row_offsets: torch.Tensor, column_indices: torch.Tensor, values: torch.Tensor, rhs: torch.Tensor,
               vec_length: int, bias: Optional[torch.Tensor], row_indices: Optional[torch.Tensor] = None,
               out_dtype=torch.float16, out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """``sspmm`` plus a number per output row (fp16, m_vec*V of them), added to the fp32 sums before the conversion."""
    if out is None:
        got = capi.native().sspmm(row_offsets, column_indices, values, rhs, vec_length, bias, row_indices, out_dtype)
        if got is not None:
            return _made(got)
    _require(row_offsets, torch.int32, "row_offsets")
    _require(column_indices, torch.int32, "column_indices")
    _require(values, torch.float16, "values")
    _require(rhs, torch.float16, "rhs")
    if row_indices is not None:
        _require(row_indices, torch.int32, "row_indices")
    m_vec = row_offsets.numel() - 1
    if bias is not None:
        _require(bias, torch.float16, "bias")
        if bias.numel() != m_vec * vec_length:
            raise ValueError(f"bias has {bias.numel()} numbers, the product {m_vec * vec_length} rows")
        if bias.device != rhs.device:
            raise ValueError(f"bias is on {bias.device}, rhs on {rhs.device}")
    K, N = rhs.shape
    if out is None:
        out = torch.empty((m_vec * vec_length, N), dtype=out_dtype, device=rhs.device)
    fn = capi.lib().sspmm_counted
    args = (m_vec, vec_length, N, K, 1, column_indices.numel(), _ptr(row_indices), row_offsets.data_ptr(), column_indices.data_ptr(),
            values.data_ptr(), 0, rhs.data_ptr(), 0, _ptr(bias), out.data_ptr(), 0, 1 if out.dtype == torch.float16 else 0)
    if torch.cuda.current_device() == rhs.device.index:
        rc = fn(*args, _stream_ptr())
    else:
        with torch.cuda.device(rhs.device):
            rc = fn(*args, _stream_ptr())
    if rc != 0:
        capi.check(rc)
    return out


def sspmm_sum(row_offsets, column_indices, values, rhs, vec_length: int, bias, row_indices, add) -> Optional[torch.Tensor]:
    """``sspmm_bias`` with a matrix like the result added to the fp32 sums before they are rounded (``sspmm_counted_sum``), or None
    when the sum has to be made from the product's result."""
    got = capi.native().sspmm_sum(row_offsets, column_indices, values, rhs, vec_length, bias, row_indices, add)
    return None if got is None else _made(got)


def dense_copies(operands, N: int, norm=None):
    """The dense copies that the block kernel works on, of operands whose products with N columns are still to come, by one launch
    (``sspmm_dense_copies``).  ``operands``: (list of row offsets, where their vectors end, column_indices, values, vec_length, K).  A copy or
    None (the product does not work on one) for each; None: not operands for it.  ``norm``: (x, gamma, beta, eps), compared by the
    caller; where there is a copy its LayerNorm is made by the same launch and follows the copies."""
    got = capi.native().dense_copies(operands, N, *((None, None, None, 0.0) if norm is None else norm))
    return None if got is None else _made(got)


def of_copy(copy: torch.Tensor, rhs: torch.Tensor, vec_length: int, bias: torch.Tensor, add: Optional[torch.Tensor] = None) -> Optional[torch.Tensor]:
    """The product of an operand's copy and rhs, plus bias and ``add`` (``sspmm_of_copy``); None: not tensors for it."""
    got = capi.native().of_copy(copy, rhs, vec_length, bias, add)
    return None if got is None else _made(got)


def sspmm_stacked(row_offsets, row_indices, ends, column_indices: torch.Tensor, values: torch.Tensor, rhs: torch.Tensor, vec_length: int,
                  bias: torch.Tensor) -> Optional[torch.Tensor]:
    """Operands of one shape, their vectors one after another up to ``ends``, times the same rhs as one product (``sspmm_stacked``):
    results one below the other, or None when they have to be multiplied one by one.  ``row_offsets`` and ``row_indices`` are lists."""
    got = capi.native().stacked(row_offsets, row_indices, ends, column_indices, values, rhs, vec_length, bias)
    return None if got is None else _made(got)


def svc(row_ptr: torch.Tensor, col_idx: torch.Tensor, values: Optional[torch.Tensor], M: int, K: int,
        vec_length: int) -> Tuple[torch.Tensor, torch.Tensor, Optional[torch.Tensor], int]:
    """Sparse vector compression of a CSR matrix held on the GPU.
    Returns (vec_row_ptr[m_vec+1], vec_col[nvec], vec_values[nvec*V] or None, replayed_rows)."""
    import ctypes as C
    got = capi.native().svc(row_ptr, col_idx, values, M, K, vec_length)
    if got is not None:
        return _made(got)
    _require(row_ptr, torch.int32, "row_ptr")
    _require(col_idx, torch.int32, "col_idx")
    if values is not None:
        _require(values, torch.float16, "values")
    dev = row_ptr.device
    m_vec = (M + vec_length - 1) // vec_length
    job = C.c_void_p()
    nvec = C.c_int64(0)
    lib = capi.lib()
    with torch.cuda.device(dev):
        st = _stream_ptr()
        capi.check(lib.svc_begin(M, K, vec_length, row_ptr.data_ptr(), col_idx.data_ptr(), _ptr(values), st,
                                 C.byref(job), C.byref(nvec)))
        try:
            n = nvec.value
            vec_ptr = torch.empty(m_vec + 1, dtype=torch.int32, device=dev)
            vec_col = torch.empty(n, dtype=torch.int32, device=dev)
            vec_val = torch.empty(n * vec_length, dtype=torch.float16, device=dev) if values is not None else None
            replayed = C.c_int64(0)
            capi.check(lib.svc_replayed_rows(job, C.byref(replayed)))
            capi.check(lib.svc_finish(job, vec_ptr.data_ptr(), vec_col.data_ptr(), _ptr(vec_val), st))
        finally:
            lib.svc_free(job)
    return vec_ptr, vec_col, vec_val, replayed.value


def svc_batch(mats, vec_length: int, nnz=None):
    """Sparse vector compression of several independent CSR matrices in one pass (``svc_batch_begin`` /
    ``svc_batch_finish``): the matrices are stacked on the device and compressed together.

    ``mats`` is a list of (row_ptr, col_idx, values_or_None, M, K) with device tensors; ``nnz`` the list of
    their non-zero counts (taken from ``col_idx.numel()`` when omitted).  Returns a list of
    (vec_row_ptr, vec_col, vec_values_or_None) per matrix -- views into three buffers that hold all matrices
    one after another -- and the total number of replayed vector rows."""
    import ctypes as C
    if not mats:
        return [], 0
    got = capi.native().svc_batch(mats, vec_length, nnz)
    if got is not None:
        return _made(got)
    V = vec_length
    n = len(mats)
    dev = mats[0][0].device
    with_vals = all(m[2] is not None for m in mats)
    if nnz is None:
        nnz = [int(m[1].numel()) for m in mats]
    for (rp, ci, va, M, K) in mats:
        _require(rp, torch.int32, "row_ptr")
        _require(ci, torch.int32, "col_idx")
        if with_vals:
            _require(va, torch.float16, "values")
    Ms = (C.c_int * n)(*[m[3] for m in mats])
    Ks = (C.c_int * n)(*[m[4] for m in mats])
    Zs = (C.c_int * n)(*nnz)
    p_ptr = (C.c_void_p * n)(*[m[0].data_ptr() for m in mats])
    p_col = (C.c_void_p * n)(*[m[1].data_ptr() for m in mats])
    p_val = (C.c_void_p * n)(*[m[2].data_ptr() for m in mats]) if with_vals else None
    nvec = (C.c_int64 * n)()
    job = C.c_void_p()
    lib = capi.lib()
    with torch.cuda.device(dev):
        st = _stream_ptr()
        capi.check(lib.svc_batch_begin(n, V, Ms, Ks, Zs, p_ptr, p_col, p_val, st, C.byref(job), nvec))
        try:
            replayed = C.c_int64(0)
            capi.check(lib.svc_batch_replayed_rows(job, C.byref(replayed)))
            m_vecs = [(m[3] + V - 1) // V for m in mats]
            total_vec = sum(nvec)
            vec_ptr = torch.empty(sum(m_vecs) + n, dtype=torch.int32, device=dev)
            vec_col = torch.empty(total_vec, dtype=torch.int32, device=dev)
            vec_val = torch.empty(total_vec * V, dtype=torch.float16, device=dev) if with_vals else None
            capi.check(lib.svc_batch_finish(job, vec_ptr.data_ptr(), vec_col.data_ptr(), _ptr(vec_val), st))
        finally:
            lib.svc_batch_free(job)
    out, po, vo = [], 0, 0
    for k in range(n):
        nv = nvec[k]
        out.append((vec_ptr[po: po + m_vecs[k] + 1], vec_col[vo: vo + nv], None if vec_val is None else vec_val[vo * V: (vo + nv) * V]))
        po += m_vecs[k] + 1
        vo += nv
    return out, replayed.value


def sorted_row_swizzle(row_offsets: torch.Tensor) -> torch.Tensor:
    got = capi.native().sorted_row_swizzle(row_offsets)
    if got is not None:
        return _made(got)
    _require(row_offsets, torch.int32, "row_offsets")
    m_vec = row_offsets.numel() - 1
    out = torch.empty(m_vec, dtype=torch.int32, device=row_offsets.device)
    with torch.cuda.device(row_offsets.device):
        capi.check(capi.lib().sspmm_sorted_row_swizzle(m_vec, row_offsets.data_ptr(), out.data_ptr(), _stream_ptr()))
    return out


def _require_fm(t: torch.Tensor, shape, like: torch.Tensor, name: str) -> None:
    """An operand of the feature-major operators: the kernels see only its address."""
    if tuple(t.shape) != tuple(shape):
        raise ValueError(f"{name} has shape {tuple(t.shape)}, not {tuple(shape)}")
    if t.device != like.device:
        raise ValueError(f"{name} is on {t.device}, not {like.device}")
    _require(t, torch.float16, name)


def layer_norm_fm(x: torch.Tensor, gamma: torch.Tensor, beta: torch.Tensor, eps: float, out: torch.Tensor,
                  add: Optional[torch.Tensor] = None, sum_out: Optional[torch.Tensor] = None,
                  bias: Optional[torch.Tensor] = None) -> None:
    """LayerNorm over dim 0 of x[hidden, tokens] + bias + add (that sum goes to ``sum_out``), ``sspmm_layer_norm_fm``."""
    hidden, tokens = x.shape
    if add is not None and sum_out is None:
        raise ValueError("add needs sum_out")
    for t, shape, name in ((x, x.shape, "x"), (gamma, (hidden,), "gamma"), (beta, (hidden,), "beta"), (bias, (hidden,), "bias"),
                           (add, x.shape, "add"), (sum_out, x.shape, "sum_out"), (out, x.shape, "out")):
        if t is not None:
            _require_fm(t, shape, x, name)
    launch_layer_norm_fm(x, gamma, beta, eps, out, add, sum_out, bias)


def launch_layer_norm_fm(x, gamma, beta, eps, out, add, sum_out, bias) -> None:
    """``layer_norm_fm`` for a caller that has compared the operands itself."""
    rc = capi.native().layer_norm_fm(x, gamma, beta, eps, out, add, sum_out, bias)
    if rc is not None:
        return capi.check(rc)
    _launch(capi.lib().sspmm_layer_norm_fm, x, x.shape[0], x.shape[1], x.data_ptr(), _ptr(bias), _ptr(add), _ptr(sum_out),
            gamma.data_ptr(), beta.data_ptr(), eps, out.data_ptr())


def add_bias_fm(x: torch.Tensor, bias: torch.Tensor, add: torch.Tensor) -> torch.Tensor:
    """x[rows, tokens] + bias[:, None] + add, ``sspmm_add_bias_fm``."""
    rows, tokens = x.shape
    for t, shape, name in ((x, x.shape, "x"), (bias, (rows,), "bias"), (add, x.shape, "add")):
        _require_fm(t, shape, x, name)
    return launch_add_bias_fm(x, bias, add)


def launch_add_bias_fm(x, bias, add) -> torch.Tensor:
    """``add_bias_fm`` for a caller that has compared the operands itself."""
    out = torch.empty_like(x)
    rc = capi.native().add_bias_fm(x, bias, add, out)
    if rc is not None:
        capi.check(rc)
        return out
    _launch(capi.lib().sspmm_add_bias_fm, x, x.shape[0], x.shape[1], x.data_ptr(), bias.data_ptr(), add.data_ptr(), out.data_ptr())
    return out


def attention_fm(q: torch.Tensor, k: torch.Tensor, v: torch.Tensor, heads: int, batch: int, seq: int, out: torch.Tensor,
                 bias_q: Optional[torch.Tensor] = None, bias_v: Optional[torch.Tensor] = None) -> None:
    """Softmax attention of heads 64 wide on feature-major q, k, v [64 * heads, batch * seq], ``sspmm_attention_fm``."""
    hidden = 64 * heads
    for t, shape, name in ((q, (hidden, batch * seq), "q"), (k, (hidden, batch * seq), "k"), (v, (hidden, batch * seq), "v"),
                           (out, (hidden, batch * seq), "out"), (bias_q, (hidden,), "bias_q"), (bias_v, (hidden,), "bias_v")):
        if t is not None:
            _require_fm(t, shape, q, name)
    launch_attention_fm(q, k, v, heads, batch, seq, out, bias_q, bias_v)


def launch_attention_fm(q, k, v, heads, batch, seq, out, bias_q, bias_v) -> None:
    """``attention_fm`` for a caller that has compared the operands itself."""
    rc = capi.native().attention_fm(q, k, v, heads, batch, seq, out, bias_q, bias_v)
    if rc is not None:
        return capi.check(rc)
    _launch(capi.lib().sspmm_attention_fm, q, heads, 64, batch, seq, q.data_ptr(), k.data_ptr(), v.data_ptr(), _ptr(bias_q), _ptr(bias_v),
            out.data_ptr())


class Plan:
    """Ahead-of-time part of the SpMM for one weight structure (``sspmm_plan_create``): with it the product runs
    as one kernel launch straight from the compressed operand, without scratch, allocation or host
    synchronisation.  Keeps ``row_offsets`` and ``column_indices`` alive; the values may change between calls."""

    def __init__(self, row_offsets: torch.Tensor, column_indices: torch.Tensor, vec_length: int, K: int):
        import ctypes as C
        _require(row_offsets, torch.int32, "row_offsets")
        _require(column_indices, torch.int32, "column_indices")
        self.row_offsets, self.column_indices = row_offsets, column_indices
        self.V, self.K = vec_length, K
        self.m_vec = row_offsets.numel() - 1
        self.device = row_offsets.device
        self._h = C.c_void_p()
        with torch.cuda.device(self.device):
            capi.check(capi.lib().sspmm_plan_create(self.m_vec, vec_length, K, row_offsets.data_ptr(),
                                                    column_indices.data_ptr(), _stream_ptr(), C.byref(self._h)))
        nvec, one, asc, nbytes = C.c_int64(), C.c_int(), C.c_int(), C.c_int64()
        capi.check(capi.lib().sspmm_plan_info(self._h, C.byref(nvec), C.byref(one), C.byref(asc), C.byref(nbytes)))
        self.nvec, self.one_launch, self.ascending, self.device_bytes = nvec.value, bool(one.value), bool(asc.value), nbytes.value

    @property
    def handle(self):
        return self._h

    def close(self) -> None:
        if self._h:
            capi.lib().sspmm_plan_destroy(self._h)
            self._h = None

    def __del__(self):
        try:
            self.close()
        except Exception:
            pass


def sspmm_planned(plan: Plan, values: torch.Tensor, rhs: torch.Tensor, out_dtype=torch.float16,
                  out: Optional[torch.Tensor] = None) -> torch.Tensor:
    """C = A_vs @ rhs through ``sspmm_planned``: one launch, nothing allocated by the library."""
    if out is None and plan.handle:
        got = capi.native().planned(plan.handle.value, plan.m_vec * plan.V, plan.K, values, rhs, out_dtype)
        if got is not None:
            return _made(got)
    _require(values, torch.float16, "values")
    _require(rhs, torch.float16, "rhs")
    K, N = rhs.shape
    if K != plan.K:
        raise ValueError(f"rhs has {K} rows, the plan was built for K = {plan.K}")
    if out is None:
        out = torch.empty((plan.m_vec * plan.V, N), dtype=out_dtype, device=rhs.device)
    with torch.cuda.device(rhs.device):
        rc = capi.lib().sspmm_planned(plan.handle, values.data_ptr(), rhs.data_ptr(), out.data_ptr(), N,
                                      1 if out.dtype == torch.float16 else 0, _stream_ptr())
    if rc != 0:
        capi.check(rc)
    return out


class Group:
    """Several products bound to their operands and run as ONE persistent launch (``sspmm_group_create`` /
    ``sspmm_group_run``).  ``products`` is a list of (plan, values, rhs, out); all outputs share one dtype.
    ``mode``: COMPRESSED builds the A tiles inside the kernel from the compressed operand (no scratch for A),
    EXPANDED lets the kernel's loader warps write dense copies of A while the first tiles are multiplied (faster per
    K step), PAIRS is EXPANDED with 256 x 256 tiles on CTA pairs, AUTO picks COMPRESSED or EXPANDED by a model of their
    times, or the row-gather kernel for small groups.  Every mode is one launch per run."""

    AUTO, COMPRESSED, EXPANDED, PAIRS = 0, 1, 2, 3

    def __init__(self, products, mode: int = 0):
        import ctypes as C
        if not products:
            raise ValueError("a group needs at least one product")
        self._keep, self._biases = list(products), {}
        out_dtype = products[0][3].dtype
        arr = (capi.GroupItem * len(products))()
        for i, (plan, values, rhs, out) in enumerate(products):
            _require(values, torch.float16, "values")
            _require(rhs, torch.float16, "rhs")
            _require(out, out_dtype, "out")
            if rhs.shape[0] != plan.K or tuple(out.shape) != (plan.m_vec * plan.V, rhs.shape[1]):
                raise ValueError(f"product {i}: operand shapes do not match the plan")
            arr[i] = capi.GroupItem(plan.handle, values.data_ptr(), rhs.data_ptr(), out.data_ptr(), rhs.shape[1])
        self.device = products[0][2].device
        self._h = C.c_void_p()
        with torch.cuda.device(self.device):
            capi.check(capi.lib().sspmm_group_create(arr, len(products), 1 if out_dtype == torch.float16 else 0, mode, C.byref(self._h)))
        bn, items, ctas, launches, nbytes = C.c_int(), C.c_int(), C.c_int(), C.c_int(), C.c_int64()
        capi.check(capi.lib().sspmm_group_info(self._h, C.byref(bn), C.byref(items), C.byref(ctas), C.byref(launches), C.byref(nbytes)))
        self.tile_columns, self.work_items, self.ctas, self.scratch_bytes = bn.value, items.value, ctas.value, nbytes.value
        self.launches = launches.value

    def bias(self, item: int, bias: Optional[torch.Tensor]) -> bool:
        """Adds a number per output row (fp16) of a product before its results are rounded, from the next run on; False: this
        group's kernel does not, and nothing has changed."""
        import ctypes as C
        if bias is not None:
            _require(bias, torch.float16, "bias")
            out = self._keep[item][3]
            if bias.numel() != out.shape[0] or bias.device != out.device:
                raise ValueError(f"bias has {bias.numel()} numbers on {bias.device}, the product {out.shape[0]} rows on {out.device}")
        taken = C.c_int(0)
        capi.check(capi.lib().sspmm_group_bias(self._h, item, _ptr(bias), C.byref(taken)))
        if taken.value:
            self._biases[item] = bias
        return bool(taken.value)

    def run_sum(self, bias: Optional[torch.Tensor], add: torch.Tensor) -> Optional[torch.Tensor]:
        """A run of a group of one product whose result, with this bias and ``add`` added before it is rounded, goes to a new tensor;
        None: this group's kernel does not do that, or ``add`` is not like the output, and nothing was launched."""
        out = self._keep[0][3]
        if not self._h or len(self._keep) != 1 or add.shape != out.shape or add.device != out.device:
            return None
        got = capi.native().group_run_sum(self._h.value, out.shape[0], bias, add)
        return None if got is None else _made(got)

    def run(self) -> None:
        rc = capi.native().group_run(self._h.value if self._h else 0, self.device.index)
        if rc:
            capi.check(rc)

    def close(self) -> None:
        if self._h:
            capi.lib().sspmm_group_destroy(self._h)
            self._h = None

    def __del__(self):
        try:
            self.close()
        except Exception:
            pass


def workspace_bytes(m_vec: int, vec_length: int, N: int, K: int, nvec: int, out_is_f16: bool = True) -> int:
    """Scratch ``sspmm_ws`` would like for these sizes (``sspmm_workspace_bytes``)."""
    import ctypes as C
    b = C.c_int64(0)
    capi.check(capi.lib().sspmm_workspace_bytes(m_vec, vec_length, N, K, nvec, 1 if out_is_f16 else 0, C.byref(b)))
    return b.value


def sspmm_ws(row_offsets: torch.Tensor, column_indices: torch.Tensor, values: torch.Tensor, rhs: torch.Tensor,
             vec_length: int, nvec: int, workspace: Optional[torch.Tensor], out: Optional[torch.Tensor] = None,
             row_indices: Optional[torch.Tensor] = None) -> torch.Tensor:
    """C = A_vs @ rhs through ``sspmm_f16_f16_ws``: the caller passes the vector count and owns the scratch, so the
    library reads nothing back, allocates nothing and never synchronises."""
    m_vec = row_offsets.numel() - 1
    K, N = rhs.shape
    if out is None:
        out = torch.empty((m_vec * vec_length, N), dtype=torch.float16, device=rhs.device)
    ws_ptr = workspace.data_ptr() if workspace is not None else None
    ws_bytes = workspace.numel() * workspace.element_size() if workspace is not None else 0
    with torch.cuda.device(rhs.device):
        rc = capi.lib().sspmm_f16_f16_ws(m_vec, vec_length, N, K, _ptr(row_indices), row_offsets.data_ptr(),
                                         column_indices.data_ptr(), values.data_ptr(), rhs.data_ptr(), out.data_ptr(),
                                         nvec, ws_ptr, ws_bytes, _stream_ptr())
    if rc != 0:
        capi.check(rc)
    return out
