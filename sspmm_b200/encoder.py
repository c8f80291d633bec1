"""Transformer encoder layer whose six weight matrices (Q, K, V, O, FFN1, FFN2) are magnitude-pruned,
compressed by the GPU SVC and applied with the vector-sparse SpMM.  LayerNorm, attention and the last residual sum
are kernels of this package for contiguous fp16 activations with heads 64 wide and whole multiples of eight
tokens, and PyTorch operations otherwise, as in the dense evaluation.

Block structure follows the reference's end-to-end script (end2end/sspmm_e2e/end_to_end.py:44-75:
LayerNorm -> attention -> residual -> LayerNorm -> linear1 -> linear2 -> residual, no activation
between the two linears), with the sparsity moved from the attention mask to the weights.

Activations are kept feature-major, x[features, tokens], because the SpMM computes
C[out_features, tokens] = W_vs[out_features, in_features] . B[in_features, tokens] with B row-major."""
from __future__ import annotations

from typing import Optional

import numpy as np
import torch
import torch.nn.functional as F
from torch.autograd import forward_ad

from . import capi, ops, synthetic


def _plain(*tensors) -> bool:
    """Tensors the kernels can take as they lie: contiguous fp16 on one GPU, 16-byte aligned, outside autograd, function
    transforms and forward-mode differentiation (a dual tensor has an address too, and no requires_grad)."""
    if torch._C._functorch.peek_interpreter_stack() is not None or forward_ad._current_level >= 0:
        return False
    if capi.native().same_plain(*tensors):
        return True
    gpu = tensors[0].get_device()
    return gpu >= 0 and all(t.get_device() == gpu and t.dtype == torch.float16 and t.is_contiguous() and t.data_ptr() % 16 == 0
               and not (t.requires_grad and torch.is_grad_enabled()) for t in tensors)


class SparseLinear:
    """y[out, tokens] = W_vs . x[in, tokens] + b, W pruned and held in the compressed format."""

    def __init__(self, weight: synthetic.CSR, vec_length: int, device, bias: Optional[torch.Tensor] = None):
        self.out_features, self.in_features, self.V = weight.M, weight.K, vec_length
        self.nnz = weight.nnz
        d = lambda a: torch.from_numpy(a).to(device)
        self.row_offsets, self.col, self.values, _ = ops.svc(d(weight.row_ptr), d(weight.col_idx), d(weight.values),
                                                             weight.M, weight.K, vec_length)
        self.row_indices = ops.sorted_row_swizzle(self.row_offsets)
        self.plan = ops.Plan(self.row_offsets, self.col, vec_length, weight.K)
        self.bias = bias
        self.dense = torch.from_numpy(weight.dense()).to(device)          # only for the dense comparison

    def bias_rows(self) -> Optional[torch.Tensor]:
        """The bias as the product's epilogue takes it, one number per row of the padded output; None: not of that form."""
        b = self.bias
        if b is None or not _plain(b) or tuple(b.shape) != (self.out_features,):
            return None
        pad = -self.out_features % self.V
        return F.pad(b, (0, pad)) if pad else b

    def of_copy(self, copy: Optional[torch.Tensor], x: torch.Tensor, add: Optional[torch.Tensor] = None) -> Optional[torch.Tensor]:
        """``self(x)``, plus ``add``, from the dense copy of this linear that ``_copies`` made for this call; None: there is none, or
        these are not tensors for it."""
        rows = None if copy is None or not (_plain(x) if add is None else _plain(x, add)) else self.bias_rows()
        return None if rows is None else ops.of_copy(copy, x, self.V, rows, add)

    def __call__(self, x: torch.Tensor) -> torch.Tensor:
        rows = self.bias_rows()
        if rows is not None:
            return ops.sspmm_bias(self.row_offsets, self.col, self.values, x, self.V, rows, row_indices=self.row_indices)[: self.out_features]
        y = ops.sspmm(self.row_offsets, self.col, self.values, x, self.V, row_indices=self.row_indices)
        y = y[: self.out_features]
        return y if self.bias is None else y + self.bias[:, None]

    def plus(self, x: torch.Tensor, add: torch.Tensor) -> torch.Tensor:
        """``self(x) + add``, rounded once where the product's kernel adds it to its sums."""
        rows = self.bias_rows() if self.out_features % self.V == 0 and _plain(x, add) else None
        got = None
        if rows is not None:
            got = ops.sspmm_sum(self.row_offsets, self.col, self.values, x, self.V, rows, self.row_indices, add)
        return self(x) + add if got is None else got

    def dense_forward(self, x: torch.Tensor) -> torch.Tensor:
        y = self.dense @ x
        return y if self.bias is None else y + self.bias[:, None]


class StackedLinears:
    """Linears of one shape that read the same activations, as one product: their compressed operands one below the other.
    Values, column ids and biases are stored once, each linear's being views of them; the row pointers stay the linears' own.
    Three of 768 x 768 on 16384 tokens: 92 us one after another (three dense copies, 3 x 192 tiles in 3 x 3 rounds), 59 as one."""

    def __init__(self, linears):
        first = linears[0]
        self.V, self.rows, self.ends = first.V, first.out_features, [0]
        for l in linears:
            self.ends.append(self.ends[-1] + l.col.numel())
        self.col, self.values = torch.cat([l.col for l in linears]), torch.cat([l.values for l in linears])
        self.bias = torch.cat([l.bias for l in linears])
        for i, (l, at, end) in enumerate(zip(linears, self.ends, self.ends[1:])):
            l.col, l.values = self.col[at:end], self.values[at * self.V: end * self.V]
            l.bias = self.bias[i * self.rows: (i + 1) * self.rows]
            l.plan = ops.Plan(l.row_offsets, l.col, l.V, l.in_features)

    @staticmethod
    def fits(linears) -> bool:
        a = linears[0]
        return all(l.V == a.V and l.out_features == a.out_features and l.in_features == a.in_features and l.out_features % l.V == 0 and
                   l.bias is not None for l in linears)

    def _holds(self, linears) -> bool:
        """Whether these are still linears whose tensors are the views of what is stacked (a tensor or a linear may have been replaced)."""
        if any(type(l) is not SparseLinear for l in linears):
            return False

        def view(t, whole, at, end):
            return t.numel() == end - at and t.dtype == whole.dtype and t.is_contiguous() and \
                t.data_ptr() == whole.data_ptr() + at * whole.element_size()
        if any(l.bias is None for l in linears) or not _plain(self.bias, self.values, *(l.bias for l in linears), *(l.values for l in linears)):
            return False
        return all(view(l.col, self.col, at, end) and view(l.values, self.values, at * self.V, end * self.V) and
                   view(l.bias, self.bias, i * self.rows, (i + 1) * self.rows)
                   for i, (l, at, end) in enumerate(zip(linears, self.ends, self.ends[1:])))

    def operand(self, linears):
        """What ``ops.dense_copies`` takes, or None."""
        if not self._holds(linears):
            return None
        return [l.row_offsets for l in linears], self.ends[1:], self.col, self.values, self.V, linears[0].in_features

    def of_copy(self, copy: Optional[torch.Tensor], x: torch.Tensor):
        """The linears' results from the copy of what ``operand`` gave in this call, or None."""
        y = ops.of_copy(copy, x, self.V, self.bias) if copy is not None and _plain(x) else None
        return None if y is None else y.split(self.rows)

    def __call__(self, linears, x: torch.Tensor):
        """The linears' results, or None when these are not the operands that were stacked, a bias is not plain or the call is not
        one for a single product."""
        if not self._holds(linears):
            return None
        y = ops.sspmm_stacked([l.row_offsets for l in linears], [l.row_indices for l in linears], self.ends[1:], self.col, self.values, x,
                              self.V, self.bias)
        return None if y is None else y.split(self.rows)


class SparseEncoderLayer:
    def __init__(self, hidden=768, ffn=3072, heads=12, sparsity=0.9, vec_length=16, device="cuda:0", seed=400):
        self.hidden, self.ffn, self.heads, self.dev = hidden, ffn, heads, torch.device(device)
        shapes = [(hidden, hidden)] * 4 + [(ffn, hidden), (hidden, ffn)]
        self.linears = []
        g = torch.Generator(device="cpu").manual_seed(seed)
        for i, (m, k) in enumerate(shapes):
            w = synthetic.magnitude_pruned(m, k, sparsity, np.random.default_rng(seed + i))
            b = (0.02 * torch.randn(m, generator=g)).to(torch.float16).to(self.dev)
            self.linears.append(SparseLinear(w, vec_length, self.dev, b))
        self.qkv = StackedLinears(self.linears[:3]) if StackedLinears.fits(self.linears[:3]) else None
        self.ln1 = (torch.ones(hidden, dtype=torch.float16, device=self.dev), torch.zeros(hidden, dtype=torch.float16, device=self.dev))
        self.ln2 = (torch.ones(hidden, dtype=torch.float16, device=self.dev), torch.zeros(hidden, dtype=torch.float16, device=self.dev))

    @staticmethod
    def _layer_norm_fm(x, wb, eps=1e-5):
        xf = x.float()
        mu = xf.mean(dim=0, keepdim=True)
        var = xf.var(dim=0, unbiased=False, keepdim=True)
        return (((xf - mu) * torch.rsqrt(var + eps)) * wb[0].float()[:, None] + wb[1].float()[:, None]).to(x.dtype)

    def _attention(self, q, k, v, batch, seq):
        h, hd = self.heads, self.hidden // self.heads
        def split(t):            # [hidden, batch*seq] -> [batch, heads, seq, head_dim]
            return t.view(h, hd, batch, seq).permute(2, 0, 3, 1)
        o = F.scaled_dot_product_attention(split(q), split(k), split(v))
        return o.permute(1, 3, 0, 2).reshape(self.hidden, batch * seq)

    @staticmethod
    def _normable(x, tensors, rows) -> bool:
        """Whether LayerNorm's kernel takes x, all these tensors, and these numbers per feature."""
        return _plain(*tensors) and x.dim() == 2 and x.shape[1] % 8 == 0 and 0 < x.shape[0] <= 3072 and all(t.shape == x.shape[:1] for t in rows)

    def _norm(self, x, wb, add=None, bias=None, out=None, sum_out=None):
        """LayerNorm of x + bias + add: (what was normalised, the result)."""
        whole = [t for t in (x, add, out, sum_out) if t is not None]
        rows = [t for t in (bias, *wb) if t is not None]
        shape = x.shape
        if self._normable(x, [*whole, *rows], rows) and (bias is None or add is not None) and all(t.shape == shape for t in whole):
            out = torch.empty_like(x) if out is None else out
            if add is not None and sum_out is None:
                sum_out = torch.empty_like(x)
            ops.launch_layer_norm_fm(x, wb[0], wb[1], 1e-5, out, add, sum_out, bias)
            return (x if add is None else sum_out), out
        if bias is not None:
            x = x + bias[:, None]
        if add is not None:
            x = x + add
        y = self._layer_norm_fm(x, wb)
        return x, (y if out is None else out.copy_(y))

    def _attend(self, q, k, v, batch, seq, biases=(None, None, None), out=None):
        tokens = (self.hidden, batch * seq)
        given = [b for b in biases if b is not None]
        whole = [q, k, v] if out is None else [q, k, v, out]
        if self.hidden == 64 * self.heads and seq % 8 == 0 and seq > 0 and 0 < batch <= 65535 and _plain(*whole, *given) and \
                all(t.shape == tokens for t in whole) and all(b.shape == (self.hidden,) for b in given):
            out = torch.empty_like(q) if out is None else out
            ops.launch_attention_fm(q, k, v, self.heads, batch, seq, out, biases[0], biases[2])      # one of k changes nothing
            return out
        q, k, v = (t if b is None else t + b[:, None] for t, b in zip((q, k, v), biases))
        att = self._attention(q, k, v, batch, seq)
        return att.contiguous() if out is None else out.copy_(att)

    def _copies(self, x: torch.Tensor):
        """Dense copies of the operands of this call's products, of Q, K and V together, O, FFN1 and FFN2 (None for a product that does
        not work on one; below 512 tokens none does), and the LayerNorm of x, by one launch; None for that where there is none."""
        L, tokens = self.linears, x.shape[-1]
        qkv = getattr(self, "qkv", None)
        if tokens < 512 or any(type(l) is not SparseLinear or l.out_features % l.V for l in L[3:]):
            return [None] * 4, None
        first = qkv.operand(L[:3]) if qkv else None
        each = [([l.row_offsets], [l.col.numel()], l.col, l.values, l.V, l.in_features) for l in L[3:]]
        norm = (x, *self.ln1, 1e-5) if self._normable(x, [x, *self.ln1], self.ln1) else None
        made = ops.dense_copies(([first] if first else []) + each, tokens, norm)
        if made is None:
            return [None] * 4, None
        y = made.pop() if len(made) > len(each) + (first is not None) else None
        return (made if first else [None] + made), y

    def _groups_for(self, tokens: int):
        """Activation buffers of fixed shape and, bound to them, one group per dependency level of the layer:
        {Q, K, V} share their input and run as one launch, then O, FFN1, FFN2.  Groups keep addresses, so they are made again when a
        linear has another plan or other values (``.data`` gives a tensor another address)."""
        L = self.linears
        bound = [l.plan for l in L], [l.values.data_ptr() for l in L]
        if getattr(self, "_tokens", None) == tokens and bound == self._bound:
            return
        self._tokens = None
        z = lambda rows: torch.empty((rows, tokens), dtype=torch.float16, device=self.dev)
        b = self.buf = {"ln1": z(self.hidden), "q": z(self.hidden), "k": z(self.hidden), "v": z(self.hidden),
                        "att": z(self.hidden), "o": z(self.hidden), "sum": z(self.hidden), "ln2": z(self.hidden),
                        "h": z(self.ffn), "y": z(self.hidden)}
        item = lambda l, src, dst: (l.plan, l.values, b[src], b[dst])
        self.groups = None
        if all(l.plan.one_launch and l.out_features % l.V == 0 for l in L):
            self.groups = [ops.Group([item(L[0], "ln1", "q"), item(L[1], "ln1", "k"), item(L[2], "ln1", "v")]),
                           ops.Group([item(L[3], "att", "o")]), ops.Group([item(L[4], "ln2", "h")]),
                           ops.Group([item(L[5], "h", "y")])]
        self._tokens, self._bound = tokens, bound

    def forward_grouped(self, x: torch.Tensor, batch: int, seq: int) -> torch.Tensor:
        """Same layer with the linears run as groups (sspmm_group_run) on preallocated activation buffers.  The biases of
        Q and V go into the attention, the one of O into the LayerNorm, FFN2's into the last sum.  For short sequences (fewer
        launches, little host work); at 32 x 512 tokens, 768 wide, ``forward`` is the faster form (0.36 against 0.53 ms: products
        of many rows run on CTA pairs there)."""
        self._groups_for(batch * seq)
        if self.groups is None:
            return self.forward(x, batch, seq)
        b, L, g = self.buf, self.linears, self.groups
        self._norm(x, self.ln1, out=b["ln1"])
        g[0].run()
        self._attend(b["q"], b["k"], b["v"], batch, seq, [l.bias for l in L[:3]], out=b["att"])
        g[1].run()
        out, _ = self._norm(b["o"], self.ln2, add=x, bias=L[3].bias, out=b["ln2"], sum_out=b["sum"])
        bias = L[4].bias_rows()
        added = g[2].bias(0, bias) and bias is not None
        g[2].run()
        if L[4].bias is not None and not added:
            b["h"] += L[4].bias[:, None]
        bias = L[5].bias_rows()
        plain = bias is not None and out is b["sum"] and bias.get_device() == out.get_device()    # as LayerNorm's kernel left it
        y = g[3].run_sum(bias, out) if plain else None
        if y is not None:
            return y
        g[3].run()
        if plain:
            return ops.launch_add_bias_fm(b["y"], bias, out)
        return (b["y"] if L[5].bias is None else b["y"] + L[5].bias[:, None]) + out

    def forward(self, x: torch.Tensor, batch: int, seq: int, dense: bool = False) -> torch.Tensor:
        """x: [hidden, batch*seq] fp16, feature-major (token t of sequence b is column b*seq + t).  ``dense``: the same layer
        with dense products and framework operations only, nothing of this package's kernels."""
        L = self.linears
        if dense:
            y = self._layer_norm_fm(x, self.ln1)
            q, k, v = (l.dense_forward(y) for l in L[:3])
            out = L[3].dense_forward(self._attention(q, k, v, batch, seq).contiguous()) + x
            return L[5].dense_forward(L[4].dense_forward(self._layer_norm_fm(out, self.ln2))) + out
        copies, y = self._copies(x)

        def product(i, a):
            y = L[i].of_copy(copies[i - 2], a) if copies[i - 2] is not None else None
            return L[i](a) if y is None else y
        if y is None:
            _, y = self._norm(x, self.ln1)
        qkv = getattr(self, "qkv", None)
        q, k, v = (qkv and (qkv.of_copy(copies[0], y) or qkv(L[:3], y))) or [l(y) for l in L[:3]]
        att = product(3, self._attend(q, k, v, batch, seq))
        out, y = self._norm(att, self.ln2, add=x)
        h = product(4, y)
        if type(L[5]) is not SparseLinear:
            return L[5](h) + out
        y = L[5].of_copy(copies[3], h, out)
        return L[5].plus(h, out) if y is None else y
