"""Host-side mirror of the reference's Python format / model-integration layer for the V:N:M path.

Mirrors (same names, argument meaning and return conventions):
  * SrNMTensor                 end2end/grouped_nmv_tensor.py:677-744 (values / columns / metadata, nnz, to_dense)
  * NMVectorSparsifier         end2end/bert_pytorch.py:56-83 (the shipped fixed-mask sparsifier)
  * sparse_dense_mul_dispatch  end2end/bert_pytorch.py:85-106
  * SrnmSpmm, linear_to_spmm   end2end/bert_pytorch.py:109-167
The compressor and the product run on the GPU through the C ABI (there is no CPU path); the `spatha`
torch extension is used when it has been built, else the ctypes binding -- both call the same library.
"""
import numpy as np
import torch

from . import capi, spatha_module
from .synth import vnm_sizes


def round_up(x, y):
    return -(-x // y) * y


class SrNMTensor:
    """V:N:M compressed matrix: `values` fp16 [nrows*Ksp], `columns` int32 column-loc, `metadata` int32.

    Built from a dense (already masked) matrix, an int mask of the kept entries and the column-loc
    array, exactly like the reference class; the arrays are bit-identical to the reference's."""

    def __init__(self, n_, m_, tileM_, dense_, mask_, columns_, device_):
        self.n, self.m, self.tileM = n_, m_, tileM_
        self.device = torch.device(device_)
        if self.device.type != "cuda":
            raise capi.VenomError("SrNMTensor needs a CUDA device (there is no CPU path)")
        self.nrows, self.ncols = dense_.shape
        ksp, nv, nm, nc = vnm_sizes(self.nrows, self.ncols, tileM_, m_, n_)
        self.nnz = nv
        d = dense_.detach().to(device=self.device, dtype=torch.float16).contiguous()
        self.columns = columns_.to(device=self.device, dtype=torch.int32).contiguous().reshape(-1)
        mask = None if mask_ is None else mask_.to(device=self.device, dtype=torch.int32).contiguous()
        self.values, self.metadata, self.violations = capi.compress(d, self.columns, tileM_, m_, n_, mask=mask)
        self._prepared = None

    @classmethod
    def from_arrays(cls, n_, m_, tileM_, shape, values, metadata, columns, violations):
        """The tensor of arrays that are compressed already (on a CUDA device)."""
        t = cls.__new__(cls)
        t.n, t.m, t.tileM = n_, m_, tileM_
        t.device = values.device
        t.nrows, t.ncols = shape
        t.nnz = values.numel()
        t.values, t.metadata, t.columns, t.violations = values, metadata, columns, violations
        t._prepared = None
        return t

    def prepared(self):
        if self._prepared is None:
            self._prepared = capi.Prepared(self.values, self.metadata, self.columns, self.nrows, self.ncols, self.tileM, self.m, self.n)
        return self._prepared

    def to_dense(self):
        return capi.decompress(self.values, self.metadata, self.columns, self.nrows, self.ncols, self.tileM, self.m, self.n)


def nm_vector_mask_sparsify(tensor, n, m, tileM):
    """Magnitude pruning to V:n:m on the GPU; same return value as the reference function of this name
    (end2end/grouped_nmv_tensor.py:746-779): (masks int32 [nrows, ncols], columns int32)."""
    return capi.prune_magnitude(tensor, tileM, m, n)


class MagnitudeSparsifier:
    """The magnitude path the reference keeps commented out in its scripts (end2end/bert_pytorch.py:63-64)."""

    def __init__(self, n, m, tileM):
        self.n, self.m, self.tileM = n, m, tileM

    def __call__(self, tensor, device=None):
        device = tensor.device if device is None else device
        w = tensor.detach().to(device)
        fused = capi.sparsify_magnitude(w, self.tileM, self.m, self.n)     # prunes and compresses in one pass
        if fused is not None:
            return SrNMTensor.from_arrays(self.n, self.m, self.tileM, tuple(tensor.shape), *fused)
        mask, columns = nm_vector_mask_sparsify(w, self.n, self.m, self.tileM)
        dense = tensor.detach().to(device=device, dtype=torch.float16) * mask.to(torch.float16)
        return SrNMTensor(self.n, self.m, self.tileM, dense, mask, columns, device)


class NMVectorSparsifier:
    """The sparsifier the reference's end-to-end scripts ship with: a fixed pattern that keeps columns
    0 and 2 of every group of m and uses column-loc {0,1,2,3} (end2end/bert_pytorch.py:66-75)."""

    def __init__(self, n, m, tileM):
        self.n, self.m, self.tileM = n, m, tileM

    def __call__(self, tensor, device=None):
        nrows, ncols = tensor.shape
        device = tensor.device if device is None else device
        ksp, nv, nm, nc = vnm_sizes(nrows, ncols, self.tileM, self.m, self.n)
        columns = torch.zeros(nc, dtype=torch.int32).reshape(-1, 4) + torch.tensor([0, 1, 2, 3], dtype=torch.int32)
        pattern = torch.zeros(self.m, dtype=torch.int32, device=tensor.device)  # built where the weight lives: GBs for large layers
        pattern[0] = 1
        pattern[2] = 1
        reps = -(-ncols // self.m)
        mask = pattern.repeat(reps)[:ncols].unsqueeze(0).expand(nrows, ncols).contiguous()
        dense = tensor.detach().to(torch.float16) * mask.to(torch.float16)
        return SrNMTensor(self.n, self.m, self.tileM, dense, mask, columns, device)


def sparse_dense_mul_dispatch(sparse_values, sparse_indices, sparse_metadata, dense, nrows_sp, ncols_sp, ncols_d, m, n, v, nnz, bias, form=capi.STRATEGY_AUTO):
    """Same call as the reference helper: returns [ncols_d, nrows_sp] = (A @ dense).T + bias.  form: see SrnmSpmm."""
    # the reference materialises `dense.contiguous()` here; the op accepts the transposed view itself and
    # copies only when it has to
    dense_ = dense
    return spatha_module().spmm(sparse_metadata, sparse_indices, sparse_values, dense_, bias, nrows_sp, ncols_sp, ncols_d, v, n, m, nnz, 0, 32, 4, form)


_linear = None     # the extension's call, looked up once


class SrnmSpmm(torch.nn.Module):
    """Drop-in replacement of torch.nn.Linear whose weight is stored in V:N:M form.

    form: the kernel-private copy of the weight that the layer holds on the device beside the arrays.  The default,
    capi.STRATEGY_AUTO, takes for every number of tokens the form estimated to be faster and keeps each form that has been
    wanted: at most 1.125 bytes (dense-B) plus 4.5 / m bytes (gather) a weight element.  capi.STRATEGY_GATHER and
    capi.STRATEGY_DENSE_B hold that one form only, whatever is faster."""

    form = capi.STRATEGY_AUTO    # layers that were pickled without one

    def __init__(self, original, n=2, m=8, v=64, sparsifier=None, form=capi.STRATEGY_AUTO):
        super().__init__()
        self.n, self.m, self.v = n, m, v
        self.form = form
        self.bias = original.bias
        w = (sparsifier or NMVectorSparsifier(n, m, v))(original.weight)
        self.values = torch.nn.Parameter(w.values, requires_grad=False)
        self.columns = w.columns
        self.metadata = w.metadata
        self.nrows_sp, self.ncols_sp, self.nnz = w.nrows, w.ncols, w.nnz

    def forward(self, input):
        # one call into the extension; parameters are read past torch.nn.Module.__getattr__ (0.4 us each at decoding sizes)
        p = self._parameters
        bias = p["bias"] if "bias" in p else self.bias
        values = p["values"] if "values" in p else self.values
        global _linear
        if _linear is None:
            _linear = spatha_module().linear
        out = _linear(input, self.metadata, self.columns, values, bias, self.nrows_sp, self.ncols_sp, self.v, self.n, self.m, self.form)
        if out is not None:
            return out
        flat = torch.flatten(input, start_dim=0, end_dim=-2)
        ncols_d = flat.shape[0]
        out = sparse_dense_mul_dispatch(values, self.columns, self.metadata, flat.T, self.nrows_sp, self.ncols_sp, ncols_d,
                                        self.m, self.n, self.v, self.nnz, bias, self.form)
        return out.reshape((*input.shape[0:-1], -1))


def linear_to_spmm(mod, n=2, m=8, v=64, skip=(), form=capi.STRATEGY_AUTO):
    """Replaces every torch.nn.Linear below `mod` by SrnmSpmm (end2end/bert_pytorch.py:155-167)."""
    if isinstance(mod, torch.nn.Linear):
        return SrnmSpmm(mod, n, m, v, form=form)
    for name, child in mod.named_children():
        if isinstance(child, SrnmSpmm) or name in skip:
            continue
        if isinstance(child, torch.nn.Linear):
            setattr(mod, name, SrnmSpmm(child, n, m, v, form=form))
        elif child is not mod:
            linear_to_spmm(child, n, m, v, skip, form)
    return mod
