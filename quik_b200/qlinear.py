"""MixedQLinear -- the mixed-precision quantized linear layer, API-compatible with the reference
module (QUIK experiments/qlinear.py:11-199): same constructor, ``from_float``, buffer names, dtypes
and shapes (so reference ``state_dict``s load), same ``SharedQuantizedInput`` protocol.

``forward`` runs two launches instead of the reference's five: the activation quantizer and one
fused kernel (integer GEMM + outlier fp16 GEMM + dequantize).  ``MixedQLinear.fused = False``
switches to the reference's own operator sequence (quantize -> int matmul -> F.linear ->
dequantize) on this package's operators.
"""
from __future__ import annotations

import numpy as np
import torch
from torch import Tensor

from . import _lib, asymmetric, matmul, symmetric

__all__ = ["two_compl", "pack_to_i4", "SharedQuantizedInput", "MixedQLinear"]


def two_compl(x: Tensor, bits: int) -> Tensor:
    """Unsigned two's-complement representation of negative values (experiments/qlinear.py:11-12)."""
    return torch.where(x < 0, 2 ** bits + x, x)


def pack_to_i4(X: Tensor) -> Tensor:
    """Pack int4 values two per byte, even column in the low nibble (experiments/qlinear.py:15-18)."""
    X_i8 = two_compl(X.to(dtype=torch.int8), 4).to(torch.uint8)
    return X_i8[:, 0::2] | (X_i8[:, 1::2] << 4)


class SharedQuantizedInput:
    """Quantized-activation cache shared by the layers of one group (q/k/v, gate/up);
    experiments/qlinear.py:21-37.  The first member quantizes, the others reuse, and the cache is
    dropped after ``group_size`` calls to :meth:`finish`."""

    def __init__(self, group_size):
        self.qint_x = None
        self.fp_x = None
        self.qscale_x = None
        self.meta = None
        self.wide = False          # layout of qint_x: one code per byte (True) or the reference layout
        self.group_size = group_size
        self.cur_group_elem = 0

    def finish(self):
        self.cur_group_elem += 1
        if self.cur_group_elem == self.group_size:
            self.qint_x = None
            self.qscale_x = None
            self.meta = None
            self.fp_x = None
            self.cur_group_elem = 0


def _to_u16(idx: Tensor, cols: int | None = None) -> Tensor:
    """int64 column ids -> the same ids as 16-bit values (stored in an int16 tensor) on idx.device.

    The kernels index the row in shared memory with these ids without a range check (like the reference's kernels,
    src/asymmetric/asymmetric.cu:351-372), so ids outside [0, cols) are refused here, once per layer."""
    a64 = idx.detach().cpu().numpy().astype(np.int64)
    limit = 65536 if cols is None else cols
    if a64.size and (a64.min() < 0 or a64.max() >= limit):
        raise RuntimeError(f"MixedQLinear: column ids must lie in [0, {limit}), got [{a64.min()}, {a64.max()}]")
    return torch.from_numpy(a64.astype(np.uint16).view(np.int16).copy()).to(idx.device)


class MixedQLinear(torch.nn.Module):
    fused = True   # class-wide default; set on an instance to override
    # optional profiling hook: called as hook(module, begin: bool) right before / after the fused
    # GEMM launch (on the launching stream), e.g. to record CUDA events
    launch_hook = None
    # optional caller-owned output buffer [M, out_features] (e.g. symmetric memory of a tensor-parallel
    # group); used by the fused path when its shape, dtype and device match
    out_buffer = None
    # weights of the last call for few tokens (see _weights_record); every layer has its own
    _seen = bytearray(32)

    def __init__(self, in_features, out_features, shared_input=None,
                 fp_features_num=0, symm=False, bits=4, dtype=torch.float16):
        super().__init__()
        self.fp_features_num = fp_features_num
        self.int_features_num = in_features - fp_features_num
        self.in_features = in_features
        self.out_features = out_features
        self.symmetric = symm
        self.bits = bits
        self.shared_input = shared_input
        self.dtype = dtype
        # buffer schema of experiments/qlinear.py:53-78
        self.register_buffer('weights_scales', torch.zeros((self.out_features, 1), dtype=self.dtype))
        if self.bits == 4:
            self.register_buffer('int_weight', torch.randint(1, 7, (self.out_features, self.int_features_num // 2),
                                                             dtype=torch.uint8))
        else:
            self.register_buffer('int_weight', torch.randint(-128, 127, (self.out_features, self.int_features_num),
                                                             dtype=torch.int8))
        self.register_buffer('bias', torch.zeros((self.out_features), dtype=dtype))
        self.register_buffer('int_indices', torch.zeros((self.int_features_num), dtype=torch.long))
        self.register_buffer('fp_indices', torch.zeros((self.fp_features_num), dtype=torch.long))
        if self.fp_features_num > 0:
            self.register_buffer('fp_weight', torch.randint(-8, 7, (self.out_features, self.fp_features_num)).to(dtype))
        if not self.symmetric:
            self.register_buffer('reduced_w', torch.zeros((1, self.out_features), dtype=dtype))
        self._cache = {}
        self._seen = bytearray(32)

    @classmethod
    def concat(cls, modules):
        """One layer whose output is the outputs of ``modules`` side by side.

        For layers that read the same input through the same column split (q/k/v, gate/up: a shared-input group of
        experiments/llama.py:402-411): per-channel scales, reduced_w, the integer and the outlier weights are simply
        stacked along the output dimension, so every output column is computed exactly as in its own layer, in one
        quantizer call and one fused launch instead of one launch per member."""
        m0 = modules[0]
        for m in modules[1:]:
            assert (m.bits, m.symmetric, m.in_features, m.fp_features_num, m.dtype) == \
                   (m0.bits, m0.symmetric, m0.in_features, m0.fp_features_num, m0.dtype), "layers differ in format"
            assert torch.equal(m.int_indices, m0.int_indices) and torch.equal(m.fp_indices, m0.fp_indices), \
                "layers differ in their outlier columns"
            assert (m.bias is None) == (m0.bias is None)
        out = cls(m0.in_features, sum(m.out_features for m in modules), fp_features_num=m0.fp_features_num,
                  symm=m0.symmetric, bits=m0.bits, dtype=m0.dtype)
        out.weights_scales = torch.cat([m.weights_scales for m in modules], 0)
        out.int_weight = torch.cat([m.int_weight for m in modules], 0).contiguous()
        out.bias = None if m0.bias is None else torch.cat([m.bias for m in modules], 0)
        out.int_indices, out.fp_indices = m0.int_indices, m0.fp_indices
        if m0.fp_features_num > 0:
            out.fp_weight = torch.cat([m.fp_weight for m in modules], 0).contiguous()
        if not m0.symmetric:
            out.reduced_w = torch.cat([m.reduced_w for m in modules], 1).contiguous()
        return out

    # ------------------------------------------------------------------ derived, lazily built operands
    def _cached(self, name, src: Tensor, make):
        """make(src), kept as long as ``src`` is the same tensor at the same version (not only at the same address)."""
        ent = self._cache.get(name)
        if ent is None or not _lib.host().same_sources(ent[0], src):
            ent = (_lib.host().sources(src), make(src))
            self._cache[name] = ent
        return ent[1]

    def __getstate__(self):
        # what was derived from this object's buffers stays here: a copy, or the object read back from a file, derives its own
        state = self.__dict__.copy()
        state.update(_cache={}, _seen=bytearray(32))
        return state

    def _idx16(self):
        k = self.in_features
        i16 = self._cached("int16", self.int_indices, lambda t: _to_u16(t, k))
        f16 = self._cached("fp16", self.fp_indices, lambda t: self._checked_fp_ids(t, k))
        return i16, f16

    def _checked_fp_ids(self, fp_idx, k):
        # integer and outlier columns must not overlap (experiments/qlinear.py:168-169 asserts the same at construction)
        both = torch.cat([self.int_indices.detach().cpu(), fp_idx.detach().cpu()])
        if both.numel() != k or torch.unique(both).numel() != k:
            raise RuntimeError("MixedQLinear: int_indices and fp_indices must together name every input column exactly once")
        return _to_u16(fp_idx, k)

    def _weight_codes_int8(self):
        """Weight codes one per byte, the operand layout of the tensor-core engine."""
        if self.bits == 8:
            return self.int_weight
        return self._cached("w8", self.int_weight, matmul.unpack_int4)

    def _operand_layouts(self, M):
        """(token codes packed?, weight codes packed?) for M tokens: which engine the fused launch will use."""
        return _lib.host().operand_layouts(self.bits, self.int_features_num, M)

    def _quantize(self, producer, x, aux, eps, wide):
        """(codes, meta, outliers) of producer(x) with this layer's columns; its ids are settled: ``_to_u16`` made them on the
        host and copied them synchronously."""
        i16, f16 = self._idx16()
        plan = self._plan
        if plan is not None and (plan[0] is None or plan[1] is None):
            self._cache.pop("plan", None)      # made before the ids were: the layer's next launch makes it again
        return _lib.host().quantize(producer, x, aux, eps, i16, f16, self.bits, wide, True)

    @property
    def _plan(self):
        """Derived operands for the native host path (see _make_plan), part of the layer's cache and dropped with it."""
        return self._cache.get("plan")

    def _make_plan(self):
        """What the native host path needs of this layer beside its buffers: 16-bit column ids and weight codes one per byte, each
        where this layer has derived them, and the buffers that these come from.  It reads the buffers itself on every call
        and declines where they are others or something is missing: the layer's own path then runs, and ends here again.  Nothing
        is derived here: a member of a group whose input another member quantizes needs no ids, and may not even have any.  No plan
        where none could serve: the path is not taken, or what it reads is not a buffer of the layer."""
        self._cache.pop("plan", None)
        if self.out_buffer is not None or MixedQLinear.launch_hook is not None:
            return
        b = self._buffers
        sources = [b.get(n) for n in ("int_indices", "fp_indices", "int_weight", "fp_weight")[:4 if self.fp_features_num > 0 else 3]]
        if "bias" not in b or b.get("weights_scales") is None or b.get("reduced_w") is None \
                or any(t is None or t.is_inference() for t in sources):
            return
        host = _lib.host()
        key = host.sources(*sources)

        def derived(name, src):
            ent = self._cache.get(name)
            return ent[1] if ent is not None and host.same_sources(ent[0], src) else None
        self._cache["plan"] = (*map(derived, ("int16", "fp16", "w8"), sources), key)

    def _weights_record(self):
        """The record of the weights of this layer's last call for few tokens, emptied where they are other tensors since: the record
        itself knows them by address and version only.  (The native path checks by its plan that they are the same.)"""
        host, weights = _lib.host(), [self.int_weight, *([self.fp_weight] if self.fp_features_num > 0 else [])]
        if not any(t.is_inference() for t in weights) and not host.same_sources(self._cache.get("weights"), *weights):
            self._seen[:] = bytes(32)
            self._cache["weights"] = host.sources(*weights)
        return self._seen

    def _quantize_by_plan(self, producer, x, aux, eps):
        """Fills the group's shared input from the native host path; False where that declines."""
        plan, shared_input = self._plan, self.shared_input
        if plan is None or shared_input is None:
            return False
        filled = _lib.host().quantize_for(self, plan, producer, x, aux, eps)
        if filled is None:
            return False
        shared_input.qint_x, shared_input.meta, shared_input.fp_x, shared_input.wide = filled
        return True

    def _fill_shared(self, quantized, wide):
        shared_input = self.shared_input
        if shared_input is None:
            raise RuntimeError("a fused producer needs a SharedQuantizedInput on the layer (group size >= 1)")
        shared_input.qint_x, shared_input.meta, shared_input.fp_x = quantized
        shared_input.wide = wide

    def quantize_rmsnorm(self, x, norm_weight, eps):
        """Quantizes RMSNorm(x) * norm_weight straight into this layer's shared input (one pass over x, the normalised
        activations never go to HBM).  The following forward calls of the group's members find the codes and skip their
        own quantizer; pass them any tensor of x's shape, dtype and device (it is not read)."""
        if self._quantize_by_plan(1, x, norm_weight, eps):
            return
        x2 = x[0] if x.dim() == 3 else x
        q_packed, _ = self._operand_layouts(x2.shape[0])
        self._fill_shared(self._quantize(1, x2.contiguous(), norm_weight, eps, not q_packed), not q_packed)

    def quantize_silu_mul(self, gate, up):
        """Quantizes SiLU(gate) * up straight into this layer's shared input (see :meth:`quantize_rmsnorm`)."""
        if self._quantize_by_plan(2, gate, up, 0.0):
            return
        g2 = gate[0] if gate.dim() == 3 else gate
        u2 = up[0] if up.dim() == 3 else up
        q_packed, _ = self._operand_layouts(g2.shape[0])
        self._fill_shared(self._quantize(2, g2.contiguous(), u2.contiguous(), 0.0, not q_packed), not q_packed)

    # ------------------------------------------------------------------ forward
    def forward(self, x):
        plan = self._cache.get("plan")
        if plan is not None and self.fused and not self.symmetric and MixedQLinear.launch_hook is None and self.out_buffer is None:
            shared_input = self.shared_input
            if shared_input is None:
                out = _lib.host().forward(self, plan, self._seen, x)
                if out is not None:
                    return out
            elif shared_input.qint_x is not None or self._quantize_by_plan(0, x, None, 0.0):
                out = _lib.host().forward_quantized(self, plan, self._seen, x, shared_input.qint_x, shared_input.meta,
                                                    shared_input.fp_x, shared_input.wide)
                if out is not None:
                    shared_input.finish()
                    return out
        return self._forward_checked(x)

    def _forward_checked(self, x):
        if self.int_features_num <= 0:
            return torch.nn.functional.linear(x, self.fp_weight, self.bias)
        if torch.cuda.current_device() != x.device.index:
            torch.cuda.set_device(x.device)

        shared_input = self.shared_input
        if shared_input is None:
            if self.fused and not self.symmetric and MixedQLinear.launch_hook is None:
                return self._forward_one_call(x)
            shared_input = SharedQuantizedInput(1)
        if len(x.shape) == 3:
            x = x[0]
        if self.symmetric:
            return self._forward_symmetric(x, shared_input)
        if not self.fused:
            return self._forward_unfused(x, shared_input)

        M = x.shape[0]
        q_packed, w_packed = self._operand_layouts(M)
        wide = not q_packed
        if shared_input.qint_x is not None and self.bits == 4 and shared_input.wide != wide:
            raise RuntimeError("MixedQLinear: the shared quantized input was written in another code layout than this "
                               "member needs (the members of a group must run on the same engine)")
        if shared_input.qint_x is None:
            shared_input.qint_x, shared_input.meta, shared_input.fp_x = self._quantize(0, x, None, 0.0, wide)
            shared_input.wide = wide
        w = self.int_weight if (w_packed or self.bits == 8) else self._weight_codes_int8()
        hook = MixedQLinear.launch_hook
        if hook is not None:
            hook(self, True)
        out = _lib.host().linear(x, self._out_buffer_for(x, M), *self._constants(), w, w_packed, shared_input.qint_x, q_packed,
                                 shared_input.meta, shared_input.fp_x, self._weights_record())
        if hook is not None:
            hook(self, False)
        shared_input.finish()
        self._make_plan()
        return out

    def _out_buffer_for(self, x, M):
        """The caller's output buffer (may be a column range of a wider row-major matrix) where it fits, else None."""
        ob = self.out_buffer
        if ob is not None and tuple(ob.shape) == (M, self.out_features) and ob.dtype == x.dtype \
                and ob.device == x.device and ob.stride(1) == 1 and ob.stride(0) >= self.out_features:
            return ob
        return None

    def _constants(self):
        """The layer's own arguments of the native host path."""
        b = self._buffers
        try:
            scales, reduced, bias = b["weights_scales"], b["reduced_w"], b["bias"]
        except KeyError:          # replaced by something that is not a buffer
            scales, reduced, bias = self.weights_scales, self.reduced_w, self.bias
        f = self.fp_features_num
        return (scales, reduced, self.fp_weight if f > 0 else None, bias, self.int_features_num, self.out_features, f, self.bits)

    def _forward_one_call(self, x):
        """The layer on its own input, [1, M, K] or [M, K]: quantizer and fused kernel from one native call."""
        w = self.int_weight
        ids, fp_ids = self._idx16()
        M = x.shape[-2] if x.dim() > 1 else 0
        wide = self._weight_codes_int8() if self.bits == 4 and not self._operand_layouts(M)[1] else None
        out = self._out_buffer_for(x, M)
        res = _lib.host().layer(x, out, *self._constants(), w, wide, ids, fp_ids, self._weights_record())
        if res is None:          # a setting that another thread has changed since asks for weight codes one per byte
            res = _lib.host().layer(x, out, *self._constants(), w, self._weight_codes_int8(), ids, fp_ids, self._seen)
        self._make_plan()
        return res

    def _forward_unfused(self, x, shared_input):
        """The reference's operator sequence (experiments/qlinear.py:105-148)."""
        group_input = shared_input
        if shared_input.qint_x is not None and self.bits == 4 and shared_input.wide:
            # a fused member of the group left its codes one per byte; the reference operators take the packed layout
            shared_input = SharedQuantizedInput(1)
        if shared_input.qint_x is None:
            shared_input.qint_x, shared_input.meta, shared_input.fp_x = asymmetric.quantize(
                x, self.int_indices, self.fp_indices, self.bits)
            shared_input.wide = False
        if self.fp_features_num > 0:
            fp_result = torch.nn.functional.linear(shared_input.fp_x, self.fp_weight, self.bias)
        elif self.bias is not None:
            fp_result = self.bias.repeat(shared_input.qint_x.shape[0], 1)
        else:
            fp_result = torch.zeros((shared_input.qint_x.shape[0], self.out_features), dtype=x.dtype, device=x.device)
        if self.bits == 4:
            int_result = matmul.int4Matmul(shared_input.qint_x, self.int_weight)
        else:
            int_result = matmul.int8Matmul(shared_input.qint_x, self.int_weight)
        output = asymmetric.dequantize(int_result, shared_input.meta, self.weights_scales, self.reduced_w,
                                       fp_result, self.bits)
        shared_input.finish()
        if group_input is not shared_input:
            group_input.finish()
        return output.reshape((1, *output.shape))

    def _forward_symmetric(self, x, shared_input):
        """Symmetric-activation branch (experiments/qlinear.py:94-103,141-142).  The reference calls
        quik.symmetric.quantize / dequantize without their ``bits`` argument there, which raises
        TypeError against its own extension; this passes ``bits`` (and 32 for the int32 accumulator)."""
        if shared_input.qint_x is None:
            if self.fp_features_num > 0:
                int_x = x[:, self.int_indices].contiguous()
                shared_input.fp_x = x[:, self.fp_indices].contiguous()
            else:
                int_x = x
            reshaped_x = int_x.reshape((-1, int_x.shape[-1]))
            shared_input.qscale_x = (torch.max(torch.abs(reshaped_x), dim=1)[0].unsqueeze(1) / (
                    1 << (self.bits - 1) - 1)).to(torch.float16)
            shared_input.qint_x = symmetric.quantize(int_x, shared_input.qscale_x, self.bits)
        if self.fp_features_num > 0:
            fp_result = torch.nn.functional.linear(shared_input.fp_x, self.fp_weight, self.bias)
        elif self.bias is not None:
            fp_result = self.bias.repeat(shared_input.qint_x.shape[0], 1)
        else:
            fp_result = torch.zeros((shared_input.qint_x.shape[0], self.out_features), dtype=x.dtype, device=x.device)
        if self.bits == 4:
            int_result = matmul.int4Matmul(shared_input.qint_x, self.int_weight)
        else:
            int_result = matmul.int8Matmul(shared_input.qint_x, self.int_weight)
        output = symmetric.dequantize(int_result, shared_input.qscale_x, self.weights_scales.reshape(1, -1).contiguous(),
                                      fp_result, 32)
        shared_input.finish()
        return output.reshape((1, *output.shape))

    # ------------------------------------------------------------------ construction
    @staticmethod
    def from_float(module: torch.nn.Linear, weight_matrix, weights_scales, shared_input=None,
                   fp_indices=None, symm=False, bits=4):
        """Build the layer from a float ``nn.Linear`` (experiments/qlinear.py:150-199).

        ``weight_matrix`` holds the (already rounded-to-grid) weights, ``weights_scales`` the
        per-output-channel scale [out_features, 1].  Integer columns are stored as
        ``round(W / scale)`` (packed two per byte for 4 bits), outlier columns verbatim, and
        ``reduced_w`` is the fp32 row sum of the integer-column weights.
        """
        assert weights_scales.shape == (module.out_features, 1), 'weights_scales should have shape (out_features, 1)'
        assert weight_matrix.shape == (module.out_features, module.in_features)
        assert (symm and bits == 4) or not symm, "Symmetric quantization with 8 bits is not supported"
        int_indices = torch.arange(module.in_features)
        if fp_indices is None or len(fp_indices) == 0:
            fp_indices = torch.tensor([], dtype=int_indices.dtype)
        else:
            fp_indices = fp_indices.cpu()
            int_indices = int_indices[~torch.isin(int_indices, fp_indices)]
        assert torch.numel(int_indices) + torch.numel(fp_indices) == module.in_features, \
            'There are some duplication in the fp_indices!'

        int_module = MixedQLinear(module.in_features, module.out_features, shared_input,
                                  fp_features_num=torch.numel(fp_indices), symm=symm, bits=bits,
                                  dtype=weight_matrix.dtype)
        if torch.cuda.is_available():
            weight_matrix = weight_matrix.cuda()
        dev = weight_matrix.device
        int_module.weights_scales.copy_(weights_scales.to(weight_matrix.dtype))
        int_rounded_weight = (weight_matrix[:, int_indices.to(dev)] / weights_scales.to(dev)).round()
        if bits == 4:
            int_module.int_weight.copy_(pack_to_i4(int_rounded_weight.to(torch.int8)).cpu())
        else:
            int_module.int_weight.copy_(int_rounded_weight.to(torch.int8).cpu())
        if not symm:
            reduced_w = torch.sum(weight_matrix[:, int_indices.to(dev)].float(), dim=1, keepdim=True).to(
                weight_matrix.dtype)
            int_module.reduced_w.copy_(reduced_w.t().cpu())
        if module.bias is not None:
            int_module.bias.copy_(module.bias)
        else:
            int_module.bias = None
        int_module.int_indices.copy_(int_indices)
        int_module.fp_indices.copy_(fp_indices)
        if int_module.fp_features_num > 0:
            int_module.fp_weight.copy_(weight_matrix[:, fp_indices.to(dev)].to(weight_matrix.dtype))
        return int_module
