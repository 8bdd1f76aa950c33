"""A linear layer on the MXFP4 path: weights held as packed E2M1 codes with their scales already in
the layout the GEMM reads, activations quantised on the fly.

Counterpart of the reference's module wrappers around its kernels (wave_lang/kernel/wave/nn/linear.py:147
`WaveLinear`, nn/quant_linear.py:196 `WaveQuantLinear`, which is FP8 per-tensor); the reference has
no MXFP4 module. forward(x) = dequant(quantise(x)) @ dequant(W)^T, output bf16 or f32.
"""

from __future__ import annotations

import torch

from . import _lib, ops
from .lang import as_output_dtype


_entry = None  # the function that the host module calls


def _native():
    """The host module, unless it cannot be used or a caller has put something in the place of what it calls, to watch or to redirect calls."""
    global _entry
    if _entry is None and _lib.fast() is not None:
        _entry = _lib._fast_entries["wb200_mxfp4_gemm_quantize_a"]
    lib = _lib._lib
    if not _lib._fast or _lib.load is not _lib._loader or lib is not _lib._fast_lib or lib.wb200_mxfp4_gemm_quantize_a is not _entry:
        return None
    return _lib._fast


class MXFP4Linear(torch.nn.Module):
    def __init__(self, weight_codes: torch.Tensor, weight_scales: torch.Tensor, output_dtype=torch.bfloat16):
        """weight_codes [N, K/2] uint8, weight_scales [N, K/32] uint8 (row-major E8M0), both on the GPU. The GEMM reads the scales in
        packings that are made here, on the current stream, and anew when a state dict is loaded."""
        super().__init__()
        ops._as_u8(weight_codes, "weight_codes")
        self.out_features, half_k = weight_codes.shape
        self.in_features = half_k * 2
        self.output_dtype = as_output_dtype(output_dtype).torch_dtype
        self.register_buffer("weight_codes", weight_codes.contiguous())
        self.register_buffer("weight_scales", weight_scales.contiguous())
        self._pack()

    # Decode calls (at most 128 rows) may read a second packing, per tile of the height h that gives every SM the same number of
    # weight tiles: one height per layer, as it follows from out_features, and 128 / h times the bytes of the usual packing. Made with that one, not
    # by the first call that reads it: other streams' calls would have to wait for that call's.
    _packed = _packed_low = None
    _native_scales = None  # of both, as the native call takes them

    def _pack(self) -> None:
        self._packed = self._pack_as(self._packed, 128)
        h = self._low_rows()
        self._packed_low = None if h == 128 else self._pack_as(self._packed_low, h)
        low = self._packed_low or self._packed
        self._native_scales = self._packed.rows, self._packed.K, self._packed.data, low.data, low.tile_rows

    def _pack_as(self, old: ops.PackedScales | None, tile_rows: int) -> ops.PackedScales:
        """In the memory of the packing that there is, if it is of that form: captured graphs hold its address, as they hold that of the codes,
        which a state dict is copied into."""
        s = self.weight_scales
        same = old is not None and old.device == s.device and (old.rows, old.K, old.tile_rows) == (s.shape[0], s.shape[1] * ops.SCALE_GROUP_SIZE, tile_rows)
        return ops.repack_scales(s, out=old.data if same else None, tile_rows=tile_rows)

    def _low_rows(self) -> int:
        """The height that decode calls of some number of rows read, 128 where none does. (One of each class that
        `ops.decode_tile_rows_for` tells apart: by rows, and by whether rows of the output start on 16 bytes, as that of one row does.)"""
        N, K, device = self.out_features, self.in_features, self.weight_scales.device
        aligned = N * self.output_dtype.itemsize % 16 == 0
        for rows, c_aligned in ((1, True), (2, aligned), (32, aligned), (64, aligned), (128, aligned)):
            h = ops.decode_tile_rows_for(rows, N, K, device, c_aligned=c_aligned)
            if h != 128:
                return h
        return 128

    def _load_from_state_dict(self, *args, **kwargs) -> None:
        super()._load_from_state_dict(*args, **kwargs)
        if self.weight_scales is not None and self.weight_scales.is_cuda:
            self._pack()

    @property
    def _packed_decode(self) -> ops.PackedScales:
        return self._packed if self._packed_low is None else self._packed_low

    @classmethod
    def from_float(cls, weight: torch.Tensor, output_dtype=torch.bfloat16) -> "MXFP4Linear":
        """Quantise an f32 / bf16 [N, K] weight on the GPU."""
        q, s, _ = ops.quantize_mxfp4(weight, want_rowmajor=True, want_packed=False)
        return cls(q, s, output_dtype)

    def forward(self, x: torch.Tensor) -> torch.Tensor:
        # a call whose tensors need no preparation; anything else comes back unhandled
        native, scales = _native(), self._native_scales
        if native is None or scales is None:
            return self._forward_checked(x)
        y = native.linear(x, self._buffers.get("weight_codes"), scales, self.output_dtype, ops._pool._fast or ops._pool.fast)
        if type(y) is int:
            _lib.check(y)
        elif y is not None:
            return y
        return self._forward_checked(x)

    def _forward_checked(self, x: torch.Tensor) -> torch.Tensor:
        lead = x.shape[:-1]
        x2 = x.reshape(-1, self.in_features)
        out = torch.empty(x2.shape[0], self.out_features, dtype=self.output_dtype, device=x.device)
        packed = self._packed
        if x2.shape[0] <= 128:
            packed = self._decode_packing(out)
        ops.quantized_gemm(x2, self.weight_codes, packed, out)
        return out.reshape(*lead, self.out_features)

    def _decode_packing(self, out: torch.Tensor) -> ops.PackedScales:
        low = self._packed_low
        if low is None:
            return self._packed
        h = ops.decode_tile_rows_for(out.shape[0], self.out_features, self.in_features, out.device, c_aligned=ops.rows_aligned(out))
        return low if h == low.tile_rows else self._packed
