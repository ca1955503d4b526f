"""Host-side mirror of the reference's quantized-matmul operator for this path: `QTensor`, `QMatMul` and
`GgufMatMul` with the same names, argument meaning and error behaviour, on torch device memory.

Reference: `QTensor` / `QMatMul` (crates/inference-tensor/src/quantized/mod.rs:85-120,1117-1187,1625-1647),
`GgufMatMul::forward` and its dispatch (crates/inference-quant/src/gguf/mod.rs:435-571), the row-count policy of
`fast_mmvq::plain` / `fast_mmq::plain` (crates/inference-quant/src/gguf/fast_mmvq.rs:84-134,477-665,
fast_mmq.rs:604-715). Every forward runs the CUDA kernels of the C-ABI library; there is no CPU fallback.
"""
from __future__ import annotations

import torch

from . import ops
from .dtypes import MATRIX_ROW_PADDING, GgmlDType, pad
from . import kernel_library as kl

MMVQ_MAX_BATCH = 8  # rows the decode GEMV launchers take (fast_mmvq.rs:84)
TENSOR_CORE_MAX_ROWS = 16  # rows the small-batch tensor-core kernel takes (fast_mmvq.rs:86)

# 3..8 rows that always took the tier, at any address: weights off the 16-byte boundaries it needs are refused there, as ever.
# `_tier_overtakes` adds the rows on which it is the faster one as well.


def _tensor_core_pays(dtype: GgmlDType, rows: int, n: int, k: int) -> bool:
    big = k >= 8192 or n >= 16384
    if dtype == GgmlDType.Q6K:
        return rows >= 7 or (rows >= 4 and big) or n >= 65536
    return rows >= 5 or big


def tensor_core_rows_supported(dtype: GgmlDType, k: int) -> bool:
    """Shapes `b200q_gemv_tc` takes: whole 256-value chunks and packed rows of a multiple of 16 bytes."""
    return k % 256 == 0 and dtype.row_bytes(k) % 16 == 0


def prefers_tensor_core_rows(dtype: GgmlDType, rows: int, n: int, k: int) -> bool:
    """The small-batch tensor-core tier without a way back (fast_mmvq.rs:118-134: 2..16 rows where a type has it). Here: 9..16 rows
    always (the alternative is the prefill GEMM), 3..8 rows on big matrices or from 5 (Q6_K 7) rows on; `_tier` decides for all."""
    if rows > TENSOR_CORE_MAX_ROWS or rows < 3 or not tensor_core_rows_supported(dtype, k):
        return False
    return rows > MMVQ_MAX_BATCH or _tensor_core_pays(dtype, rows, n, k)


class QTensor:
    """Packed GGUF blocks of a `[n, k]` weight on a CUDA device (rows contiguous, then the reference's padding)."""

    def __init__(self, data: torch.Tensor, dtype: GgmlDType, shape: tuple[int, int]):
        n, k = int(shape[0]), int(shape[1])  # a shape read through numpy holds numpy integers
        if k % dtype.block_size:
            # mod.rs:872-884: the last dimension must hold whole blocks
            raise ValueError(f"quantized tensor last dim {k} is not a multiple of the {dtype.name} block size {dtype.block_size}")
        need = n * dtype.row_bytes(k)
        if data.dtype != torch.uint8 or data.numel() < need:
            raise ValueError(f"{dtype.name} tensor of shape {shape} needs {need} bytes, got {data.numel()} of {data.dtype}")
        self.data, self.dtype, self.shape = data, dtype, (n, k)

    @classmethod
    def from_packed(cls, packed, dtype: GgmlDType, shape: tuple[int, int], device="cuda") -> "QTensor":
        """From host bytes (numpy uint8 or torch CPU tensor), uploaded with the trailing padding."""
        return cls(ops.upload_weights(packed, dtype, device), dtype, shape)

    @classmethod
    def quantize(cls, src: torch.Tensor, dtype: GgmlDType) -> "QTensor":
        """`QTensor::quantize(&tensor, dtype)` (mod.rs:903-918): an f32 `[n, k]` tensor packed on its device by the library's
        quantizer, byte for byte what the reference's host quantizer writes. `k` must hold whole blocks."""
        if src.dim() != 2:
            raise ValueError(f"quantize takes a matrix, got {tuple(src.shape)}")
        n, k = src.shape
        if k % dtype.block_size:
            raise ValueError(f"quantized tensor last dim {k} is not a multiple of the {dtype.name} block size {dtype.block_size}")
        x = src.detach().to(dtype=torch.float32).contiguous()
        if not x.is_cuda:
            x = x.cuda()
        return cls(ops.quantize_weights(x, dtype), dtype, (n, k))

    def dequantize(self, out_dtype: torch.dtype = torch.float32) -> torch.Tensor:
        """`QTensor::dequantize` (mod.rs:920-940): the values as a dense `[n, k]` tensor on the same device."""
        return ops.dequantize(self.dtype, self.data, self.shape[0], self.shape[1], out_dtype)

    def embedding(self, ids: torch.Tensor, out_dtype: torch.dtype = torch.float32) -> torch.Tensor:
        """The rows `ids` names, dequantized: the quantized embedding lookup (crates/inference-quant/src/gguf/mod.rs:546-548)."""
        return ops.get_rows(self.dtype, self.data, ids, self.shape[0], self.shape[1], out_dtype)

    @property
    def storage_size_in_bytes(self) -> int:
        return self.shape[0] * self.dtype.row_bytes(self.shape[1])

    def packed_bytes(self) -> torch.Tensor:
        """The blocks without the padding."""
        return self.data[: self.storage_size_in_bytes]

    @property
    def device(self) -> torch.device:
        return self.data.device


class QMatMul:
    """`y = x @ W^T` for a quantized `W`; x `[..., k]` contiguous -> y `[..., n]` in x's dtype (mod.rs:1625-1647)."""

    def __init__(self, qtensor: QTensor):
        self.qtensor = qtensor

    @classmethod
    def from_qtensor(cls, qtensor: QTensor) -> "QMatMul":
        return cls(qtensor)

    def forward(self, xs: torch.Tensor, act_quant: int = ops.ACT_QUANT_Q8_1) -> torch.Tensor:
        w = self.qtensor
        n, k = w.shape
        y = kl.host().forward(w.dtype, w.data, n, k, xs, act_quant, _tier(w.dtype, xs.numel() // k, n, k, act_quant))
        if y is not None:
            return y
        # what the native path declines as it stands: errors among them
        if xs.dim() < 2:
            raise ValueError(f"input tensor has only one dimension {tuple(xs.shape)}")
        if not xs.is_contiguous():
            raise ValueError(f"input tensor is not contiguous {tuple(xs.shape)}")
        if xs.shape[-1] != k:
            raise ValueError(f"input tensor {tuple(xs.shape)} incompatible with {(n, k)}")
        if xs.device != w.device:
            raise ValueError(f"input on {xs.device}, weights on {w.device}")
        x2 = xs.reshape(-1, k)
        y = _forward_rows(w, x2, act_quant)
        return y.reshape(*xs.shape[:-1], n)

    __call__ = forward


def prefers_mmvq(rows: int) -> bool:
    """Decode GEMV for up to MMVQ_MAX_BATCH rows where the tensor-core tier does not take them, the prefill GEMM above
    (fast_mmvq.rs:96-134)."""
    return rows <= MMVQ_MAX_BATCH


def _tier_overtakes(dtype: GgmlDType, rows: int, n: int, k: int) -> bool:
    """2..8 rows beyond that rule on which the tier's two launches cost less than the dp4a GEMV, if it takes the weights as they lie.
    The tier takes 6 us at least and hardly grows with the rows; the GEMV starts at 3.3 and grows with rows * n * k, the faster the
    wider the rows are. GEMV / tier, us, weights out of HBM, on both sides of the lines: Q4_K k = 1024 3 rows 12288 7.47 / 7.66, 16384
    8.56 / 8.19, 4 rows 8192 6.26 / 7.16, 12288 8.43 / 7.69; k = 2048 3 rows 4096 6.58 / 7.14, 8192 8.79 / 8.48; k = 4096 3 rows 1024
    6.76 / 6.75, 2048 7.69 / 7.06. Q8_0 k = 1024 3 rows 12288 8.52 / 9.02, 16384 10.0 / 9.78; k = 4096 3 rows 1024 7.19 / 8.24, 2048
    8.10 / 8.07; even counts cost its GEMV more, 4 rows k = 512 12288 5.82 / 7.03, k = 1024 4096 6.00 / 6.38, 6144 6.86 / 6.87, k = 1536
    2048 6.60 / 6.17. Q6_K k = 2048 3 rows 8192 9.80 / 11.0, 12288 13.0 / 13.0, 5 rows 1024 6.67 / 6.42, 4096 8.98 / 8.12; k = 4096 3
    rows 2048 8.12 / 8.29, 4096 10.6 / 10.9. 2 rows, at any size: Q4_K 8.28 / 6.16 (512 x 256) to 82 / 50 (4096 x 65536), Q8_0 6.66 / 5.85
    (256 x 256) to 179 / 79 (6144 x 65536), Q6_K 10.8 / 6.25 (2048 x 256) to 203 / 99; 6 rows of Q6_K 7.99 / 6.41 to 358 / 100."""
    if not tensor_core_rows_supported(dtype, k):
        return False
    if rows == 2 or rows >= 6:
        return True
    narrow = k < 3072
    if dtype == GgmlDType.Q6K:
        least = 9 if narrow and rows < 5 else 4
    elif dtype == GgmlDType.Q4K:
        least = 5 if narrow else 2
    elif rows == 3:
        least = 5 if narrow else 3
    else:
        least = 5 if k < 1024 else (3 if k < 1536 else 2)
    return rows * n * k >= least << 23


def _tier(dtype: GgmlDType, rows: int, n: int, k: int, act_quant: int) -> int:
    """Which kernel serves a row count: 0 the decode GEMV, 1 the small-batch tensor-core kernel, 2 the tile GEMM, 3 the small-batch
    kernel or else the GEMV (weights off the 16-byte boundaries that the former needs)."""
    if rows <= 1:
        return 0
    if rows > TENSOR_CORE_MAX_ROWS:
        return 2
    if act_quant == ops.ACT_QUANT_Q8_1:
        if prefers_tensor_core_rows(dtype, rows, n, k):
            return 1
        if prefers_mmvq(rows) and _tier_overtakes(dtype, rows, n, k):
            return 3
    return 0 if prefers_mmvq(rows) else 2


def _forward_rows(w: QTensor, x: torch.Tensor, act_quant: int) -> torch.Tensor:
    """The same kernels by the same rule where the native path declines a call: empty inputs, wide batches whose K is not a multiple
    of the tile GEMM's step, the CPU format on widths it is not defined for, and whatever the kernels' own checks refuse."""
    n, k = w.shape
    rows = x.shape[0]
    if rows == 0:
        return torch.empty((0, n), dtype=x.dtype, device=x.device)
    tier = _tier(w.dtype, rows, n, k, act_quant)
    if tier in (1, 3):
        try:
            return ops.gemv_tc(w.dtype, w.data, x, n)
        except kl.KernelLibraryError as exc:
            if tier == 1 or exc.status != -1:  # -1: weights off the 16-byte boundaries
                raise
    if tier == 2 and k % 64 == 0:
        if x.dtype == torch.float32:
            # the tensor-core path takes 16-bit activations; f32 inputs are narrowed as the reference narrows them for
            # its own CUDA path (crates/inference-quant/src/gguf/mod.rs:667-691 keeps bf16 when given bf16)
            return ops.gemm(w.dtype, w.data, x.to(torch.bfloat16), n).to(torch.float32)
        return ops.gemm(w.dtype, w.data, x, n)
    if tier != 2 and k % 128 == 0:
        try:
            return ops.gemv(w.dtype, w.data, x, n, act_quant=act_quant)
        except kl.KernelLibraryError as exc:
            # no staged plan for this call (weights not 16-byte aligned, the simple kernel forced, no ring that fits): the
            # library can still serve Q8_1 activations in two launches
            if act_quant != ops.ACT_QUANT_Q8_1 or exc.status != -1:
                raise
    elif tier != 2 and act_quant != ops.ACT_QUANT_Q8_1:
        raise ValueError(f"the CPU path's activation format needs K a multiple of 128, got {k}")
    # the reference's own two-launch protocol, in batches of its launcher
    outs = []
    for i in range(0, rows, MMVQ_MAX_BATCH):
        xb = x[i:i + MMVQ_MAX_BATCH].contiguous()
        vy = ops.quantize_q8_1(xb, pad(k, MATRIX_ROW_PADDING))
        outs.append(ops.mmvq_plain(w.dtype, w.data, vy, n, k, xb.shape[0], x.dtype))
    return outs[0] if len(outs) == 1 else torch.cat(outs, 0)


class GgufMatMul:
    """The `QuantMethod` of GGUF weights: forward = quantized matmul plus optional bias
    (crates/inference-quant/src/gguf/mod.rs:92-100,513-571; trait crates/inference-quant/src/lib.rs:2014-2291)."""

    def __init__(self, w: QMatMul, b: torch.Tensor | None = None):
        self.w, self.b = w, b

    @classmethod
    def from_qtensor(cls, q: QTensor, bias: torch.Tensor | None = None) -> "GgufMatMul":
        return cls(QMatMul.from_qtensor(q), bias)

    def quantized_act_type(self):
        return None  # CUDA GGUF takes activations as they are (gguf/mod.rs:667-691)

    def dtype_and_device(self):
        return self.w.qtensor.dtype, self.w.qtensor.device

    def is_distributed(self) -> bool:
        return False

    def get_qtensor(self) -> QTensor:
        return self.w.qtensor

    def forward_raw(self, x: torch.Tensor) -> torch.Tensor:
        y = self.w.forward(x)
        return y if self.b is None else y + self.b.to(y.dtype)

    def forward(self, x: torch.Tensor) -> torch.Tensor:
        return self.forward_raw(x)

    __call__ = forward

