"""Row-count routing of the operator mirror (host logic only): which kernel `QMatMul` picks for a shape, mirroring
`prefers_mmvq` / `TENSOR_CORE_MAX_ROWS` of the reference (crates/inference-quant/src/gguf/fast_mmvq.rs:84-134)."""
import numpy as np
import pytest
import torch

from inference_rs_b200 import GgmlDType, QMatMul, QTensor
from inference_rs_b200 import qmatmul as qm

LLAMA_SHAPES = [(4096, 6144), (4096, 4096), (4096, 28672), (14336, 4096), (4096, 128256)]  # (k, n)


@pytest.mark.parametrize("dtype", [GgmlDType.Q4K, GgmlDType.Q6K, GgmlDType.Q8_0])
def test_rows_1_2_stay_on_the_gemv_and_9_to_16_take_the_tensor_core_tier(dtype):
    for k, n in LLAMA_SHAPES:
        for rows in (1, 2):
            assert not qm.prefers_tensor_core_rows(dtype, rows, n, k) and qm.prefers_mmvq(rows)
        for rows in range(9, 17):
            assert qm.prefers_tensor_core_rows(dtype, rows, n, k)
        assert not qm.prefers_tensor_core_rows(dtype, 17, n, k) and not qm.prefers_mmvq(17)


def test_rows_3_to_8_follow_the_measured_crossovers():
    # light unpacking (Q4_K, Q8_0): from 5 rows everywhere, from 3 rows on big matrices
    for dtype in (GgmlDType.Q4K, GgmlDType.Q8_0):
        assert not qm.prefers_tensor_core_rows(dtype, 4, 4096, 4096)
        assert qm.prefers_tensor_core_rows(dtype, 5, 4096, 4096)
        assert qm.prefers_tensor_core_rows(dtype, 3, 28672, 4096) and qm.prefers_tensor_core_rows(dtype, 3, 4096, 14336)
    # Q6_K: from 7 rows everywhere, from 4 rows on big matrices, 3 rows only on the output head
    q6 = GgmlDType.Q6K
    assert not qm.prefers_tensor_core_rows(q6, 6, 4096, 4096) and qm.prefers_tensor_core_rows(q6, 7, 4096, 4096)
    assert qm.prefers_tensor_core_rows(q6, 4, 4096, 14336) and not qm.prefers_tensor_core_rows(q6, 3, 4096, 14336)
    assert qm.prefers_tensor_core_rows(q6, 3, 128256, 4096)


def test_shapes_the_tier_cannot_take_fall_back():
    assert qm.tensor_core_rows_supported(GgmlDType.Q4K, 256) and not qm.tensor_core_rows_supported(GgmlDType.Q4K, 128)
    # Q6_K rows are a multiple of 16 bytes only when K is a multiple of 2048
    assert qm.tensor_core_rows_supported(GgmlDType.Q6K, 14336) and not qm.tensor_core_rows_supported(GgmlDType.Q6K, 4096 + 256)
    assert qm.tensor_core_rows_supported(GgmlDType.Q8_0, 512) and not qm.tensor_core_rows_supported(GgmlDType.Q8_0, 96)
    assert not qm.prefers_tensor_core_rows(GgmlDType.Q6K, 12, 4096, 4096 + 256)


def _without_launches(monkeypatch):
    """The Python form alone, with the kernels' calls recorded instead of made."""
    class Declines:
        def forward(self, *args):
            return None
    seen = []

    def call(name, out):
        def fn(*args, **kw):
            seen.append(name)
            return out(*args)
        return fn
    monkeypatch.setattr(qm.kl, "host", Declines)
    rows = lambda dtype, w, x, n, *a: torch.zeros(x.shape[0], n, dtype=x.dtype)
    for name in ("gemv", "gemv_tc", "gemm"):
        monkeypatch.setattr(qm.ops, name, call(name, rows))
    monkeypatch.setattr(qm.ops, "quantize_q8_1", call("quantize_q8_1", lambda x, kp: x))
    monkeypatch.setattr(qm.ops, "mmvq_plain", call("mmvq_plain", lambda dtype, w, vy, n, k, b, t: torch.zeros(b, n, dtype=t)))
    return seen


@pytest.mark.parametrize("rows,kernel", [(1, "gemv"), (4, "gemv"), (12, "gemv_tc"), (40, "gemm")])
def test_a_call_that_the_native_path_declines_takes_the_same_kernel(monkeypatch, rows, kernel):
    q = QTensor(torch.zeros(16 * 144, dtype=torch.uint8), GgmlDType.Q4K, (np.int64(16), np.int64(256)))
    assert q.shape == (16, 256) and all(type(v) is int for v in q.shape)
    seen = _without_launches(monkeypatch)
    y = QMatMul(q).forward(torch.zeros(rows, 256, dtype=torch.bfloat16))
    assert y.shape == (rows, 16) and seen == [kernel]


def test_wide_batches_off_the_tile_step_go_through_the_two_launch_protocol(monkeypatch):
    q = QTensor(torch.zeros(16 * 102, dtype=torch.uint8), GgmlDType.Q8_0, (16, 96))
    seen = _without_launches(monkeypatch)
    assert QMatMul(q).forward(torch.zeros(20, 96)).shape == (20, 16) and seen == 3 * ["quantize_q8_1", "mmvq_plain"]
    with pytest.raises(ValueError, match="multiple of 128"):
        QMatMul(q).forward(torch.zeros(4, 96), act_quant=qm.ops.ACT_QUANT_CPU)


@pytest.mark.parametrize("rows", [1, 4, 12, 40])
def test_tensors_off_the_gpu_are_named_as_the_error(rows):
    q = QTensor(torch.zeros(16 * 144, dtype=torch.uint8), GgmlDType.Q4K, (16, 256))
    with pytest.raises(ValueError, match="CUDA tensor"):
        QMatMul(q).forward(torch.zeros(rows, 256, dtype=torch.bfloat16))


def test_launchers_name_tensors_off_the_gpu_as_the_error():
    w, acts = torch.zeros(16 * 144, dtype=torch.uint8), torch.zeros(2, 20, 144, dtype=torch.uint8)
    with pytest.raises(ValueError, match="CUDA tensor"):
        qm.ops.mmq(GgmlDType.Q4K, w, acts, 20, 16, 256, torch.bfloat16)
    with pytest.raises(ValueError, match="CUDA tensor"):
        qm.ops.quantize_mmq_q8_1(torch.zeros(20, 256), "DS4")
