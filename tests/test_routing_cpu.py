"""Row-count routing of the operator mirror (host logic only): which kernel `QMatMul` picks for a shape, mirroring
`prefers_mmvq` / `TENSOR_CORE_MAX_ROWS` of the reference (crates/inference-quant/src/gguf/fast_mmvq.rs:84-134)."""
import numpy as np
import pytest
import torch

from inference_rs_b200 import GgmlDType, QMatMul, QTensor
from inference_rs_b200 import qmatmul as qm

LLAMA_SHAPES = [(4096, 6144), (4096, 4096), (4096, 28672), (14336, 4096), (4096, 128256)]  # (k, n)


@pytest.mark.parametrize("dtype", [GgmlDType.Q4K, GgmlDType.Q6K, GgmlDType.Q8_0])
def test_rows_9_to_16_take_the_tensor_core_tier_and_1_2_never_without_a_way_back(dtype):
    for k, n in LLAMA_SHAPES:
        for rows in (1, 2):
            assert not qm.prefers_tensor_core_rows(dtype, rows, n, k) and qm.prefers_mmvq(rows)
        for rows in range(9, 17):
            assert qm.prefers_tensor_core_rows(dtype, rows, n, k)
        assert not qm.prefers_tensor_core_rows(dtype, 17, n, k) and not qm.prefers_mmvq(17)


def test_rows_3_to_8_that_take_the_tier_without_a_way_back():
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


# (type, rows, k, rows of the matrix at which the GEMV is still the faster one, at which the tier is): measured on B200
@pytest.mark.parametrize("dtype,rows,k,gemv,tier", [
    (GgmlDType.Q4K, 3, 512, 16383, 16384), (GgmlDType.Q4K, 3, 1024, 12288, 16384), (GgmlDType.Q4K, 4, 1024, 8192, 12288),
    (GgmlDType.Q4K, 3, 2048, 4096, 8192), (GgmlDType.Q4K, 4, 2048, 2048, 6144), (GgmlDType.Q4K, 3, 4096, 1024, 2048),
    (GgmlDType.Q8_0, 4, 512, 12288, 16384), (GgmlDType.Q8_0, 3, 1024, 12288, 16384), (GgmlDType.Q8_0, 4, 1024, 4096, 6144),
    (GgmlDType.Q8_0, 3, 4096, 1024, 2048), (GgmlDType.Q6K, 3, 2048, 8192, 12288), (GgmlDType.Q6K, 4, 2048, 6144, 12288),
    (GgmlDType.Q6K, 5, 2048, 1024, 4096), (GgmlDType.Q6K, 3, 4096, 2048, 4096)])
def test_3_to_5_rows_leave_the_gemv_where_the_tier_is_not_slower(dtype, rows, k, gemv, tier):
    assert qm._tier(dtype, rows, gemv, k, qm.ops.ACT_QUANT_Q8_1) == 0
    assert qm._tier(dtype, rows, tier, k, qm.ops.ACT_QUANT_Q8_1) in (1, 3)


@pytest.mark.parametrize("dtype", [GgmlDType.Q4K, GgmlDType.Q6K, GgmlDType.Q8_0])
def test_the_kernel_of_each_row_count(dtype):
    q8_1, cpu = qm.ops.ACT_QUANT_Q8_1, qm.ops.ACT_QUANT_CPU
    for k, n in LLAMA_SHAPES:
        assert [qm._tier(dtype, r, n, k, q8_1) for r in (1, 2)] == [0, 3]
        assert all(qm._tier(dtype, r, n, k, q8_1) in (1, 3) for r in range(6, 9)) and {qm._tier(dtype, r, n, k, q8_1) for r in range(9, 17)} == {1}
        assert qm._tier(dtype, 17, n, k, q8_1) == 2
        assert [qm._tier(dtype, r, n, k, cpu) for r in (2, 8, 9)] == [0, 0, 2]
    assert qm._tier(dtype, 2, 4096, 4096 + 128, q8_1) == 0 and qm._tier(dtype, 12, 4096, 4096 + 128, q8_1) == 2
