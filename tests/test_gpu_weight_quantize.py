"""GPU parity of the weight quantizers, dequantizers and the row gather (`b200q_quantize`, `b200q_dequantize`,
`b200q_get_rows`), through the C ABI: packed bytes identical to the oracle's (the reference CPU quantizer's default mode),
dequantized values identical to the oracle's `to_float`, and, for the two types the reference has device quantizers for,
identical to those (oracle/_ref) as well."""
import numpy as np
import pytest
import torch

from oracle import kquants as kq
from oracle import refkernels as rk

from inference_rs_b200 import QMatMul, QTensor, ops
from gpu_util import DT, TYPES, as_f32_numpy, assert_device_ok, seeded_acts, seeded_weights

pytestmark = pytest.mark.gpu


def edge_rows(k):
    """Rows the searches treat specially: zeros, one spike, constants of either sign, tiny and huge magnitudes, ties."""
    rng = np.random.default_rng(3)
    rows = [np.zeros(k), np.full(k, 0.25), np.full(k, -0.25), rng.standard_normal(k) * 1e-20, rng.standard_normal(k) * 1e4,
            np.where(np.arange(k) % 256 == 7, 3.0, 0.0), np.arange(k) % 16 - 7.5, rng.standard_normal(k) * 0.02,
            np.abs(rng.standard_normal(k)) * 0.02, -np.abs(rng.standard_normal(k)) * 0.02]
    return np.stack(rows).astype(np.float32)


@pytest.mark.parametrize("type_id", TYPES)
def test_packed_bytes_equal_the_oracle(type_id):
    for w in (seeded_weights(512, 1024, 11), edge_rows(1024), seeded_weights(3, 256, 12) * 50.0):
        mine = ops.quantize_weights(torch.from_numpy(w).cuda(), DT[type_id])
        torch.cuda.synchronize()
        want = kq.quantize(type_id, w).reshape(-1)
        got = mine.cpu().numpy()[: want.size]
        bad = np.nonzero(got != want)[0]
        if bad.size:
            blk, bb = bad[0] // kq.BLOCK_BYTES[type_id], kq.BLOCK_BYTES[type_id]
            raise AssertionError(f"{kq.TYPE_NAMES[type_id]}: {bad.size} bytes differ, first at {bad[:8].tolist()}; block {blk}: got "
                                 f"{got[blk * bb:(blk + 1) * bb].tolist()} want {want[blk * bb:(blk + 1) * bb].tolist()}")
        assert not mine.cpu().numpy()[want.size:].any(), "the padding behind the blocks must be zero"
    assert_device_ok()


@pytest.mark.parametrize("type_id", TYPES)
def test_config_1_weights_quantized_by_the_library(type_id):
    """f32 4096 x 4096 ~N(0, 0.02), seed 0, packed by the product's own quantizer; the bytes equal the
    oracle's and the matmul on them is within the stated tolerance of the CPU path."""
    g = torch.Generator().manual_seed(0)
    w = (torch.randn(4096, 4096, generator=g) * 0.02)
    q = QTensor.quantize(w.cuda(), DT[type_id])
    torch.cuda.synchronize()
    want = kq.quantize(type_id, w.numpy())
    assert np.array_equal(q.packed_bytes().cpu().numpy(), want.reshape(-1))
    x = seeded_acts(4, 4096, 1, torch.float32)
    y = QMatMul.from_qtensor(q).forward(x.cuda(), act_quant=ops.ACT_QUANT_CPU)
    cpu = kq.matmul(type_id, x.numpy(), want, 4096)
    assert (np.abs(as_f32_numpy(y) - cpu) <= 1e-3 + 1e-2 * np.abs(cpu)).all()
    assert_device_ok()


@pytest.mark.parametrize("type_id", [kq.Q6_K, kq.Q8_0])
def test_packed_bytes_equal_the_reference_device_quantizers(type_id):
    if not rk.available():
        pytest.skip("oracle/_ref was not built")
    w = torch.from_numpy(seeded_weights(300, 2048, 13)).cuda()
    mine = ops.quantize_weights(w, DT[type_id])
    theirs, _ = (rk.encode_q6_k if type_id == kq.Q6_K else rk.encode_q8_0)(w)
    torch.cuda.synchronize()
    if type_id == kq.Q8_0:
        assert torch.equal(mine[: theirs.numel()], theirs.reshape(-1))
    else:
        # the reference's device Q6_K quantizer follows its fused-multiply-add mode (Quantizer::IkLlama), this library's the
        # default one: theirs must equal the oracle in that mode, this library's the oracle in the default mode
        assert np.array_equal(theirs.cpu().numpy().reshape(-1), kq.quantize(type_id, w.cpu().numpy(), mode=kq.IKLLAMA).reshape(-1))
        assert np.array_equal(mine.cpu().numpy()[: theirs.numel()], kq.quantize(type_id, w.cpu().numpy()).reshape(-1))


@pytest.mark.parametrize("type_id", TYPES)
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.float16])
def test_dequantize_and_row_gather(type_id, dtype):
    n, k = 257, 768
    packed = kq.quantize(type_id, seeded_weights(n, k, 14))
    q = QTensor.from_packed(packed, DT[type_id], (n, k))
    want = torch.from_numpy(kq.dequantize(type_id, packed, k)).to(dtype)
    got = q.dequantize(dtype)
    torch.cuda.synchronize()
    assert torch.equal(got.cpu(), want)
    ids = torch.tensor([[0, 256, 5], [5, 17, 255]], dtype=torch.int64)
    rows = q.embedding(ids, dtype)
    torch.cuda.synchronize()
    assert rows.shape == (2, 3, k) and torch.equal(rows.cpu(), want[ids])
    assert_device_ok()


def test_quantize_errors_and_bad_row_ids():
    from inference_rs_b200 import kernel_library as kl
    with pytest.raises(ValueError, match="not a multiple"):
        QTensor.quantize(torch.zeros(4, 100), DT[kq.Q4_K])
    with pytest.raises(TypeError):
        ops.quantize_weights(torch.zeros(4, 256, dtype=torch.float16, device="cuda"), DT[kq.Q4_K])
    q = QTensor.quantize(torch.from_numpy(seeded_weights(8, 256, 1)).cuda(), DT[kq.Q8_0])
    rows = q.embedding(torch.tensor([1, 99]))
    torch.cuda.synchronize()
    assert not rows[1].any() and rows[0].any()
    st = kl.device_status()
    assert st[0] == 6 and st[2] == 1, st  # code 6: row id outside the table; detail = position of the id
    kl.check(kl.library().b200q_reset_device_status(), "reset")


def search_rows(k):
    """Distributions that crowd the candidates of the scale searches together, or whose products leave the normal f32 range (above
    1e6 the block scale itself no longer fits f16)."""
    rng = np.random.default_rng(5)
    g = rng.standard_normal((8, k))
    return np.concatenate([g * s for s in (1e-36, 1e-30, 1e-18, 1e-12, 1e-6, 1.0, 1e4)] +
                          [rng.standard_t(1.5, (16, k)), rng.uniform(0, 1, (8, k)), 1.0 + g * 1e-6, -3.0 + g * 1e-3, np.round(g * 2), np.sign(g),
                           g * (rng.random((8, k)) < 0.05), np.repeat(g[:, ::32], 32, axis=1)]).astype(np.float32)


@pytest.mark.parametrize("type_id", TYPES)
@pytest.mark.parametrize("case", ["search", "tail", "unaligned"])
def test_register_searches_pick_the_oracles_candidate(type_id, case):
    """Levels kept as floats, and the sub-blocks that fall back to the integer form (search); block counts that fill neither a CTA
    nor a warp (tail); an input on a 4-byte and an output on a 2-byte boundary (unaligned)."""
    from inference_rs_b200 import kernel_library as kl
    if case == "search":
        w = search_rows(1024)
    else:
        w = seeded_weights(7 if case == "tail" else 33, 256, 21)
    n, k = w.shape
    want = kq.quantize(type_id, w).reshape(-1)
    shift = 2 if case == "unaligned" else 0
    src = torch.zeros(n * k + 4, device="cuda")
    x = src[1:1 + n * k] if case == "unaligned" else src[:n * k]
    x.copy_(torch.from_numpy(w.reshape(-1)))
    out = torch.zeros(want.size + shift + 16, dtype=torch.uint8, device="cuda")
    kl.check(kl.library().b200q_quantize(int(DT[type_id]), x.data_ptr(), out.data_ptr() + shift, n * k, torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    got = out.cpu().numpy()
    assert np.array_equal(got[shift:shift + want.size], want)
    assert not got[:shift].any() and not got[shift + want.size:].any(), "bytes outside the blocks were written"


@pytest.mark.parametrize("type_id", TYPES)
@pytest.mark.parametrize("n,k", [(1, 256), (3, 2816), (129, 256)])
def test_dequantize_rows_of_any_width_and_alignment(type_id, n, k):
    from inference_rs_b200 import kernel_library as kl
    packed = kq.quantize(type_id, seeded_weights(n, k, 15))
    want = kq.dequantize(type_id, packed, k)
    flat = packed.reshape(-1)
    for w_off, o_off in ((0, 0), (2, 0), (1, 0), (0, 4)):
        buf = torch.zeros(flat.size + 64, dtype=torch.uint8, device="cuda")
        buf[w_off:w_off + flat.size].copy_(torch.from_numpy(flat.copy()))
        out = torch.zeros(n * k + 8, device="cuda")
        kl.check(kl.library().b200q_dequantize(int(DT[type_id]), 0, buf.data_ptr() + w_off, out.data_ptr() + o_off, n, k,
                                               torch.cuda.current_stream().cuda_stream))
        torch.cuda.synchronize()
        got = out.cpu().numpy()
        assert np.array_equal(got[o_off // 4:o_off // 4 + n * k].reshape(n, k), want)
        assert not got[:o_off // 4].any() and not got[o_off // 4 + n * k:].any()


def test_q8_0_blocks_with_nan_and_infinite_values():
    """The reference's maximum starts from 0 and passes NaNs over (quantized/mod.rs:43-56): a block of NaNs alone has the scale 0."""
    w = seeded_weights(2, 160, 31)
    w[0, :32] = np.nan
    w[0, 32:36] = np.nan
    w[0, 64] = np.inf
    w[0, 96:127] = np.nan
    w[1, 5] = -np.inf
    w[1, 128:] = np.nan
    got = ops.quantize_weights(torch.from_numpy(w).cuda(), DT[kq.Q8_0])
    want = kq.quantize(kq.Q8_0, w).reshape(-1)
    assert np.array_equal(got.cpu().numpy()[: want.size], want)
