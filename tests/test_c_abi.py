"""The C-ABI library loads and exports every symbol include/inferencequant_b200.h declares (no compute here)."""
import os
import re

import pytest

import inference_rs_b200 as pkg
from inference_rs_b200 import kernel_library as kl

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _declared_symbols():
    text = open(os.path.join(ROOT, "include", "inferencequant_b200.h")).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    names = set(re.findall(r"\b((?:launch|b200q)_[A-Za-z0-9_]+)\s*\(", text))
    names |= set(re.findall(r"extern const char (\w+)\[\]", text))
    return names


def test_header_and_loader_agree():
    declared = _declared_symbols()
    assert declared, "no declarations parsed"
    known = set(kl.SYMBOLS) | set(kl.DATA_SYMBOLS)
    assert declared == known, (sorted(declared - known), sorted(known - declared))


def test_library_exports_every_declared_symbol():
    lib = pkg.library()  # raises if any symbol is missing
    for name in _declared_symbols():
        if name in kl.DATA_SYMBOLS:
            continue
        assert getattr(lib, name) is not None
    assert kl.build_id().startswith("b200q-sm100a")
    assert lib.b200q_version().decode().count(".") == 2


def test_missing_library_is_an_error_not_a_fallback(monkeypatch, tmp_path):
    monkeypatch.setattr(kl, "_lib", None)
    monkeypatch.setattr(kl, "HERE", str(tmp_path))
    monkeypatch.delenv("INFERENCE_KERNEL_DIR", raising=False)
    with pytest.raises(kl.KernelLibraryError, match="no CPU fallback"):
        kl.library()


def test_kernel_dir_env_takes_precedence(monkeypatch, tmp_path):
    monkeypatch.setenv("INFERENCE_KERNEL_DIR", str(tmp_path))
    assert kl.search_paths()[0] == os.path.join(str(tmp_path), "sm100a", kl.LIB_NAME)


def test_options_and_errors_round_trip():
    from inference_rs_b200 import ops
    ops.set_option("pdl", 0)
    assert ops.get_option("pdl") == 0
    with pytest.raises(kl.KernelLibraryError, match="unknown option"):
        ops.set_option("no_such_option", 1)
    assert ops.get_option("sm_count") > 0
    # the L2 prefetch size follows the launch mode until it is set, and again after -1
    assert ops.get_option("l2_prefetch_bytes") == 256 * 1024
    ops.set_option("pdl", 1)
    assert ops.get_option("l2_prefetch_bytes") == 64 * 1024
    ops.set_option("l2_prefetch_bytes", 4100)
    assert ops.get_option("l2_prefetch_bytes") == 4096
    ops.set_option("l2_prefetch_bytes", -1)
    ops.set_option("pdl", 0)
    assert ops.get_option("l2_prefetch_bytes") == 256 * 1024


@pytest.mark.parametrize("tag,k,n,b", [("Q4K", 4096, 4096, 1), ("Q6K", 14336, 4096, 4), ("Q8_0", 4096, 128256, 8),
                                       ("Q6K", 768, 100, 1), ("Q4K", 28672, 8192, 1)])
def test_gemv_plans_respect_hardware_limits(tag, k, n, b):
    from inference_rs_b200 import ops
    dt = pkg.GgmlDType[tag]
    plan = ops.gemv_plan(dt, k, n, b)
    if not plan["staged"]:
        return
    assert plan["smem"] <= 227 * 1024
    assert 2 <= plan["stages"] <= 16
    assert plan["rows_per_stage"] % plan["row_align"] == 0
    items = k // 128
    assert plan["warps_per_row"] * 32 * plan["items_per_lane"] >= items
    assert plan["stage_bytes"] >= plan["rows_per_stage"] * dt.row_bytes(k) + 16
    assert (plan["row_align"] * dt.row_bytes(k)) % 16 == 0
    assert 1 <= plan["grid"] <= 148


def test_short_launches_are_split_in_whole_stages_where_few_ctas_get_the_remainder():
    """The row partition's unit: a whole ring stage for ffn_gate / ffn_up of the 8B model (3 stages per CTA, 4 CTAs with a
    fourth), the 16-byte-aligned unit where half of the CTAs would get the extra stage (ffn_down) and for long launches
    (the output head), where a ragged last stage is amortised."""
    from inference_rs_b200 import ops
    if ops.get_option("sm_count") != 148:
        pytest.skip("the expectations are for 148 SMs")
    gate = ops.gemv_plan(pkg.GgmlDType.Q4K, 4096, 14336, 1)
    assert gate["staged"] and gate["row_align"] == gate["rows_per_stage"]
    down = ops.gemv_plan(pkg.GgmlDType.Q6K, 14336, 4096, 1)
    assert down["staged"] and down["row_align"] < down["rows_per_stage"]
    head = ops.gemv_plan(pkg.GgmlDType.Q6K, 4096, 128256, 1)
    assert head["staged"] and head["row_align"] < head["rows_per_stage"]
    small = ops.gemv_plan(pkg.GgmlDType.Q4K, 4096, 4096, 1)
    assert small["staged"] and small["row_align"] < small["rows_per_stage"]


def test_trace_buffer_needs_a_trace_build():
    """The launch timelines are a build option; the default library says so instead of silently ignoring the buffer."""
    import ctypes
    lib = pkg.library()
    assert lib.b200q_set_trace_buffer(None, 0) == 0
    rc = lib.b200q_set_trace_buffer(ctypes.c_void_p(4096), 4)
    assert rc in (0, -1)  # B200Q_ERR_UNSUPPORTED; 0 only in a library built with -DB200Q_GEMV_TRACE=1
    if rc != 0:
        assert b"B200Q_GEMV_TRACE" in lib.b200q_last_error()
    lib.b200q_set_trace_buffer(None, 0)


def test_native_call_path_binds_to_the_library():
    host = kl.host()
    assert set(host.symbols()) <= set(kl.SYMBOLS)
    # arguments it does not take as they stand are declined, never launched
    assert host.gemv(12, None, None, 16, None, 0) is None
    assert host.forward(12, None, 16, 256, None, 0, 0) is None
    assert host.gemv_group([12], [None], None, [16], None, 0) is None


def test_the_expanded_form_is_chosen_where_it_is_not_slower():
    """b200q_gemm_workspace_bytes: 0 = the single launch. Up to 128 rows it stays where enough SMs have a tile of 128 weight rows (the
    measured crossovers, of 148 SMs), up to 256 where every SM has one."""
    lib = pkg.library()
    q8, q4, q6 = 8, 12, 14
    pair = lambda t, m, n, k: lib.b200q_gemm_workspace_bytes(t, m, n, k) > 0
    for t, k, n in ((q4, 4096, 11776), (q8, 4096, 12672), (q6, 4096, 14208), (q4, 2048, 15744), (q8, 512, 15744), (q6, 2048, 18816)):
        assert lib.b200q_gemm_workspace_bytes(t, 128, n, k) in (0, 2 * n * k)
        assert pair(t, 17, n - 256, k) and pair(t, 128, n - 256, k), (t, n, k)
        assert not pair(t, 17, n + 128, k) and not pair(t, 128, n + 128, k), (t, n, k)
        assert pair(t, 257, n + 128, k) and pair(t, 8192, n, k)
    for t in (q8, q4, q6):
        assert pair(t, 129, 18816, 4096) and not pair(t, 256, 18945, 4096) and pair(t, 257, 28672, 4096)
    # rows that cannot be staged are expanded by every tile from byte loads: the single launch is the slower one at any size
    assert pair(q8, 17, 28672, 4160) and pair(q6, 17, 28672, 5120)
    assert lib.b200q_gemm_workspace_bytes(q4, 40, 64, 100) == 0


@pytest.mark.parametrize("content", [None, b"not a library"])
def test_without_the_native_call_path_calls_are_left_to_python(monkeypatch, tmp_path, content):
    kl.library()
    monkeypatch.setattr(kl, "_host", None)
    monkeypatch.setattr(kl, "HERE", str(tmp_path))
    if content is not None:
        (tmp_path / "lib").mkdir()
        (tmp_path / "lib" / kl.HOST_LIB_NAME).write_bytes(content)
    with pytest.warns(RuntimeWarning, match="native call path"):
        host = kl.host()
    assert kl.host() is host and host.forward(1, 2) is None and host.gemv() is None
