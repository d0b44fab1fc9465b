"""Host-side logic and the C-ABI surface, without a GPU: group parsing, shape guards, symbol
export, argument validation that returns before any CUDA call, and the loud failure modes."""
from __future__ import annotations

import ctypes
import re
from pathlib import Path

import pytest
import torch

ROOT = Path(__file__).resolve().parent.parent


def test_group_names_round_trip():
    from braid_b200.quant import GROUPS, parse_groups
    assert parse_groups("") == frozenset()
    assert parse_groups(None) == frozenset()
    assert parse_groups("mlp") == {"mlp"}
    assert parse_groups("mlp, attn") == {"mlp", "attn"}
    assert parse_groups(["gdn", "head"]) == {"gdn", "head"}
    assert parse_groups("all") == frozenset(GROUPS)


def test_an_unknown_group_raises():
    from braid_b200.quant import parse_groups
    with pytest.raises(ValueError, match="unknown quant group"):
        parse_groups("mpl")
    with pytest.raises(ValueError, match="unknown quant group"):
        parse_groups("mlp,attention")


def test_public_names_match_the_reference_module():
    """Everything other reference modules import from braid.model.quant exists here."""
    from braid_b200 import quant
    for name in ("GROUPS", "parse_groups", "FP8", "FP8_MAX", "EPS", "FP8Weight", "quantize_weight",
                 "warm_fused", "fused_state", "quantize_act", "fp8_matmul", "fp8_linear", "linear",
                 "project", "maybe_quantize", "_act_scale", "_weight_scale", "_CAST_CHUNK_BYTES"):
        assert hasattr(quant, name), name
    assert quant.FP8 is torch.float8_e4m3fn and quant.FP8_MAX == 448.0 and quant.EPS == 1e-12


def test_weight_quantization_on_cpu_follows_the_reference_spelling(golden):
    """Load-time work keeps the torch spelling; on a CPU it reproduces the golden weight exactly."""
    from _util import from_bits16
    from braid_b200.quant import FP8Weight, maybe_quantize, quantize_weight
    import numpy as np
    w = from_bits16(golden["weight_w"])
    fw = quantize_weight(w)
    assert isinstance(fw, FP8Weight) and fw.shape == (256, 128) and fw.nbytes == 256 * 128 + 4
    assert fw.scale.shape == (1, 1) and fw.scale.dtype is torch.float32
    assert np.array_equal(fw.data.view(torch.uint8).numpy(), golden["weight_q"])
    assert int(fw.scale.view(torch.int32).item()) & 0xFFFFFFFF == int(golden["weight_scale"].reshape(-1)[0])
    # banding invariance (tests/test_quant.py:81-96)
    from braid_b200 import quant as Q
    old = Q._CAST_CHUNK_BYTES
    Q._CAST_CHUNK_BYTES = 128 * 4 * 3
    try:
        banded = quantize_weight(w)
    finally:
        Q._CAST_CHUNK_BYTES = old
    assert torch.equal(banded.data.view(torch.uint8), fw.data.view(torch.uint8))
    assert maybe_quantize(w, False) is w
    z = quantize_weight(torch.zeros(64, 32, dtype=torch.bfloat16))
    assert torch.isfinite(z.data.float()).all() and (z.scale > 0).all()
    for a in (w, -w.abs(), w * 100):
        assert torch.equal(Q._weight_scale(a), Q._act_scale(a))


@pytest.mark.parametrize("shape", [(30, 256), (512, 250)])
def test_shapes_the_gemm_cannot_take_are_refused(shape):
    from braid_b200.quant import maybe_quantize, quantize_weight
    w = torch.randn(*shape, dtype=torch.bfloat16)
    with pytest.raises(ValueError, match="multiples of 16"):
        quantize_weight(w)
    assert maybe_quantize(w, True) is w


def test_the_library_exports_every_declared_symbol(lib):
    """Each `bq_*` function declared in include/braid_b200.h resolves in the built library and has
    a ctypes signature."""
    from braid_b200 import _lib
    header = (ROOT / "include" / "braid_b200.h").read_text()
    header = re.sub(r"/\*.*?\*/", "", header, flags=re.S)
    declared = set(re.findall(r"\b(bq_[a-z0-9_]+)\s*\(", header))
    assert declared, "no declarations found"
    assert declared == set(_lib.SIGNATURES), declared ^ set(_lib.SIGNATURES)
    for name in declared:
        assert getattr(lib, name) is not None
    assert lib.bq_version() >= 100
    assert lib.bq_quant_workspace_bytes() == 16
    assert lib.bq_gemm_workspace_bytes(128, 4096, 4096) >= 16


def test_argument_validation_returns_before_any_cuda_call(lib):
    from braid_b200 import _lib
    assert lib.bq_quantize_act(None, 1, 8, None, None, None, 0, None) == _lib.BQ_ERR_BAD_ARG
    assert lib.bq_quantize_act(16, 9, 8, 16, 16, 16, 16, None) == _lib.BQ_ERR_BAD_ARG
    assert lib.bq_quantize_act(16, 1, 0, 16, 16, 16, 16, None) == _lib.BQ_ERR_BAD_ARG
    assert lib.bq_quantize_act(16, 1, 8, 16, 16, None, 0, None) == _lib.BQ_ERR_WORKSPACE
    assert lib.bq_quantize_act(24, 1, 8, 16, 16, 16, 16, None) == _lib.BQ_ERR_UNSUPPORTED
    assert lib.bq_silu_mul_quant(16, 16, 1, 4, 12, 12, 12, 16, 16, 16, 16, None) == _lib.BQ_ERR_UNSUPPORTED
    assert lib.bq_gemm_w8a8(16, 16, 16, 16, 16, 1, 8, 64, 24, 64, 16, 16, None) == _lib.BQ_ERR_UNSUPPORTED
    assert lib.bq_gemm_w8a8(16, 16, 16, 16, 16, 1, 8, 60, 32, 64, 16, 16, None) == _lib.BQ_ERR_UNSUPPORTED
    assert lib.bq_gemm_w8a8(16, 16, 16, 16, 16, 7, 8, 64, 32, 64, 16, 16, None) == _lib.BQ_ERR_BAD_ARG
    assert lib.bq_gemm_w8a8(16, 16, 16, 16, 16, 1, 8, 64, 32, 64, None, 0, None) == _lib.BQ_ERR_WORKSPACE
    # the prefill-size and column-parallel entry points: every check precedes any CUDA call
    assert lib.bq_cast_act(None, 1, 8, 16, 16, None) == _lib.BQ_ERR_BAD_ARG
    assert lib.bq_cast_act(24, 1, 8, 16, 16, None) == _lib.BQ_ERR_UNSUPPORTED
    assert lib.bq_rmsnorm_quant_rows(16, 1, 4, 64, 64, 16, 1e-6, 16, 16, None, 16, 16, None) == _lib.BQ_ERR_BAD_ARG
    assert lib.bq_rmsnorm_quant_rows(16, 1, 4, 60, 64, 16, 1e-6, 16, 16, 16, 16, 16, None) == _lib.BQ_ERR_UNSUPPORTED
    assert lib.bq_rmsnorm_scale(16, 1, 4, 64, 64, 16, 1e-6, None, 64, 16, 16, 16, None) == _lib.BQ_ERR_BAD_ARG
    assert lib.bq_rmsnorm_scale(16, 1, 4, 64, 64, 16, 1e-6, 16, 64, 16, None, 0, None) == _lib.BQ_ERR_WORKSPACE
    assert lib.bq_rmsnorm_scale(16, 1, 4, 62, 64, 16, 1e-6, 16, 64, 16, 16, 16, None) == _lib.BQ_ERR_UNSUPPORTED
    assert lib.bq_gated_rmsnorm_scale(16, 0, 256, 16, 1, 256, 16, 1e-6, 4, 2, 64, 16, 256, 16, 16, 16,
                                      None) == _lib.BQ_ERR_UNSUPPORTED          # head_dim must be 128
    assert lib.bq_silu_mul_dense_scale(16, 16, 1, 4, 16, 16, 16, None, 16, 16, 16, None) == _lib.BQ_ERR_BAD_ARG
    assert lib.bq_silu_mul(16, 16, 1, 4, 12, 12, 12, 16, None) == _lib.BQ_ERR_UNSUPPORTED
    assert lib.bq_sigmoid_mul(16, 16, 1, 4, 16, 16, 16, 0, 0, 16, None) == _lib.BQ_ERR_BAD_ARG
    ptrs = (ctypes.c_void_p * 2)(16, 32)
    bad = (ctypes.c_void_p * 2)(16, None)
    assert lib.bq_word_push(None, 2, ptrs, ptrs, None) == _lib.BQ_ERR_BAD_ARG
    assert lib.bq_word_push(16, 9, ptrs, ptrs, None) == _lib.BQ_ERR_BAD_ARG
    assert lib.bq_word_push(16, 2, bad, ptrs, None) == _lib.BQ_ERR_BAD_ARG
    assert lib.bq_wait_flag_scale(16, 16, 0, 16, 16, 2, 0, 16, None) == _lib.BQ_ERR_BAD_ARG
    assert lib.bq_wait_flag_scale(16, 16, 2, 16, 16, 9, 0, 16, None) == _lib.BQ_ERR_BAD_ARG
    assert lib.bq_cast_act_push(16, 1, 4, 16, 16, None, 2, ptrs, 64, ptrs, 16, 16, None) == _lib.BQ_ERR_BAD_ARG
    assert lib.bq_cast_act_push(16, 1, 4, 12, 16, 16, 2, ptrs, 64, ptrs, 16, 16, None) == _lib.BQ_ERR_UNSUPPORTED
    assert lib.bq_rows_push(16, 1, 4, 16, 16, 2, bad, 64, ptrs, 16, 16, None) == _lib.BQ_ERR_BAD_ARG
    assert lib.bq_rows_push(16, 1, 4, 16, 16, 2, ptrs, 64, ptrs, None, 0, None) == _lib.BQ_ERR_WORKSPACE
    room = lib.bq_quantize_weight_workspace_bytes()
    assert lib.bq_quantize_weight(16, 1, 64, None, 16, 16, room, None) == _lib.BQ_ERR_BAD_ARG
    assert lib.bq_quantize_weight(16, 1, 64, 16, 16, 16, room - 1, None) == _lib.BQ_ERR_WORKSPACE
    assert lib.bq_quantize_weight(16, 1, 68, 16, 16, 16, room, None) == _lib.BQ_ERR_UNSUPPORTED
    assert lib.bq_quantize_weight(24, 1, 64, 16, 16, 16, room, None) == _lib.BQ_ERR_UNSUPPORTED
    assert lib.bq_scratchless_status(None) == _lib.BQ_ERR_BAD_ARG
    assert lib.bq_set_option(b"no_such_option", 1) == _lib.BQ_ERR_BAD_ARG
    assert lib.bq_set_option(b"quant_ring", 1) == _lib.BQ_OK and lib.bq_set_option(b"push_tma", 1) == _lib.BQ_OK
    assert lib.bq_set_option(b"decode_split_k", 0) == _lib.BQ_OK
    for code in range(0, 9):
        assert _lib.status_string(code)
    with pytest.raises(ValueError):
        _lib.check(_lib.BQ_ERR_UNSUPPORTED, "x")
    with pytest.raises(RuntimeError):
        _lib.check(_lib.BQ_ERR_DEVICE_WAIT, "x")


def test_linear_of_few_rows_is_refused_where_an_option_rules_it_out(lib):
    """The one-launch form is the weight-streaming kernel's, with the rings it chooses itself.  Options that send
    the batch to another kernel or force a ring's depth leave the call to the two launches, before any
    CUDA call is made."""
    from braid_b200 import _lib
    ptr, n = (ctypes.c_void_p * 1)(16), (ctypes.c_int64 * 1)(64)

    def rc(M):
        return lib.bq_linear_w8a8(16, 1, M, 64, 1, ptr, ptr, None, 0, ptr, n, n, 16, 16, None)

    for key, value, back, rows in (("stream_max_m", 8, 256, 9), ("decode_wide", 1, -1, 1), ("decode_stages", 2, 0, 1),
                                   ("decode_b_stages", 2, 0, 1), ("decode_b_stages", -1, 0, 1)):
        assert lib.bq_set_option(key.encode(), value) == _lib.BQ_OK
        try:
            assert rc(rows) == _lib.BQ_ERR_UNSUPPORTED, (key, value)
        finally:
            assert lib.bq_set_option(key.encode(), back) == _lib.BQ_OK
    assert rc(17) == _lib.BQ_ERR_UNSUPPORTED


def test_mlp_of_few_rows_is_refused_before_anything_is_launched(lib):
    """Sizes, addresses and options that the two-launch MLP leaves to the separate calls.  Without a device the calls it
    would take end with another error."""
    from braid_b200 import _lib

    def rc(M=2, K=4096, I=12288, N=4096, code=1, down=16, h=16, ldy=None, residual=None, ld_res=0):
        return lib.bq_mlp_w8a8(16, 16, 16, 16, down, 16, 16, 16, residual, ld_res, M, K, I, N, code, h, 16,
                               N if ldy is None else ldy, 16, 16, None)

    for refused in (dict(M=7), dict(M=4, code=0), dict(I=8128), dict(I=12288 + 32), dict(N=4104), dict(down=24), dict(h=8),
                    dict(ldy=4098), dict(ldy=4092), dict(residual=16, ld_res=4092), dict(residual=20, ld_res=4096)):
        assert rc(**refused) == _lib.BQ_ERR_UNSUPPORTED, refused
        sizes = {"M": 2, "I": 12288, "N": 4096, "code": 1, **refused}
        if not set(refused) - {"M", "I", "N", "code"}:
            assert lib.bq_mlp_w8a8_takes(sizes["M"], sizes["I"], sizes["N"], sizes["code"]) == 0, refused
    for bad in (dict(M=0), dict(N=0), dict(code=3), dict(h=None)):
        assert rc(**bad) == _lib.BQ_ERR_BAD_ARG, bad
    for key, value, back in (("stream_max_m", 1, 256), ("decode_wide", 1, -1), ("decode_stages", 2, 0), ("decode_b_stages", 2, 0),
                             ("decode_smem_cap", 65536, 0), ("decode_quant_inside", 0, -1)):
        assert lib.bq_set_option(key.encode(), value) == _lib.BQ_OK
        try:
            assert rc() == _lib.BQ_ERR_UNSUPPORTED and lib.bq_mlp_w8a8_takes(2, 12288, 4096, 1) == 0, key
        finally:
            assert lib.bq_set_option(key.encode(), back) == _lib.BQ_OK


def test_a_missing_library_is_loud(monkeypatch, tmp_path):
    from braid_b200 import _lib, quant
    monkeypatch.setattr(_lib, "_lib", None)
    monkeypatch.setattr(_lib, "LIB_PATH", tmp_path / "libbraid_b200.so")
    monkeypatch.setattr(quant, "_FUSED", None)
    monkeypatch.setattr(quant, "_FUSED_STATE", "not tried")
    with pytest.raises(_lib.LibraryMissing):
        quant.warm_fused(True)
    assert quant.fused_state().startswith("unavailable: LibraryMissing")


def test_native_calls_of_another_torch_are_not_loaded(lib, monkeypatch):
    """The module reads torch's objects by the layout it was compiled with: a file of another torch or Python is
    stale for the build and stays unloaded, also where it would load."""
    from braid_b200 import build, quant
    build.build_host()
    assert build.host_problem() is None
    here = build.host_key()
    monkeypatch.setattr(torch, "__version__", "0.0.1")
    assert here in build.host_problem() and build.host_key() in build.host_problem()
    for name, value in (("_HOST", None), ("_NATIVE", None), ("_FUSED", None), ("_FUSED_STATE", "not tried")):
        monkeypatch.setattr(quant, name, value)
    assert quant.warm_fused(True)
    assert quant._HOST is None and quant._NATIVE is None
    assert quant.fused_state() == f"active, calls from Python: {build.host_problem()}"


def test_the_library_is_built_without_the_native_calls(monkeypatch):
    """No g++ or no torch headers: the library is compiled all the same, and the build says what is missing."""
    import subprocess
    from types import SimpleNamespace
    from braid_b200 import build
    ran = []

    def run(cmd, **kw):
        ran.append(cmd[0])
        if cmd[0] == "g++":
            raise FileNotFoundError("g++")
        return SimpleNamespace(returncode=0, stdout="", stderr="")

    monkeypatch.setattr(subprocess, "run", run)
    with pytest.warns(UserWarning, match="native calls .* g\\+\\+"):
        assert build.build(force=True) == build.LIB
    assert len(ran) == 2 and ran[0].endswith("nvcc") and ran[1] == "g++"


def test_a_build_that_is_current_is_returned(monkeypatch):
    from braid_b200 import build
    monkeypatch.setattr(build, "is_stale", lambda: False)
    monkeypatch.setattr(build, "build_host", lambda force=False: build.HOST)
    assert build.build() == build.LIB


def test_scratch_is_published_after_the_native_calls_know_it(monkeypatch):
    """A second thread that finds a device's scratch without the lock takes its slot from the native
    counter at once, so that has to know the slots by then."""
    from braid_b200 import quant
    found = []

    class Host:
        def set_scratch(self, device, address):
            found.append((device, address, device in quant._scratch))

        def next_slot(self, device):
            return 0

    zeros = torch.zeros
    monkeypatch.setattr(quant, "_HOST", Host())
    monkeypatch.setattr(quant, "_scratch", {})
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    monkeypatch.setattr(torch.cuda, "synchronize", lambda device=None: None)
    monkeypatch.setattr(torch, "zeros", lambda *size, device=None, **kw: zeros(*size, **kw))
    buf = quant._scratch_for(3)
    assert found == [(3, buf.data_ptr(), False)] and quant._scratch == {3: buf}


def test_mlp_whose_input_the_native_quantizer_refuses_takes_the_native_products(monkeypatch):
    """A strided, misaligned or recorded input is quantized outside the native MLP call, which then takes the codes; one
    that it takes as it is is not quantized outside."""
    from braid_b200 import quant
    calls, made = [], []

    class Native:
        def mlp(self, xq, sx, dtype, *rest):
            calls.append((xq, sx))
            return rest[-1] if sx is not None or xq.is_contiguous() else None

    def quantize(x):
        made.append(x)
        return torch.zeros(x.shape).to(quant.FP8), torch.ones(1, 1)

    monkeypatch.setattr(quant, "_NATIVE", Native())
    monkeypatch.setattr(quant, "quantize_act", quantize)
    w = quant.FP8Weight(torch.zeros(32, 32).to(quant.FP8), torch.ones(1, 1), (32, 32))
    wide, out = torch.zeros(4, 64, dtype=torch.bfloat16), torch.zeros(4, 32, dtype=torch.bfloat16)
    assert quant.mlp_forward(wide[:, :32], w, w, w, residual=out) is out
    assert len(calls) == 2 and len(made) == 1 and calls[1][0].dtype is quant.FP8
    assert quant.mlp_forward(wide[:, :32].contiguous(), w, w, w, residual=out) is out
    assert len(calls) == 3 and len(made) == 1


def test_projections_that_the_native_call_refuses_are_offered_once(monkeypatch):
    """An engine in fp32 keeps its gates as `F.linear`: the native call refuses the mixed set, and is not asked again."""
    from braid_b200 import quant
    calls = []

    class Native:
        def project(self, *args):
            calls.append(args)

    monkeypatch.setattr(quant, "_NATIVE", Native())
    monkeypatch.setattr(quant, "_project_mixed", lambda *args: None)
    monkeypatch.setattr(quant, "fp8_matmul_grouped", lambda xq, sx, ws, out_dtype: [torch.zeros(4, w.shape[0]) for w in ws])
    w = quant.FP8Weight(torch.zeros(32, 32).to(quant.FP8), torch.ones(1, 1), (32, 32))
    x = torch.zeros(4, 32)
    pre = quant.QuantizedActivation(x.to(quant.FP8), torch.ones(1, 1), x.shape, x.dtype, x)
    assert [y.shape for y in quant.project(pre, w, torch.zeros(8, 32))] == [(4, 32), (4, 8)] and len(calls) == 1
    assert [y.shape for y in quant.project(pre, w, w)] == [(4, 32), (4, 32)] and len(calls) == 2


def test_cpu_tensors_are_refused_not_emulated():
    from braid_b200 import quant
    x = torch.zeros(4, 16, dtype=torch.bfloat16)
    with pytest.raises(RuntimeError, match="no CPU path"):
        quant.quantize_act(x)
    with pytest.raises(RuntimeError, match="no CPU path"):
        quant.silu_mul_quant(x, x)
    fw = quant.quantize_weight(torch.randn(16, 16, dtype=torch.bfloat16))
    with pytest.raises(RuntimeError, match="no CPU path"):
        quant.fp8_matmul(x.to(quant.FP8), torch.ones(1, 1), fw)
    # weights left in bf16 never touch the kernels
    w = torch.randn(8, 16, dtype=torch.bfloat16)
    assert torch.equal(quant.project(x, w)[0], torch.nn.functional.linear(x, w))
    assert torch.equal(quant.linear(x, w), torch.nn.functional.linear(x, w))


def test_the_product_package_never_imports_the_oracle():
    for path in (ROOT / "braid_b200").rglob("*.py"):
        text = path.read_text()
        assert not re.search(r"^\s*(from|import)\s+oracle\b", text, flags=re.M), path


def test_install_into_rebinds_a_reference_shaped_module():
    """`install_into` on a stand-in with the reference's attribute names (no reference needed)."""
    import sys
    import types
    from braid_b200 import quant
    from braid_b200.integrate import adopt_weight, install_into
    ref = types.ModuleType("fake_ref_quant")
    for name in ("quantize_act", "fp8_matmul", "fp8_linear", "linear", "project", "warm_fused",
                 "fused_state", "FP8Weight", "quantize_weight", "maybe_quantize"):
        setattr(ref, name, object())
    user = types.ModuleType("fake_ref_mlp")
    user.fp8_matmul = user.quantize_act = object()
    sys.modules["fake_ref_mlp"] = user
    try:
        done = install_into(ref, extra_modules=("fake_ref_mlp", "not.loaded"))
    finally:
        del sys.modules["fake_ref_mlp"]
    assert ref.fp8_matmul is quant.fp8_matmul and ref.project is quant.project
    assert user.fp8_matmul is quant.fp8_matmul and user.quantize_act is quant.quantize_act
    assert "fake_ref_mlp.fp8_matmul" in done and ref._FUSED_STATE == "active"
    w = quant.quantize_weight(torch.randn(16, 16, dtype=torch.bfloat16))
    assert adopt_weight(w).data is w.data


# -- engine drop-in helpers (host side; the reference install is optional) ---------------------------
def _ref_install():
    from pathlib import Path
    ref = Path(__file__).resolve().parent.parent / "baseline" / "_ref"
    return ref if (ref / "braid" / "model" / "engine.py").exists() else None


def test_text_config_is_the_9b_shape():
    from braid_b200.engine_dropin import text_config
    from braid_b200.projection_set import StackShapes
    c, s = text_config(), StackShapes()
    assert (c["hidden_size"], c["intermediate_size"], c["num_hidden_layers"]) == (s.hidden, s.intermediate, s.n_layers)
    assert c["layer_types"].count("full_attention") == 8 and c["layer_types"][3] == "full_attention"
    assert 2 * c["num_attention_heads"] * c["head_dim"] == s.attn_q
    assert c["num_key_value_heads"] * c["head_dim"] == s.attn_kv
    assert c["linear_num_value_heads"] * c["linear_value_head_dim"] == s.gdn_inner
    assert (2 * c["linear_num_key_heads"] * c["linear_key_head_dim"]
            + c["linear_num_value_heads"] * c["linear_value_head_dim"]) == s.gdn_qkv
    assert text_config(layers=8, vocab=4096)["vocab_size"] == 4096


@pytest.mark.skipif(_ref_install() is None, reason="no reference install under baseline/_ref")
def test_random_checkpoint_runs_through_the_reference_engine_on_cpu():
    """A CPU-sized stack of the same structure: the reference's loader validation accepts the
    tensors and its engine decodes with every group quantized (stock torch arm)."""
    import sys
    ref = _ref_install()
    sys.path.insert(0, str(ref))
    try:
        from braid_b200 import engine_dropin as E
        cfg = E.text_config(layers=4, vocab=1024, hidden_size=64, intermediate_size=128,
                            num_attention_heads=4, num_key_value_heads=2, head_dim=32,
                            linear_num_value_heads=4, linear_num_key_heads=2,
                            linear_value_head_dim=16, linear_key_head_dim=16,
                            rope_parameters={"rope_type": "default", "rope_theta": 1e7,
                                             "partial_rotary_factor": 0.25, "mrope_section": [2, 1, 1],
                                             "mrope_interleaved": True})
        ck = E.random_checkpoint(cfg, "cpu", torch.bfloat16)
        assert ck.config.gdn_layers == (0, 1, 2) and ck.config.attention_layers == (3,)
        eng = E.build_engine(ck, quant="all", use_kernels=False, state_dtype=torch.float32)
        cache = eng.allocate_cache(32, max_slots=3)
        E.seed_cache(eng, cache, 3, 5)
        out = eng.decode_step(torch.tensor([[1], [2], [3]]), cache.select([0, 1, 2]))
        assert out.shape == (3, 1024) and torch.isfinite(out.float()).all()
        assert " 3/3 " in eng.quant_report() or "fp8" in eng.quant_report()
    finally:
        sys.path.remove(str(ref))
        for name in [m for m in sys.modules if m == "braid" or m.startswith("braid.")]:
            del sys.modules[name]


def test_push_entry_points_check_their_arguments():
    """Host-only: the column-parallel entry points refuse missing pointers before any CUDA call."""
    from braid_b200 import _lib
    lib = _lib.load()
    assert lib.bq_wait_flag(None, None, 1, None, None) == _lib.BQ_ERR_BAD_ARG
    assert lib.bq_gemm_w8a8_push(None, None, None, None, 1, 8, 4096, 4096, 0, None, 4096, None,
                                 None, 0, None) == _lib.BQ_ERR_BAD_ARG
    assert lib.bq_peer_open(None, None) == _lib.BQ_ERR_BAD_ARG
    assert lib.bq_peer_alloc(0, None, None) == _lib.BQ_ERR_BAD_ARG


def test_the_read_only_load_path_is_kept_for_load_time_constants():
    """Kernels start ahead of the ones whose outputs they read; a load the compiler takes for one of
    constant memory (`__ldg`) may be moved above the wait.  Only norm weights and weight scales,
    which no kernel of a forward pass writes, may be read that way."""
    csrc = ROOT / "braid_b200" / "csrc"
    seen = 0
    for f in sorted(csrc.iterdir()):
        for i, line in enumerate(f.read_text().splitlines(), 1):
            code = line.split("//")[0]
            assert "ld.global.nc" not in code, f"{f.name}:{i}"
            for arg in re.findall(r"__ldg\((.*)", code):
                seen += 1
                assert re.match(r"reinterpret_cast<const float4\*>\(p\.gamma\)|seg\.sw\)|p\.pair\.sw_up\)", arg), f"{f.name}:{i}: {line}"
    assert seen > 0
