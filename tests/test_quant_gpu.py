"""The sm_100a quantizer against the reference's torch spelling on the same device (bit identity),
against the CPU oracle, and against the committed golden vectors.  Mirrors the reference's own
gates (tests/test_quant.py:65-70, :146-152, :371-477) and widens them."""
from __future__ import annotations

import numpy as np
import pytest
import torch
import torch.nn.functional as F

import oracle
from oracle import torch_spelling as TS
from _util import captured_kernels, codes_np, f32_bits, from_bits16, randn_cpu, to_np_f32, u8

pytestmark = pytest.mark.gpu

DTYPES = [torch.bfloat16, torch.float32, torch.float16]
DT_IDS = ["bf16", "fp32", "fp16"]


def _assert_same(q, s, qr, sr, what=""):
    assert torch.equal(s, sr), f"{what} scale differs: {s.item():.9e} vs {sr.item():.9e}"
    diff = int((u8(q) != u8(qr)).sum())
    assert diff == 0, f"{what}: {diff} of {q.numel()} fp8 bytes differ"


@pytest.mark.parametrize("dt", DTYPES, ids=DT_IDS)
@pytest.mark.parametrize("shape", [(1, 4096), (8, 4096), (37, 12288), (128, 12288)],
                         ids=["m1", "m8", "m37", "m128"])
def test_bit_identical_to_the_torch_spelling(Q, dt, shape):
    """The reference's own gate, same generator and seed (tests/test_quant.py:387-401)."""
    g = torch.Generator(device="cuda").manual_seed(17)
    x = (torch.randn(*shape, generator=g, device="cuda", dtype=torch.float32) * 3.5).to(dt)
    q, s = Q.quantize_act(x)
    qr, sr = TS.quantize_act(x)
    assert q.dtype is Q.FP8 and q.shape == x.shape
    assert s.shape == (1, 1) and s.dtype is torch.float32 and s.is_cuda
    _assert_same(q, s, qr, sr, f"{dt} {shape}")


@pytest.mark.parametrize("shape", [(1, 8), (1, 1), (3, 100), (5, 7), (16, 4096), (64, 4096),
                                   (128, 4096), (333, 12288), (2048, 4096), (8192, 4096)])
@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float32], ids=["bf16", "fp32"])
def test_ragged_small_and_streaming_sizes(Q, shape, dt):
    """Tails that are not a multiple of 8, single-CTA grids, the register-held regime and the
    streaming regime (8192x4096 = BASELINE's prefill activation)."""
    x = randn_cpu(shape, seed=shape[0] * 31 + shape[1], dtype=dt, scale=2.0).cuda()
    q, s = Q.quantize_act(x)
    qr, sr = TS.quantize_act(x)
    _assert_same(q, s, qr, sr, f"{dt} {shape}")


@pytest.mark.parametrize("dt,n", [(torch.bfloat16, 4_850_000 + 4099), (torch.bfloat16, 9_000_001),
                                  (torch.bfloat16, 20_000_003), (torch.bfloat16, 296 * 3 * 16384 + 8),
                                  (torch.bfloat16, 296 * 4 * 16384), (torch.float16, 7_777_777),
                                  (torch.float32, 2_500_001), (torch.float32, 9_000_005),
                                  (torch.bfloat16, 9_699_328 + 11), (torch.bfloat16, 12_000_007), (torch.float16, 9_699_328 + 9),
                                  (torch.float16, 296 * 3 * 16384 + 13), (torch.float16, 20_000_003), (torch.float32, 4_849_664 + 9),
                                  (torch.float32, 6_000_003), (torch.float32, 296 * 3 * 8192 + 12)],
                         ids=["bf16-held-8", "bf16-held-16", "bf16-refetch", "bf16-ring-full+1",
                              "bf16-4-each", "fp16-held-16", "fp32-held-8", "fp32-refetch", "bf16-first", "bf16-16KB-chunks",
                              "fp16-first", "fp16-ring-full+1", "fp16-refetch", "fp32-first", "fp32-16KB-chunks", "fp32-ring-full+1"])
def test_ragged_sizes_through_the_shared_memory_ring(Q, dt, n):
    """Plain quantizer beyond the register-held regime (148 SMs: 9.7 M 16-bit values, 4.85 M of fp32; sizes below it are those of the
    cast alone): a ring of bulk copies per CTA (96 KB; chunks of 16 or 32 KB by input size, of the cast alone 8 KB too).  The first size
    that takes it, sizes where every chunk of a CTA stays in the ring between the passes, where chunks are fetched again,
    where the ring is exactly full (three 32 KB chunks per CTA on 148 SMs), a short last chunk and a tail that is no whole group;
    the cast half alone at the same sizes; and the register-fed streaming kernel on the same
    input (option `quant_ring` off) gives the same bits."""
    held = torch.cuda.get_device_properties(0).multi_processor_count * 512 * 64 * (1 if dt is torch.float32 else 2)
    (kernel,), _ = captured_kernels(lambda x=torch.empty(n, dtype=dt, device="cuda"): Q.quantize_act(x))
    assert ("quant_ring_kernel" in kernel["name"]) == (n >= held + 8), kernel["name"]
    x = randn_cpu((n,), seed=n % 1000, dtype=dt, scale=1.7).cuda()
    q, s = Q.quantize_act(x)
    qr, sr = TS.quantize_act(x)
    _assert_same(q, s, qr, sr, f"{dt} {n}")
    qc = Q.cast_act(x, sr)
    assert torch.equal(u8(qc).reshape(-1), u8(qr).reshape(-1))
    try:
        Q.set_option("quant_ring", 0)
        q0, s0 = Q.quantize_act(x)
        qc0 = Q.cast_act(x, sr)
    finally:
        Q.set_option("quant_ring", 1)
    _assert_same(q0, s0, qr, sr, f"register-fed {dt} {n}")
    assert torch.equal(u8(qc0).reshape(-1), u8(qr).reshape(-1))
    assert Q.device_status() == 0


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16, torch.float32], ids=["bf16", "fp16", "fp32"])
def test_values_held_up_to_64_registers(Q, dt):
    """Every count of groups that a thread holds has its last size, one group more and a tail; beyond the last count the ring
    takes over.  The largest value is the last one, and a NaN anywhere makes the scale NaN."""
    per = torch.cuda.get_device_properties(0).multi_processor_count * 512 * 8
    most = 8 if dt is torch.float32 else 16
    for held in (4, most // 2, most - 1, most):
        for n in (per * held, per * held + 8, per * held - 3):
            x = randn_cpu((n,), seed=held, dtype=dt, scale=1.7).cuda()
            x[-1] = 50.0
            qr, sr = TS.quantize_act(x)
            _assert_same(*Q.quantize_act(x), qr, sr, f"{dt} {held} {n}")
    x[n // 2] = float("nan")
    assert Q.quantize_act(x)[1].isnan().all()
    assert Q.device_status() == 0


@pytest.mark.parametrize("cols", [4096, 12288])
def test_config_4_activations_on_the_streaming_kernel(Q, cols):
    """16 packed sequences (M ~ 8192 rows) of width 4096 (layer input) and
    12288 (MLP intermediate), far beyond what one co-resident grid can hold in registers."""
    g = torch.Generator().manual_seed(4)
    M = int(torch.randint(64, 1025, (16,), generator=g).sum())
    x = randn_cpu((M, cols), seed=cols).cuda()
    q, s = Q.quantize_act(x)
    qr, sr = TS.quantize_act(x)
    _assert_same(q, s, qr, sr, f"{M}x{cols}")
    if cols == 12288:
        gu = randn_cpu((M, 2 * cols), seed=7, scale=2.0).cuda()
        q, s = Q.silu_mul_quant(gu[:, :cols], gu[:, cols:])
        qr, sr = TS.quantize_act(TS.silu_mul(gu[:, :cols], gu[:, cols:]))
        _assert_same(q, s, qr, sr, "silu_mul prologue at prefill size")
    assert Q.device_status() == 0


@pytest.mark.parametrize("dt", DTYPES, ids=DT_IDS)
@pytest.mark.parametrize("shape", [(1, 64), (37, 1536), (128, 12288), (4096, 1536)])
def test_scale_and_cast_halves_equal_the_whole_quantizer(Q, dt, shape):
    """`silu_mul_scale` + `silu_mul_cast` (the column-parallel MLP's exchange) against
    `silu_mul_quant`; and a shard cast under the scale of the whole tensor equals the matching
    columns of the whole tensor's codes."""
    M, I = shape
    gu = randn_cpu((M, 2 * I), seed=M + I, dtype=dt, scale=2.0).cuda()
    g_, u_ = gu[:, :I], gu[:, I:]
    q, s = Q.silu_mul_quant(g_, u_)
    s2 = Q.silu_mul_scale(g_, u_)
    assert torch.equal(s, s2)
    assert torch.equal(u8(Q.silu_mul_cast(g_, u_, s2)), u8(q))
    if I % 32 == 0:
        half = I // 2
        shards = [(g_[:, :half], u_[:, :half]), (g_[:, half:], u_[:, half:])]
        scales = torch.stack([Q.silu_mul_scale(a, b) for a, b in shards])
        smax = scales.max().reshape(1, 1)
        assert torch.equal(smax, s)
        parts = [Q.silu_mul_cast(a, b, smax) for a, b in shards]
        assert torch.equal(u8(torch.cat(parts, dim=1)), u8(q))
    assert Q.device_status() == 0


@pytest.mark.parametrize("shape", [(8, 4096), (37, 12288)])
def test_matches_the_cpu_oracle_with_the_cuda_scale_spelling(Q, shape):
    x = randn_cpu(shape, seed=5, scale=3.5)
    q, s = Q.quantize_act(x.cuda())
    qo, so = oracle.quantize(to_np_f32(x), oracle.SCALE_RCP)
    assert f32_bits(s) == int(np.float32(so).view(np.uint32))
    assert np.array_equal(codes_np(q), qo)


def test_every_bf16_value_through_the_cast(Q):
    """All finite bf16 patterns with |x| <= 448: amax is 448, the scale exactly 1.0."""
    bits = np.arange(65536, dtype=np.uint16)
    x = from_bits16(bits)
    keep = torch.isfinite(x.float()) & (x.float().abs() <= 448.0)
    x = x[keep].contiguous().cuda()
    q, s = Q.quantize_act(x)
    qr, sr = TS.quantize_act(x)
    _assert_same(q, s, qr, sr, "all bf16")
    assert np.array_equal(codes_np(q), oracle.cast(to_np_f32(x), np.float32(s.item())))


def _code_mismatches(q, want):
    """Indices where two e4m3 code tensors differ; two NaN codes (0x7F, 0xFF) count as equal."""
    a, b = u8(q).reshape(-1), u8(want).reshape(-1)
    both_nan = ((a & 0x7F) == 0x7F) & ((b & 0x7F) == 0x7F)
    return ((a != b) & ~both_nan).nonzero().reshape(-1)


def _division_scales():
    """Scales that stress a division done with one rounded reciprocal: random mantissas over the
    exponents activations produce, mantissas of all ones and 1 + 1 ulp (where 1/scale rounds
    worst), powers of two, the reference's floor 1e-12, both ends of the range the kernel takes
    with the reciprocal, values beyond it (the division instruction), infinity."""
    rng = np.random.default_rng(2024)
    mant = rng.integers(0, 1 << 23, size=160, dtype=np.uint32)
    expo = rng.integers(127 - 45, 127 + 20, size=160, dtype=np.uint32)
    bits = list((expo << 23) | mant)
    for e in (127 - 40, 127 - 7, 127, 127 + 5):
        bits += [(e << 23) | 0x7FFFFF, (e << 23) | 1, (e << 23) | 0x7FFFFE, e << 23,
                 (e << 23) | 0x400000, (e << 23) | 0x555555, (e << 23) | 0x2AAAAB]
    vals = list(np.array(bits, dtype=np.uint32).view(np.float32))
    vals += [np.float32(v) for v in (1e-12, 2.0 ** -60, np.nextafter(np.float32(2.0 ** -60), np.float32(0)),
                                      2.0 ** 60, np.nextafter(np.float32(2.0 ** 60), np.float32(np.inf)),
                                      1e-30, 3e35, 3.0, 1.0 / 3.0, np.inf)]
    return vals


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16], ids=["bf16", "fp16"])
def test_cast_under_a_shared_scale_is_the_ieee_division_for_every_16_bit_value(Q, dt):
    """The cast divides by a scale all elements share through one rounded reciprocal and two
    residual corrections; the codes must be those of the IEEE division the reference spells
    (braid/model/quant.py:113) for every one of the 65536 bit patterns (NaN, infinities,
    subnormals and -0 included) under every scale of the list."""
    x = torch.arange(-32768, 32768, dtype=torch.int16).view(dt).cuda()
    for sv in _division_scales():
        scale = torch.full((1, 1), float(sv), dtype=torch.float32, device="cuda")
        q = Q.cast_act(x, scale)
        want = (x.float() / scale).reshape(-1).clamp(-Q.FP8_MAX, Q.FP8_MAX).to(Q.FP8)
        bad = _code_mismatches(q, want)
        assert bad.numel() == 0, (f"scale {float(sv)!r}: {bad.numel()} codes differ, first at bits "
                                  f"{int(x.view(torch.int16)[bad[0]]) & 0xFFFF:#06x}")
    # the oracle's cast agrees with the device's division on a sample of the same grid
    sv = np.float32(0.0123456)
    q = Q.cast_act(x, torch.full((1, 1), float(sv), dtype=torch.float32, device="cuda"))
    fin = torch.isfinite(x.float()).cpu().numpy()
    assert np.array_equal(codes_np(q)[fin], oracle.cast(to_np_f32(x.cpu()), sv)[fin])


def test_cast_of_fp32_values_under_a_shared_scale_is_the_ieee_division(Q):
    """fp32 activations: 2^22 random bit patterns per scale (any exponent, any mantissa)."""
    g = torch.Generator(device="cuda").manual_seed(99)
    bits = torch.randint(-2 ** 31, 2 ** 31 - 1, (1 << 22,), generator=g, device="cuda", dtype=torch.int64)
    x = bits.to(torch.int32).view(torch.float32)
    near = (torch.randn(1 << 22, generator=g, device="cuda") * 3.0)
    for sv in _division_scales()[::5]:
        scale = torch.full((1, 1), float(sv), dtype=torch.float32, device="cuda")
        for t in (x, near * float(sv) if np.isfinite(sv) else near):
            q = Q.cast_act(t, scale)
            want = (t / scale).reshape(-1).clamp(-Q.FP8_MAX, Q.FP8_MAX).to(Q.FP8)
            diff = _code_mismatches(q, want).numel()
            assert diff == 0, f"scale {float(sv)!r}: {diff} codes differ"


def test_golden_vectors_with_the_device_scale(Q, golden):
    """Golden inputs from the reference's CPU run: codes must equal the oracle cast at the scale
    the device computed, and the scale must be the CUDA spelling of the same amax."""
    for key in ("act_bf16_8x4096", "act_bf16_1x4096"):
        x = from_bits16(golden[key + "_x"])
        q, s = Q.quantize_act(x.cuda())
        want_s = oracle.scale_from_amax(oracle.amax(to_np_f32(x)), oracle.SCALE_RCP)
        assert f32_bits(s) == int(want_s.view(np.uint32))
        assert np.array_equal(codes_np(q), oracle.cast(to_np_f32(x), want_s))
        if int(want_s.view(np.uint32)) == int(golden[key + "_scale"].reshape(-1)[0]):
            assert np.array_equal(codes_np(q), golden[key + "_q"])


def test_degenerate_scales(Q):
    for label, fill in (("zeros", 0.0), ("huge", 60000.0), ("tiny", 1e-10)):
        x = torch.full((4, 4096), fill, device="cuda", dtype=torch.bfloat16)
        q, s = Q.quantize_act(x)
        qr, sr = TS.quantize_act(x)
        assert torch.isfinite(s).all(), f"{label}: scale not finite"
        _assert_same(q, s, qr, sr, label)


def test_full_range_is_used(Q):
    x = torch.randn(16, 256, device="cuda", dtype=torch.bfloat16)
    xq, sx = Q.quantize_act(x)
    assert xq.dtype is Q.FP8 and sx.shape == (1, 1)
    assert xq.float().abs().max().item() > Q.FP8_MAX * 0.5


def test_non_contiguous_activation_takes_the_exact_torch_arm(Q):
    base = randn_cpu((64, 4096), seed=5).cuda()
    view = base.t()
    assert not view.is_contiguous()
    q, s = Q.quantize_act(view)
    qc, sc = Q.quantize_act(view.contiguous())
    _assert_same(q, s, qc, sc, "strided")


def test_nan_survives(Q):
    x = randn_cpu((4, 4096), seed=3).cuda()
    x[2, 100] = float("nan")
    q, s = Q.quantize_act(x)
    qr, sr = TS.quantize_act(x)
    assert torch.isnan(s).all() and torch.isnan(sr).all()
    assert torch.equal(u8(q), u8(qr))


def test_warm_fused_switch_selects_the_torch_arm(Q):
    x = randn_cpu((8, 4096), seed=9).cuda()
    fused = Q.quantize_act(x)
    assert Q.fused_state() == "active"
    Q.warm_fused(False)
    try:
        assert Q.fused_state() == "disabled by caller"
        ref = Q.quantize_act(x)
    finally:
        Q.warm_fused(True)
    _assert_same(*fused, *ref, "switch")


def test_back_to_back_calls_leave_the_scratch_clean(Q):
    """The barrier words return to zero: 600 calls (more than the slot pool) stay exact."""
    x = randn_cpu((128, 4096), seed=1).cuda()
    qr, sr = TS.quantize_act(x)
    for _ in range(600):
        q, s = Q.quantize_act(x)
    _assert_same(q, s, qr, sr, "repeat")
    assert Q.device_status() == 0


# ---- prologues ---------------------------------------------------------------------------

@pytest.mark.parametrize("dt", DTYPES, ids=DT_IDS)
@pytest.mark.parametrize("shape", [(1, 12288), (8, 12288), (37, 256), (128, 12288), (512, 12288)])
def test_silu_mul_quant_is_bit_identical(Q, dt, shape):
    gate = randn_cpu(shape, seed=41, dtype=dt, scale=2.0).cuda()
    up = randn_cpu(shape, seed=42, dtype=dt, scale=1.5).cuda()
    q, s = Q.silu_mul_quant(gate, up)
    qr, sr = TS.quantize_act(TS.silu_mul(gate, up))
    _assert_same(q, s, qr, sr, f"silu {dt} {shape}")


def test_silu_mul_quant_reads_column_blocks_in_place(Q):
    """gate and up as the two halves of one [M, 2I] buffer, the layout the grouped GEMM writes."""
    M, I = 16, 1024
    gu = randn_cpu((M, 2 * I), seed=43, scale=2.0).cuda()
    q, s = Q.silu_mul_quant(gu[:, :I], gu[:, I:])
    qr, sr = TS.quantize_act(TS.silu_mul(gu[:, :I].contiguous(), gu[:, I:].contiguous()))
    _assert_same(q, s, qr, sr, "column blocks")


@pytest.mark.parametrize("dt", DTYPES, ids=DT_IDS)
def test_sigmoid_gate_quant_dense_and_per_head_view(Q, dt):
    B, T, H, D = 2, 5, 16, 256
    qg = randn_cpu((B, T, H * 2 * D), seed=44, dtype=dt, scale=2.0).cuda()
    o = randn_cpu((B, T, H * D), seed=45, dtype=dt).cuda()
    _, gate_v = qg.view(B, T, H, 2 * D).chunk(2, dim=-1)        # strided, as in the attention layer
    gate_dense = gate_v.reshape(B, T, H * D)
    qr, sr = TS.quantize_act(TS.sigmoid_gate(o, gate_dense))
    q1, s1 = Q.sigmoid_gate_quant(o, gate_dense)
    _assert_same(q1, s1, qr, sr, "dense gate")
    q2, s2 = Q.sigmoid_gate_quant(o, gate_v)
    _assert_same(q2, s2, qr, sr, "per-head view")
    assert q2.shape == o.shape


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16], ids=["bf16", "fp16"])
def test_silu_and_sigmoid_of_every_16_bit_value(Q, dt):
    """The prologues' silu and sigmoid, seen through the dense forms: the result has to be
    torch's (`F.silu(gate) * up`, braid/model/mlp.py:48; `o * torch.sigmoid(gate)`,
    braid/model/attention.py:215) for every one of the 65536 gate bit patterns, NaN and
    infinities included, under several partners."""
    gate = torch.arange(-32768, 32768, dtype=torch.int16).view(dt).cuda().reshape(64, 1024)
    for partner in (1.0, -3.71875, 0.0009765625, 250.0):
        other = torch.full_like(gate, partner)
        for got, want in ((Q.silu_mul(gate, other), F.silu(gate) * other),
                          (Q.sigmoid_mul(other, gate), other * torch.sigmoid(gate))):
            a, b = got.view(torch.int16), want.view(torch.int16)
            both_nan = torch.isnan(got) & torch.isnan(want)
            bad = ((a != b) & ~both_nan).nonzero()
            assert bad.numel() == 0, (f"{dt} partner {partner}: {bad.shape[0]} values differ, first at gate "
                                      f"bits {int(gate.view(torch.int16)[tuple(bad[0])]) & 0xFFFF:#06x}")
    # random partners: the second rounding sees every first-rounding outcome
    g = torch.Generator(device="cuda").manual_seed(8)
    up = (torch.randn(64, 1024, generator=g, device="cuda") * 2.0).to(dt)
    assert torch.equal(Q.silu_mul(gate, up).view(torch.int16)[~torch.isnan(gate)],
                       (F.silu(gate) * up).view(torch.int16)[~torch.isnan(gate)])


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float32], ids=["bf16", "fp32"])
def test_prologue_quantizers_at_prefill_sizes_take_two_launches(Q, dt):
    """From 2^22 elements on, SiLU*mul and the sigmoid gate run as product + scale (no grid-wide
    wait) followed by the cast pass; same bits as the torch spelling, column blocks and the
    per-head gate view read in place, NaN carried."""
    M, I = 2100, 2048
    gu = randn_cpu((M, 2 * I), seed=51, dtype=dt, scale=2.0).cuda()
    calls = Q.launch_count()
    q, s = Q.silu_mul_quant(gu[:, :I], gu[:, I:])
    assert Q.launch_count() - calls == 2
    qr, sr = TS.quantize_act(TS.silu_mul(gu[:, :I].contiguous(), gu[:, I:].contiguous()))
    _assert_same(q, s, qr, sr, f"silu two-launch {dt}")
    B, T, H, D = 2, 1100, 16, 128
    qg = randn_cpu((B, T, H * 2 * D), seed=52, dtype=dt, scale=2.0).cuda()
    o = randn_cpu((B, T, H * D), seed=53, dtype=dt).cuda()
    _, gate_v = qg.view(B, T, H, 2 * D).chunk(2, dim=-1)
    qr, sr = TS.quantize_act(TS.sigmoid_gate(o, gate_v.reshape(B, T, H * D)))
    calls = Q.launch_count()
    q2, s2 = Q.sigmoid_gate_quant(o, gate_v)
    assert Q.launch_count() - calls == 2
    _assert_same(q2, s2, qr, sr, f"sigmoid two-launch {dt}")
    o[1, 7, 3] = float("nan")
    q3, s3 = Q.sigmoid_gate_quant(o, gate_v)
    assert torch.isnan(s3).all()
    assert Q.device_status() == 0


def test_dense_prologues_in_fp32_and_on_column_blocks(Q):
    x = randn_cpu((33, 2 * 512), seed=12, dtype=torch.float32, scale=3.0).cuda()
    assert torch.equal(Q.silu_mul(x[:, :512], x[:, 512:]), F.silu(x[:, :512]) * x[:, 512:])
    assert torch.equal(Q.sigmoid_mul(x[:, :512].contiguous(), x[:, 512:].contiguous()),
                       x[:, :512] * torch.sigmoid(x[:, 512:]))
    xb = x.to(torch.bfloat16)
    assert torch.equal(Q.silu_mul(xb[:, :512], xb[:, 512:]), F.silu(xb[:, :512]) * xb[:, 512:])


def test_prologues_against_the_golden_vectors(Q, golden):
    """Inputs and outputs of the reference's CPU run.  The device evaluates expf with its own
    library, so agreement with the CPU codes is near-total rather than exact; the bit-exact
    arbiter is the torch-on-device comparison above."""
    gate, up = from_bits16(golden["mlp_gate"]).cuda(), from_bits16(golden["mlp_up"]).cuda()
    q, s = Q.silu_mul_quant(gate, up)
    want = golden["mlp_hq"]
    assert (codes_np(q) != want).mean() < 0.02
    H, D = 4, 64
    qg = from_bits16(golden["sig_qg"]).view(2, 3, H, 2 * D).cuda()
    o = from_bits16(golden["sig_o"]).view(2, 3, H * D).cuda()
    q, s = Q.sigmoid_gate_quant(o, qg[..., D:])
    assert (codes_np(q).reshape(6, H * D) != golden["sig_oq"].reshape(6, H * D)).mean() < 0.02


def test_bad_arguments_raise(Q):
    with pytest.raises(ValueError):
        Q.quantize_act(torch.zeros(4, 8, device="cuda", dtype=torch.int32))
    with pytest.raises(ValueError):
        Q.quantize_act(torch.zeros(0, 8, device="cuda", dtype=torch.bfloat16))
    with pytest.raises(RuntimeError):
        Q.quantize_act(torch.zeros(4, 8, dtype=torch.bfloat16))
    with pytest.raises(ValueError):
        Q.silu_mul_quant(torch.zeros(4, 12, device="cuda", dtype=torch.bfloat16),
                         torch.zeros(4, 12, device="cuda", dtype=torch.bfloat16))
    assert Q.device_status() == 0


@pytest.mark.parametrize("dt", DTYPES, ids=DT_IDS)
@pytest.mark.parametrize("shape", [(16, 16), (272, 1040), (4096, 4096), (12288, 4096)])
def test_quantize_weight_gives_the_bits_of_the_torch_spelling(Q, dt, shape):
    """One launch against the parity arm, infinities and NaN included; strided views keep the torch
    spelling."""
    w = randn_cpu(shape, seed=shape[0], dtype=dt, scale=0.02).cuda()
    cases = [w, w * 1e-3, torch.zeros_like(w), w[:, : shape[1] // 32 * 16] if shape[1] > 16 else w.t()]
    for bad in (float("inf"), float("nan")):
        v = w.clone()
        v[shape[0] // 2, 3] = bad
        cases.append(v)
    for i, v in enumerate(cases):
        got = Q.quantize_weight(v)
        assert (Q._quantize_weight_fused(v) is not None) == v.is_contiguous()
        try:
            Q.warm_fused(False)
            want = Q.quantize_weight(v)
        finally:
            Q.warm_fused(True)
        assert got.shape == want.shape and got.data.shape == want.data.shape
        assert torch.equal(u8(got.scale), u8(want.scale)), f"{dt} {shape} case {i}"
        assert torch.equal(u8(got.data), u8(want.data)), f"{dt} {shape} case {i}"


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16], ids=["bf16", "fp16"])
def test_cast_of_every_16_bit_value_under_many_scales(Q, dt):
    """The cast divides with one residual correction for 16-bit types: all 65,536 values (NaN, infinities
    and subnormals too) under scales of every kind give the codes of the IEEE division."""
    x = torch.arange(65536, dtype=torch.int32, device="cuda").to(torch.int16).view(dt)
    g = torch.Generator().manual_seed(3)
    scales = (torch.rand(400, generator=g) + 1.0) * 2.0 ** torch.randint(-40, 20, (400,), generator=g).float()
    special = torch.tensor([1.0, 3.0, 448.0, 1.0 / 448.0, 1e-12, 2.0 ** -61, 2.0 ** 61, 1.9999999, 1.0000001])
    for s in torch.cat([scales, special]).cuda():
        s = s.reshape(1, 1)
        want = (x.float() / s[0]).clamp(-448.0, 448.0).to(torch.float8_e4m3fn)
        got = Q.cast_act(x, s)
        assert torch.equal(u8(got), u8(want)), f"scale {s.item():.9e}"


def test_weights_load_on_a_side_stream_while_a_graph_replays(Q):
    """Loading shares no state with the forward path: it takes none of its scratch slots, and 300
    weights (more than there are slots) quantized beside a replaying graph leave both sides' bits as
    they are alone.  It works inside a capture too."""
    hidden = 1024
    x = randn_cpu((64, hidden), seed=1).cuda()
    fw = Q.quantize_weight((randn_cpu((hidden, hidden), seed=2) * 0.02).cuda())
    raw = [(randn_cpu((hidden, n), seed=n) * 0.02).cuda() for n in (16, 272, 8192)]
    want = [Q.quantize_weight(w) for w in raw]
    slots = dict(Q._next_slot)

    def step():
        y = x
        for _ in range(8):
            y = Q.linear(y, fw)
        return y, Q.quantize_weight(raw[1]).data

    with torch.cuda.stream(torch.cuda.Stream()):
        step()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = step()
    graph.replay()
    torch.cuda.synchronize()
    alone = [t.clone() for t in out]
    assert torch.equal(u8(alone[1]), u8(want[1].data))
    taken = dict(Q._next_slot)
    assert taken != slots
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    for i in range(100):
        graph.replay()
        with torch.cuda.stream(side):
            got = [Q.quantize_weight(w) for w in raw]
    torch.cuda.synchronize()
    assert Q._next_slot == taken
    for a, b in zip(out, alone):
        assert torch.equal(u8(a), u8(b))
    for a, b in zip(got, want):
        assert torch.equal(u8(a.data), u8(b.data)) and torch.equal(u8(a.scale), u8(b.scale))
    assert Q.device_status() == 0


def test_quantize_weight_can_be_traced_and_transformed(Q):
    """A call that is seen through a tracer or a transform takes the torch spelling: a kernel launched
    by pointer is invisible to them, and a functional tensor's pointer is no memory."""
    import torch.autograd.forward_ad as fwad
    from torch.fx.experimental.proxy_tensor import make_fx
    a, b = ((randn_cpu((32, 48), seed=s) * 0.02).cuda() for s in (1, 2))

    def f(w):
        r = Q.quantize_weight(w)
        return r.data, r.scale

    def same(got, w):
        return all(torch.equal(u8(x), u8(y)) for x, y in zip(got, f(w), strict=True))

    assert Q._quantize_weight_fused(a) is not None
    assert same(make_fx(f)(a)(b), b)
    assert same(torch.jit.trace(f, (a,), check_trace=False)(b), b)
    assert same(torch.func.functionalize(f)(b), b)
    with fwad.dual_level():
        assert Q._quantize_weight_fused(fwad.make_dual(b, a)) is None
    assert torch.func.jvp(lambda w: Q.quantize_weight(w).scale, (b,), (a,))[0].equal(f(b)[1])
    neg = torch._neg_view(b)
    assert same(f(neg), b.neg())
    with pytest.raises(RuntimeError):          # as with the torch spelling
        torch.func.vmap(f)(torch.stack([a, b]))


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16], ids=["bf16", "fp16"])
def test_codes_by_one_product_under_the_scale_of_every_maximum(Q, dt):
    """The passes over large inputs take a code from ONE product where the scale allows it (`ScaleMul`); max |x| / 448 is the
    scale that lies closest to the ties, since 3/4 of the maximum may be one exactly.  Every mantissa a maximum can have, all
    values of the type up to it: the quantizer held in registers and as a ring (beyond what registers hold), the weight
    quantizer, and the cast alone, with few groups per thread (quotients) and with many, under the maximum's own scale and
    under scales one and two units away; against the torch spelling."""
    bits = torch.arange(1 << 16, dtype=torch.int32).to(torch.int16).cuda().view(dt)
    mant = 7 if dt is torch.bfloat16 else 10
    base = (127 << 7) if dt is torch.bfloat16 else (18 << 10)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    ring = sms * 512 * 16 * 8 // bits.numel() + 1         # copies that no longer fit the registers
    many = bits.repeat(2 * 2 * sms * 512 * 8 // bits.numel() + 1)
    for m in range(0, 1 << mant, 1 if mant == 7 else 5):
        top = torch.tensor([base + m], dtype=torch.int16).cuda().view(dt)
        x1 = torch.where((bits.float().abs() <= top.float()), bits, torch.zeros_like(bits))
        x = x1.repeat(32).contiguous()
        q, s = Q.quantize_act(x)
        qr, sr = TS.quantize_act(x)
        _assert_same(q, s, qr, sr, f"{dt} maximum {top.item()}")
        want1 = u8(qr).reshape(-1)[:bits.numel()]
        q, s = Q.quantize_act(x1.repeat(ring))
        assert torch.equal(s, sr) and bool((u8(q).view(ring, -1) == want1).all()), f"{dt} ring, maximum {top.item()}"
        w = Q.quantize_weight(x.view(-1, 1024))
        _assert_same(w.data.reshape(-1), w.scale, qr, sr, f"{dt} weight, maximum {top.item()}")
        for ulps in (-2, -1, 0, 1, 2):
            other = (sr.view(torch.int32) + ulps).view(torch.float32)
            want = (bits.float() / other).clamp(-448.0, 448.0).to(torch.float8_e4m3fn)
            assert torch.equal(u8(Q.cast_act(bits, other)).reshape(-1), u8(want).reshape(-1)), f"{dt} {top.item()} {ulps}"
            got = u8(Q.cast_act(many, other)).view(-1, bits.numel())
            assert bool((got == u8(want).reshape(-1)).all()), f"{dt} {top.item()} {ulps}, many groups per thread"
    assert Q.device_status() == 0


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16, torch.float32], ids=["bf16", "fp16", "fp32"])
@pytest.mark.parametrize("rows,cols,chunk", [(1184, 1024, 256), (1185, 1024, 256), (2368, 1024, 128), (2369, 1024, 128), (4095, 1024, 64),
                                             (4097, 1000, 8), (2600, 1000, 40), (1747, 2400, 24), (40001, 104, 104), (3, 24, 24)])
def test_prologues_held_in_registers_up_to_the_two_launches(Q, dt, rows, cols, chunk):
    """One launch up to 2^22 elements: one to eight groups per thread (either side of four, and of two for fp32), groups left
    over, and row lengths and head widths that are no powers of two (their divisions are multiplications); beyond, the
    two-launch form with the same coordinates."""
    gu = randn_cpu((rows, 2 * cols), seed=rows, dtype=dt, scale=3.0).cuda()
    gate, up = gu[:, :cols], gu[:, cols:]
    n0 = Q.launch_count()
    q, s = Q.silu_mul_quant(gate, up)
    assert Q.launch_count() - n0 == (1 if rows * cols < 1 << 22 else 2)
    _assert_same(q, s, *TS.quantize_act(TS.silu_mul(gate.contiguous(), up.contiguous())), f"silu {rows} x {cols}")
    qg = randn_cpu((rows, cols // chunk, 2 * chunk), seed=rows + 1, dtype=dt, scale=3.0).cuda()
    view, o = qg[..., chunk:], up.contiguous()
    q, s = Q.sigmoid_gate_quant(o, view)
    _assert_same(q, s, *TS.quantize_act(TS.sigmoid_gate(o, view.reshape(rows, cols))), f"sigmoid {rows} x {cols} by {chunk}")
    assert Q.device_status() == 0


@pytest.mark.parametrize("option,value,kernels", [
    ("quant_cluster", 1, (16, 512, 16, 1)), ("quant_pdl", 0, (16, 512, 16, 0)), ("quant_cluster", 0, (32, 256, 0, 1)),
    ("quant_block", 512, (16, 512, 0, 1)), ("quant_block", 256, (32, 256, 0, 1)), ("quant_held", 2, (16, 256, 0, 1))])
def test_launch_options_hold_for_decode_batches(Q, option, value, kernels):
    """A batch that would be one cluster takes the launch that the options ask for: its CTAs, threads, CTAs per cluster, and
    whether the next launch may start early; the same codes."""
    x = randn_cpu((16, 4096), seed=1).cuda()
    qr, sr = TS.quantize_act(x)
    default = {"quant_cluster": 1, "quant_pdl": 1}.get(option, 0)
    try:
        Q.set_option(option, value)
        _assert_same(*Q.quantize_act(x), qr, sr)
        found, programmatic = captured_kernels(lambda: (Q.quantize_act(x), Q.quantize_act(x)))
    finally:
        Q.set_option(option, default)
    assert [(k["ctas"], k["threads"], k["cluster"], programmatic) for k in found] == [kernels] * 2
    assert Q.device_status() == 0


@pytest.mark.parametrize("dt,n", [(torch.bfloat16, 2048), (torch.bfloat16, 64 * 4096 + 3), (torch.bfloat16, 9_000_001), (torch.bfloat16, 9_800_005),
                                  (torch.float16, 20_000_000), (torch.float32, 4_700_000), (torch.float32, 5_000_001)])
def test_a_gathered_buffer_is_quantized_and_counted_as_seen(Q, dt, n):
    """`quantize_act_after` with its arrivals in place: one CTA, values held in registers, and beyond (read twice, by the streaming
    kernel); the codes of `quantize_act`, `seen` advanced once, the scratch clean for the next call."""
    x = randn_cpu((n,), seed=n % 1000, dtype=dt, scale=1.7).cuda()
    qr, sr = TS.quantize_act(x)
    flag, seen = (torch.tensor([v], dtype=torch.int32, device="cuda") for v in (8, 5))
    for count, total in ((3, 8), (2, 10)):
        flag.fill_(total)
        _assert_same(*Q.quantize_act_after(x, flag, seen, count), qr, sr, f"{dt} {n}")
        assert seen.item() == total
    assert Q.device_status() == 0
