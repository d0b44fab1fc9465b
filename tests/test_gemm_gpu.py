"""The tcgen05 W8A8 GEMM against the CPU oracle (exact dequantize-and-multiply), the library GEMM
the reference calls (`torch._scaled_mm`), the golden vectors, and its own structural properties:
determinism, split-K invariance within tolerance, grouped == separate, untouched canaries.

Tolerance (BASELINE): max|y - ref| / max|ref| <= 1e-2 on bf16 outputs against an fp32
dequant-matmul; fp32 outputs are held to 1e-4."""
from __future__ import annotations

import numpy as np
import pytest
import torch
import torch.nn.functional as F

import oracle
from oracle import torch_spelling as TS
from _util import captured_kernels, codes_np, config1_inputs, from_bits16, from_bits32, max_rel, randn_cpu, u8

pytestmark = pytest.mark.gpu

TOL_BF16 = 1e-2
TOL_F32 = 1e-4


def _operands(Q, M, N, K, seed=0):
    x = randn_cpu((M, K), seed=seed).cuda()
    w = randn_cpu((N, K), seed=seed + 1, scale=0.02).cuda()
    fw = Q.quantize_weight(w)
    xq, sx = Q.quantize_act(x)
    return x, w, xq, sx, fw


def _oracle(xq, sx, fw):
    return torch.from_numpy(oracle.gemm(codes_np(xq), codes_np(fw.data), sx.item(), fw.scale.item()))


@pytest.mark.parametrize("M", [1, 7, 8, 16, 37, 128, 200, 256])
@pytest.mark.parametrize("N,K", [(16, 16), (128, 128), (512, 256), (1040, 272), (4096, 4096)])
def test_decode_regime_against_the_oracle(Q, M, N, K):
    if N * K * M > 4096 * 4096 * 37 and M not in (37, 128):
        pytest.skip("oracle time")
    _, _, xq, sx, fw = _operands(Q, M, N, K, seed=M + N)
    y = Q.fp8_matmul(xq, sx, fw)
    assert y.shape == (M, N) and y.dtype is torch.bfloat16
    ref = _oracle(xq, sx, fw)
    assert max_rel(y.cpu(), ref) <= TOL_BF16
    y32 = Q.fp8_matmul(xq, sx, fw, out_dtype=torch.float32)
    assert max_rel(y32.cpu(), ref) <= TOL_F32
    assert Q.last_gemm_launch()["kernel"] == "stream"


@pytest.mark.parametrize("M,N,K", [(257, 256, 256), (512, 4096, 4096), (1000, 272, 4096),
                                   (2048, 1024, 128), (2048, 4096, 4096), (4100, 512, 1040)])
def test_prefill_regime_against_fp32_dequant_matmul(Q, M, N, K):
    _, _, xq, sx, fw = _operands(Q, M, N, K, seed=M)
    y = Q.fp8_matmul(xq, sx, fw)
    assert Q.last_gemm_launch()["kernel"] in ("tile", "pair")
    ref = TS.dequant_matmul(xq, sx, fw.data, fw.scale)
    assert max_rel(y, ref) <= TOL_BF16
    y32 = Q.fp8_matmul(xq, sx, fw, out_dtype=torch.float32)
    assert max_rel(y32, ref) <= TOL_F32
    if M * N * K <= 512 * 4096 * 4096:
        sub = slice(0, M, max(1, M // 16))
        ref_o = torch.from_numpy(oracle.gemm(codes_np(xq[sub]), codes_np(fw.data),
                                             sx.item(), fw.scale.item()))
        assert max_rel(y32[sub].cpu(), ref_o) <= TOL_F32


def ragged_pack_rows(seed: int = 4) -> tuple[list[int], int]:
    """16 sequence lengths ~U[64, 1024] (seeded), packed into one row block."""
    g = torch.Generator().manual_seed(seed)
    lens = torch.randint(64, 1025, (16,), generator=g).tolist()
    return lens, int(sum(lens))


CONFIG4_GROUPS = {          # the projection groups of the 9B-class stack (one launch each)
    "mlp.gate_up": ((12288, 12288), 4096),
    "gdn.qkv_z": ((8192, 4096), 4096),
    "mlp.down": ((4096,), 12288),
    "gdn.out_proj": ((4096,), 4096),
    "attn.qkv": ((8192, 1024, 1024), 4096),
}


@pytest.mark.parametrize("name", list(CONFIG4_GROUPS))
def test_config_4_ragged_prefill_at_full_size(Q, name):
    """Chunked ragged prefill at BASELINE's size: 16 packed sequences (M ~ 8192 rows, not a
    multiple of any tile) against the exact fp32 dequantize-and-multiply on the device over the
    whole output, and against the CPU oracle on a strided subsample of rows and columns that
    visits every tile row and tile column of the launch."""
    Ns, K = CONFIG4_GROUPS[name]
    lens, M = ragged_pack_rows()
    assert len(lens) == 16 and 16 * 64 <= M <= 16 * 1024
    x = randn_cpu((M, K), seed=41).cuda()
    ws = [Q.quantize_weight(randn_cpu((n, K), seed=42 + i, scale=0.02).cuda()) for i, n in enumerate(Ns)]
    xq, sx = Q.quantize_act(x)
    ys = Q.fp8_matmul_grouped(xq, sx, ws)
    assert Q.last_gemm_launch()["kernel"] in ("pair", "tile")
    ys32 = Q.fp8_matmul_grouped(xq, sx, ws, out_dtype=torch.float32)
    rows = torch.arange(0, M, 61, device="cuda")
    for y, y32, w in zip(ys, ys32, ws):
        ref = TS.dequant_matmul(xq, sx, w.data, w.scale)
        assert max_rel(y, ref) <= TOL_BF16
        assert max_rel(y32, ref) <= TOL_F32
        del ref
        cols = torch.arange(0, w.shape[0], 37, device="cuda")
        ref_o = torch.from_numpy(oracle.gemm(codes_np(xq[rows]), codes_np(w.data[cols]),
                                             sx.item(), w.scale.item()))
        assert max_rel(y32[rows][:, cols].cpu(), ref_o) <= TOL_F32
    # a row of the product does not depend on which rows share its launch: the packed call equals
    # the per-sequence calls (the reference pads sequences to rectangles instead of packing them)
    lo = sum(lens[:5])
    part = Q.fp8_matmul_grouped(xq[lo:lo + lens[5]].contiguous(), sx, ws, out_dtype=torch.float32)
    for y32, yp in zip(ys32, part):
        assert max_rel(yp, y32[lo:lo + lens[5]]) <= 1e-6
    assert Q.device_status() == 0


@pytest.mark.parametrize("M", [1, 128])
def test_lm_head_at_full_vocabulary(Q, M):
    """The `head` group's weight (braid/model/engine.py:348-349): 248,320 x 4096, 1,940 row tiles
    of the weight-streaming kernel in one launch.  Whole output against the library GEMM the
    reference calls; a strided subsample of the vocabulary against the CPU oracle."""
    V, K = 248320, 4096
    g = torch.Generator(device="cuda").manual_seed(43)
    w = (torch.randn(V, K, generator=g, device="cuda") * 0.02).to(torch.bfloat16)
    fw = Q.quantize_weight(w)
    del w
    x = randn_cpu((M, K), seed=44).cuda()
    xq, sx = Q.quantize_act(x)
    y = Q.fp8_matmul(xq, sx, fw)
    assert y.shape == (M, V) and Q.last_gemm_launch()["kernel"] == "stream"
    ref = TS.scaled_mm(xq, sx, fw.data, fw.scale)
    assert max_rel(y, ref) <= TOL_BF16
    assert (y != ref).float().mean().item() < 0.05
    y32 = Q.fp8_matmul(xq, sx, fw, out_dtype=torch.float32)
    cols = torch.arange(0, V, 251, device="cuda")
    ref_o = torch.from_numpy(oracle.gemm(codes_np(xq), codes_np(fw.data[cols]), sx.item(),
                                         fw.scale.item()))
    assert max_rel(y32[:, cols].cpu(), ref_o) <= TOL_F32
    assert torch.equal(y, Q.fp8_matmul(xq, sx, fw))            # run-to-run identical
    assert Q.device_status() == 0


@pytest.mark.parametrize("M,N,K,dt", [(4096, 512, 12288, torch.bfloat16), (1000, 1040, 4096, torch.bfloat16),
                                      (300, 144, 512, torch.float32), (2048, 4096, 4096, torch.bfloat16),
                                      (768, 4096, 512, torch.bfloat16)],
                         ids=["down-shard-of-8", "ragged", "tiny-fp32", "wide-weight", "two-rounds-if-narrow"])
def test_prefill_tiles_of_128_columns_give_the_bits_of_256(Q, M, N, K, dt):
    """A lone narrow weight at prefill sizes is tiled 256 x 128 instead of 256 x 256 so that more
    CTA pairs have work; every output element is the same sum in the same order either way."""
    _, _, xq, sx, fw = _operands(Q, M, N, K, seed=M + N)
    try:
        Q.set_option("pair_narrow", 0)
        wide = Q.fp8_matmul(xq, sx, fw, out_dtype=dt)
        assert Q.last_gemm_launch()["mma_n"] == 256
        Q.set_option("pair_narrow", 1)
        narrow = Q.fp8_matmul(xq, sx, fw, out_dtype=dt)
        assert Q.last_gemm_launch()["mma_n"] == 128
    finally:
        Q.set_option("pair_narrow", -1)
    assert torch.equal(wide, narrow)
    auto = Q.fp8_matmul(xq, sx, fw, out_dtype=dt)
    tiles_wide = -(-N // 256) * -(-M // 256)
    assert Q.last_gemm_launch()["mma_n"] == (128 if tiles_wide * 2 <= 74 else 256)
    assert torch.equal(auto, wide)
    assert Q.device_status() == 0


@pytest.mark.parametrize("K", [16, 128, 768, 896, 1024, 1152, 2064])
def test_prefill_ring_of_eight_stages_gives_the_bits_of_six(Q, K):
    """Launches of 128-column tiles alone have eight stages: K blocks fewer than, as many as and more than either
    ring holds, several tiles per pair, with a residual and grouped."""
    M, N = 600, 5136
    _, _, xq, sx, fw = _operands(Q, M, N, K, seed=K)
    res = randn_cpu((M, N), seed=3).cuda()
    got = {}
    try:
        for narrow, stages in ((0, 6), (1, 8)):
            Q.set_option("pair_narrow", narrow)
            got[stages] = [Q.fp8_matmul(xq, sx, fw), Q.fp8_matmul(xq, sx, fw, residual=res),
                           *Q.fp8_matmul_grouped(xq, sx, (fw, fw))]
            assert Q.last_gemm_launch()["stages"] == stages
    finally:
        Q.set_option("pair_narrow", -1)
    assert all(torch.equal(a, b) for a, b in zip(got[6], got[8]))
    assert Q.device_status() == 0


@pytest.mark.parametrize("M,N,K,dt", [(1500, 4096, 1024, torch.bfloat16), (300, 400, 2048, torch.float16),
                                      (257, 192, 1024, torch.float32), (768, 4096, 4096, torch.bfloat16)])
def test_prefill_tiles_of_192_columns_give_the_bits_of_256(Q, M, N, K, dt):
    """Tiles between the two widths: every output element is the same sum in the same order, tails in N
    and M included, alone and grouped."""
    _, _, xq, sx, fw = _operands(Q, M, N, K, seed=M + N)
    try:
        Q.set_option("pair_narrow", 0)
        wide = Q.fp8_matmul(xq, sx, fw, out_dtype=dt)
        Q.set_option("pair_narrow", 192)
        got = Q.fp8_matmul(xq, sx, fw, out_dtype=dt)
        assert Q.last_gemm_launch()["mma_n"] == 192
        pair = Q.fp8_matmul_grouped(xq, sx, (fw, fw), out_dtype=dt)
    finally:
        Q.set_option("pair_narrow", -1)
    assert torch.equal(wide, got) and all(torch.equal(wide, p) for p in pair)
    assert torch.equal(wide, Q.fp8_matmul(xq, sx, fw, out_dtype=dt))
    assert Q.device_status() == 0


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float32], ids=["bf16", "fp32"])
@pytest.mark.parametrize("M,N,K,cols", [(257, 16, 1024, 64), (413, 1024, 4096, 64), (512, 1152, 1024, 64), (2300, 208, 2064, 64),
                                        (513, 784, 1040, 128), (512, 1200, 1024, 128), (300, 1024, 912, 64), (300, 1024, 896, 128)])
def test_prefill_tiles_of_64_columns_give_the_bits_of_256(Q, M, N, K, cols, dt):
    """Tiles of 64 columns while half of the pairs hold them: both sides of that line (37 of 74 pairs) and of eight K blocks,
    tails in M, N and K, more K blocks than stages, residuals of either row stride, grouped."""
    _, _, xq, sx, fw = _operands(Q, M, N, K, seed=M + N)
    res = randn_cpu((M, N), seed=2, dtype=dt).cuda()
    res_rows = randn_cpu((M, N + 4), seed=3, dtype=dt).cuda()[:, :N]

    def run():
        return [Q.fp8_matmul(xq, sx, fw, out_dtype=dt), Q.fp8_matmul(xq, sx, fw, out_dtype=dt, residual=res),
                Q.fp8_matmul(xq, sx, fw, out_dtype=dt, residual=res_rows), *Q.fp8_matmul_grouped(xq, sx, (fw, fw), out_dtype=dt)]

    auto = Q.fp8_matmul(xq, sx, fw, out_dtype=dt)
    assert Q.last_gemm_launch()["mma_n"] == cols
    try:
        Q.set_option("pair_narrow", 0)
        want = run()
        Q.set_option("pair_narrow", 64)
        got = run()
        assert Q.last_gemm_launch()["mma_n"] == 64
    finally:
        Q.set_option("pair_narrow", -1)
    assert torch.equal(auto, want[0]) and all(torch.equal(a, b) for a, b in zip(got, want))
    assert all(torch.equal(a, b) for a, b in zip(run(), want))
    assert Q.device_status() == 0


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float32], ids=["bf16", "fp32"])
@pytest.mark.parametrize("M,Ns", [(4864, (1024,)), (4860, (1040,)), (1500, (8192, 1024, 16))])
def test_prefill_weights_whose_end_is_tiled_apart_give_the_bits_of_256(Q, dt, M, Ns):
    """Sizes whose last round is evened out with the end of the widest weight in 128-column tiles: outputs,
    with and without a residual, equal those of 256-column tiles throughout."""
    K = 1024
    x = randn_cpu((M, K), seed=M, dtype=dt).cuda()
    xq, sx = Q.quantize_act(x)
    ws = [Q.quantize_weight(randn_cpu((n, K), seed=n, scale=0.02).cuda()) for n in Ns]
    res = randn_cpu((M, Ns[0]), seed=1, dtype=dt).cuda()

    def run():
        return [*Q.fp8_matmul_grouped(xq, sx, ws, out_dtype=dt), Q.fp8_matmul(xq, sx, ws[0], out_dtype=dt, residual=res)]

    try:
        Q.set_option("pair_narrow", 0)
        want = run()
    finally:
        Q.set_option("pair_narrow", -1)
    for a, b in zip(run(), want):
        assert torch.equal(a, b)
    assert Q.device_status() == 0


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16, torch.float32], ids=["bf16", "fp16", "fp32"])
@pytest.mark.parametrize("M,V,K", [(1, 248320, 4096), (128, 248320, 4096), (37, 1040, 272),
                                   (4, 4096, 256), (256, 16, 16)])
def test_lm_head_argmax_equals_argmax_of_the_logits(Q, dt, M, V, K):
    """braid/model/engine.py:349 + braid/serve/scheduler.py:346: the greedy token of every row,
    taken in the GEMM's epilogue, equals `linear(h, lm_head).argmax(-1)` exactly -- ties between
    equal logits (bf16 rounding makes them common, and duplicated vocabulary rows force them)
    go to the lowest index; the logits, when asked for, are the plain GEMM's bits."""
    if dt is not torch.bfloat16 and V > 5000:
        pytest.skip("dtype variants on the small shapes")
    g = torch.Generator(device="cuda").manual_seed(V + M)
    w = (torch.randn(V, K, generator=g, device="cuda") * 0.02).to(torch.bfloat16)
    fw = Q.quantize_weight(w)
    del w
    if V >= 1040:      # duplicated rows: exact ties far apart in the vocabulary (different tiles)
        codes = fw.data.view(torch.uint8)
        codes[V - 7] = codes[3]
        codes[V // 2 + 1] = codes[V // 2 - 300]
    x = randn_cpu((M, K), seed=M + K, dtype=dt).cuda()
    if V >= 1040:      # make the duplicated rows the winners of two batch rows
        lut = fw.data[3].to(dt)
        x[0] = lut * 8
        if M > 1:
            x[M - 1] = fw.data[V // 2 - 300].to(dt) * 8
    want_logits = Q.linear(x, fw)
    want = want_logits.argmax(-1)
    n0 = Q.launch_count()
    got = Q.lm_head_argmax(x, fw)
    assert Q.launch_count() - n0 == 3                # quantizer, GEMM with the pick, tiny reduction
    assert got.dtype is torch.int64 and got.shape == (M,)
    assert torch.equal(got, want), (got[:4], want[:4])
    if V >= 1040:
        assert int(got[0]) == 3                       # the lower of the two tied indices
    idx2, logits = Q.lm_head_argmax(x, fw, return_logits=True)
    assert torch.equal(idx2, want) and torch.equal(logits, want_logits)
    # a NaN in a row makes every logit of that row NaN: index 0, as torch picks
    if M >= 4:
        x[2, 5] = float("nan")
        assert torch.equal(Q.lm_head_argmax(x, fw), Q.linear(x, fw).argmax(-1))
    # leading dims and a tensor that carries its quantization
    x3 = x.reshape(M, 1, K)
    assert Q.lm_head_argmax(x3, fw).shape == (M, 1)
    assert Q.device_status() == 0


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16, torch.float32], ids=["bf16", "fp16", "fp32"])
def test_prefill_store_paths_agree_and_stay_in_bounds(Q, dt):
    """The prefill epilogue hands 128-byte row pieces to TMA stores when the output can be
    described to TMA (16-byte aligned base and row pitch) and writes the same staged pieces with
    plain coalesced stores otherwise: same bits either way, ragged M and N clipped, nothing
    outside the output touched."""
    M, N, K = 1000, 4096 + 16, 1040
    _, _, xq, sx, fw = _operands(Q, M, N, K, seed=77)
    want = Q.fp8_matmul(xq, sx, fw, out_dtype=dt)                 # contiguous: the TMA path
    assert Q.last_gemm_launch()["kernel"] == "pair"
    ref = TS.dequant_matmul(xq, sx, fw.data, fw.scale)
    assert max_rel(want, ref) <= (TOL_F32 if dt is torch.float32 else TOL_BF16)
    # 16-bit outputs: a pitch of N + 4 elements is 8-byte but not 16-byte aligned (plain stores);
    # fp32 outputs must be 16-byte aligned anyway, so every legal one takes the TMA path
    for off, pitch in ((0, N + 4), (4, N + 4), (8, N + 24)):
        big = torch.full((M + 2, pitch + 16), 7.0, device="cuda", dtype=dt)
        out = big[1:M + 1, off:off + N]
        Q.fp8_matmul_grouped(xq, sx, (fw,), out_dtype=dt, out=(out,))
        assert torch.equal(out, want), (off, pitch)
        mask = torch.ones_like(big, dtype=torch.bool)
        mask[1:M + 1, off:off + N] = False
        assert (big[mask] == 7.0).all(), (off, pitch)
    assert Q.device_status() == 0


@pytest.mark.parametrize("M,N,K", [(8, 4096, 4096), (128, 4096, 4096), (128, 1024, 4096),
                                   (64, 4096, 12288), (2048, 4096, 4096)])
def test_agrees_with_the_library_gemm_the_reference_calls(Q, M, N, K):
    _, _, xq, sx, fw = _operands(Q, M, N, K, seed=3)
    y = Q.fp8_matmul(xq, sx, fw)
    ref = TS.scaled_mm(xq, sx, fw.data, fw.scale)
    assert max_rel(y, ref) <= TOL_BF16
    # both round the same fp32 sums to bf16: almost every element is bit-equal
    assert (y != ref).float().mean().item() < 0.05


def test_config_1_against_the_reference_cpu_output(Q, golden):
    import hashlib
    x, w = config1_inputs(0)
    sha = lambda t: np.frombuffer(hashlib.sha256(t.view(torch.uint8).numpy().tobytes()).digest(), np.uint8)
    if not (np.array_equal(sha(x), golden["c1_xsha"]) and np.array_equal(sha(w), golden["c1_wsha"])):
        pytest.skip("this torch build draws different random numbers")
    fw = Q.quantize_weight(w.cuda())
    xq, sx = Q.quantize_act(x.cuda())
    y = Q.fp8_matmul(xq, sx, fw)
    ref = from_bits16(golden["c1_y"]).float()
    assert max_rel(y.cpu().float(), ref) <= TOL_BF16
    # end to end through the public call, as the reference's test does
    y2 = Q.fp8_linear(x.cuda(), fw)
    assert torch.equal(y, y2)


def test_small_golden_gemm(Q, golden):
    xq = torch.from_numpy(golden["gemm_xq"]).cuda().view(Q.FP8)
    sx = from_bits32(golden["gemm_sx"]).cuda().reshape(1, 1)
    for wq_key, sw_key, y_key in (("weight_q", "weight_scale", "gemm_ya"),
                                  ("gemm_wbq", "gemm_wb_scale", "gemm_yb")):
        wq = torch.from_numpy(golden[wq_key]).cuda().view(Q.FP8)
        fw = Q.FP8Weight(data=wq, scale=from_bits32(golden[sw_key]).cuda().reshape(1, 1),
                         shape=tuple(wq.shape))
        y = Q.fp8_matmul(xq, sx, fw)
        assert max_rel(y.cpu().float(), from_bits16(golden[y_key]).float()) <= TOL_BF16


def test_run_to_run_determinism_and_split_k(Q):
    _, _, xq, sx, fw = _operands(Q, 128, 4096, 4096, seed=8)
    ref = TS.dequant_matmul(xq, sx, fw.data, fw.scale)
    try:
        for split in (1, 2, 4):
            Q.set_option("decode_split_k", split)
            a = Q.fp8_matmul(xq, sx, fw)
            assert Q.last_gemm_launch()["split"] == split
            for _ in range(3):
                assert torch.equal(a, Q.fp8_matmul(xq, sx, fw)), f"split {split} is not deterministic"
            assert max_rel(a, ref) <= TOL_BF16
    finally:
        Q.set_option("decode_split_k", 0)


def test_pipeline_depth_does_not_change_results(Q):
    _, _, xq, sx, fw = _operands(Q, 16, 512, 4096, seed=9)
    try:
        Q.set_option("decode_split_k", 1)
        base = Q.fp8_matmul(xq, sx, fw, out_dtype=torch.float32)
        for stages in (1, 2, 3, 5):
            Q.set_option("decode_stages", stages)
            assert torch.equal(base, Q.fp8_matmul(xq, sx, fw, out_dtype=torch.float32))
            assert Q.last_gemm_launch()["stages"] <= stages     # never deeper than the work
    finally:
        Q.set_option("decode_split_k", 0)
        Q.set_option("decode_stages", 0)


@pytest.mark.parametrize("M", [4, 128, 1024])
def test_project_matches_linear_per_weight(Q, M):
    """tests/test_quant.py:211-218 — grouped launch equals the separate calls bit for bit."""
    x = randn_cpu((M, 256), seed=12).cuda()
    qa = Q.quantize_weight(randn_cpu((512, 256), seed=13, scale=0.02).cuda())
    qb = Q.quantize_weight(randn_cpu((128, 256), seed=14, scale=0.03).cuda())
    qc = Q.quantize_weight(randn_cpu((272, 256), seed=15, scale=0.01).cuda())
    got = Q.project(x, qa, qb, qc)
    for g, w in zip(got, (qa, qb, qc)):
        assert torch.equal(g, Q.fp8_linear(x, w))


def test_project_leaves_bf16_weights_on_the_bf16_path(Q):
    """tests/test_quant.py:221-242: a weight left in bf16 is multiplied unquantized.  Through
    `F.linear` (the reference's arm, selectable) the result is that call's bits; as a 16-bit
    segment of the one launch (default) it is the same product up to summation order."""
    x = randn_cpu((4, 256), seed=16).cuda()
    a = randn_cpu((512, 256), seed=17, scale=0.02).cuda()
    b = randn_cpu((32, 256), seed=18, scale=0.02).cuda()
    Q.set_dense_segments(False)
    try:
        got_a, got_b = Q.project(x, Q.quantize_weight(a), b)
        assert torch.equal(got_b, F.linear(x, b))
    finally:
        Q.set_dense_segments(True)
    n0 = Q.launch_count()
    seg_a, seg_b = Q.project(x, Q.quantize_weight(a), b)
    assert Q.launch_count() - n0 == 2                       # one quantizer, one GEMM launch
    assert torch.equal(seg_a, got_a)                        # the FP8 member does not change
    assert seg_b.dtype is torch.bfloat16 and seg_b.shape == (4, 32)
    assert max_rel(seg_b, F.linear(x.float(), b.float())) <= 2 ** -8
    ga, gb = Q.project(x, a, b)                             # no FP8 member: untouched torch path
    assert torch.equal(ga, F.linear(x, a)) and torch.equal(gb, F.linear(x, b))


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16], ids=["bf16", "fp16"])
@pytest.mark.parametrize("M", [1, 16, 37, 128, 256])
def test_gdn_input_projection_as_one_launch(Q, dt, M):
    """braid/model/gdn.py:254-255: `project(x, qkv, z, a, b)` with qkv / z in FP8 and the gates
    a / b unquantized (32 x 4096 each, braid/model/gdn.py:73-81), at the 9B widths.  FP8 members
    bit-equal to the grouped FP8 launch; a and b within bf16 rounding of the exact product and
    almost everywhere bit-equal to `F.linear`; run-to-run identical; graph-capturable."""
    H = 4096
    x = randn_cpu((M, H), seed=M, dtype=dt).cuda()
    qkv = Q.quantize_weight(randn_cpu((8192, H), seed=1, scale=0.02).cuda())
    z = Q.quantize_weight(randn_cpu((4096, H), seed=2, scale=0.02).cuda())
    a = randn_cpu((32, H), seed=3, dtype=dt, scale=0.02).cuda()
    b = randn_cpu((32, H), seed=4, dtype=dt, scale=0.05).cuda()
    ys = Q.project(x, qkv, z, a, b)
    assert Q.last_gemm_launch()["kernel"] == "stream"
    xq, sx = Q.quantize_act(x)
    for got, want in zip(ys[:2], Q.fp8_matmul_grouped(xq, sx, (qkv, z), out_dtype=dt)):
        assert torch.equal(got, want)
    for got, w in zip(ys[2:], (a, b)):
        exact = F.linear(x.double(), w.double())
        assert got.dtype is dt and got.shape == (M, 32)
        assert max_rel(got, exact) <= (2 ** -8 if dt is torch.bfloat16 else 2 ** -10)
        assert (got != F.linear(x, w)).float().mean().item() < 0.1
    again = Q.project(x, qkv, z, a, b)
    assert all(torch.equal(p, q) for p, q in zip(ys, again))
    # a pre-quantized activation that kept its dense form takes the same launch
    pre = Q.QuantizedActivation(xq, sx, x.shape, dt, dense=x)
    assert all(torch.equal(p, q) for p, q in zip(ys, Q.project(pre, qkv, z, a, b)))
    assert Q.device_status() == 0


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16], ids=["bf16", "fp16"])
@pytest.mark.parametrize("M,K,widths", [(257, 4096, (32, 32)), (300, 1040, (16, 256)), (513, 512, (240, 80)),
                                        (1500, 2048, (48,))])
def test_prefill_mixed_projection_as_one_launch(Q, dt, M, K, widths):
    """M > 256: 16-bit weights of up to 256 rows are tiles of the one launch.  FP8 members bit-equal to
    their own launch, 16-bit ones within half a unit of the type of the exact product (fp32 sums over K
    add far less); wider ones and those that record gradients go through `F.linear`."""
    x = randn_cpu((M, K), seed=M, dtype=dt).cuda()
    w = Q.quantize_weight(randn_cpu((2 * K, K), seed=1, scale=0.02).cuda())
    dense = [randn_cpu((n, K), seed=2 + n, dtype=dt, scale=0.02).cuda() for n in widths]
    n0 = Q.launch_count()
    ys = Q.project(x, w, *dense)
    assert Q.launch_count() - n0 == 2 and Q.last_gemm_launch()["kernel"] == "pair"
    xq, sx = Q.quantize_act(x)
    assert torch.equal(ys[0], Q.fp8_matmul(xq, sx, w, out_dtype=dt))
    for y, d in zip(ys[1:], dense):
        assert y.dtype is dt and y.shape == (M, d.shape[0])
        assert max_rel(y, F.linear(x.double(), d.double())) <= (2 ** -8 if dt is torch.bfloat16 else 2 ** -10)
    assert all(torch.equal(p, q) for p, q in zip(ys, Q.project(x, w, *dense)))
    wide = randn_cpu((272, K), seed=5, dtype=dt, scale=0.02).cuda()
    assert torch.equal(Q.project(x, w, wide)[1], F.linear(x, wide))
    d = dense[0].clone().requires_grad_()
    got = Q.project(x, w, d)[1]
    assert got.requires_grad and torch.equal(got, F.linear(x, d))
    assert Q.device_status() == 0


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16], ids=["bf16", "fp16"])
@pytest.mark.parametrize("M", [1, 16, 48, 49, 100, 128, 161, 256, 257, 300])
def test_sixteen_bit_weights_of_few_odd_rows_ride_along(Q, dt, M):
    """Gates of 8, 20 or 40 rows (hidden 1024, 2560, 5120), and of 4, 36 or 244: a 16-bit weight's rows are a multiple of 4.
    One launch on each of the three kernels, FP8 members bit-equal to their own, 16-bit ones within half a unit of the type of
    the exact product; nothing beyond a row's end is written; what records gradients or has another count of rows
    goes through `F.linear`, as before."""
    K = 1040
    x = randn_cpu((M, K), seed=M, dtype=dt).cuda()
    w = Q.quantize_weight(randn_cpu((2 * K, K), seed=1, scale=0.02).cuda())
    xq, sx = Q.quantize_act(x)
    pre = Q.QuantizedActivation(xq, sx, x.shape, dt, dense=x)
    for widths in ((8, 20), (40, 4), (36, 244, 48)):
        dense = [randn_cpu((n, K), seed=2 + n, dtype=dt, scale=0.02).cuda() for n in widths]
        n0 = Q.launch_count()
        ys = Q.project(pre, w, *dense)
        assert Q.launch_count() - n0 == 1
        assert torch.equal(ys[0], Q.fp8_matmul(xq, sx, w, out_dtype=dt))
        for y, d in zip(ys[1:], dense):
            assert y.dtype is dt and y.shape == (M, d.shape[0]) and y.is_contiguous()
            assert max_rel(y, F.linear(x.double(), d.double())) <= (2 ** -8 if dt is torch.bfloat16 else 2 ** -10)
        assert all(torch.equal(p, q) for p, q in zip(ys, Q.project(x, w, *dense)))
    odd = randn_cpu((18, K), seed=5, dtype=dt, scale=0.02).cuda()
    assert torch.equal(Q.project(pre, w, odd)[1], F.linear(x, odd))
    d = randn_cpu((20, K), seed=6, dtype=dt, scale=0.02).cuda().requires_grad_()
    got = Q.project(pre, w, d)[1]
    assert got.requires_grad and torch.equal(got, F.linear(x, d))
    assert Q.device_status() == 0


def test_leading_dims_and_dispatch(Q):
    x = randn_cpu((2, 3, 256), seed=19).cuda()
    w = randn_cpu((512, 256), seed=20, scale=0.02).cuda()
    fw = Q.quantize_weight(w)
    out = Q.fp8_linear(x, fw)
    assert out.shape == (2, 3, 512) and out.dtype is torch.bfloat16
    assert torch.equal(Q.linear(x, w), F.linear(x, w))
    ref = F.linear(x, w)
    rel = ((out.float() - ref.float()).norm() / ref.float().norm()).item()
    assert rel < 8e-2
    assert F.cosine_similarity(out.float().flatten(), ref.float().flatten(), dim=0) > 0.99
    (p,) = Q.project(x, fw)
    assert p.shape == (2, 3, 512)


def test_outputs_stay_inside_their_buffers(Q):
    """Canary rows/columns around a strided output must survive (M and N off the tile grid)."""
    for M, N, K in ((37, 272, 256), (300, 272, 256)):
        _, _, xq, sx, fw = _operands(Q, M, N, K, seed=21)
        big = torch.full((M + 2, N + 32), 7.0, device="cuda", dtype=torch.bfloat16)
        out = big[1:M + 1, 16:16 + N]
        Q.fp8_matmul_grouped(xq, sx, (fw,), out=(out,))
        assert torch.equal(out, Q.fp8_matmul(xq, sx, fw))
        mask = torch.ones_like(big, dtype=torch.bool)
        mask[1:M + 1, 16:16 + N] = False
        assert (big[mask] == 7.0).all()


def test_scaling_the_activation_scale_scales_the_output(Q):
    """Linearity at full decode size: doubling sx doubles every output exactly (power of two)."""
    _, _, xq, sx, fw = _operands(Q, 128, 12288, 4096, seed=22)
    y1 = Q.fp8_matmul(xq, sx, fw, out_dtype=torch.float32)
    y2 = Q.fp8_matmul(xq, sx * 2, fw, out_dtype=torch.float32)
    assert torch.equal(y2, y1 * 2)


def test_fused_mlp_equals_the_unfused_sequence(Q):
    """braid/model/mlp.py:44-49 spelled with separate kernels vs `mlp_forward` (4 launches)."""
    M, H, I = 128, 4096, 12288
    x = randn_cpu((M, H), seed=23).cuda()
    wg = Q.quantize_weight(randn_cpu((I, H), seed=24, scale=0.02).cuda())
    wu = Q.quantize_weight(randn_cpu((I, H), seed=25, scale=0.02).cuda())
    wd = Q.quantize_weight(randn_cpu((H, I), seed=26, scale=0.02).cuda())
    xq, sx = Q.quantize_act(x)
    gate = Q.fp8_matmul(xq, sx, wg)
    up = Q.fp8_matmul(xq, sx, wu)
    h = F.silu(gate) * up
    want = Q.linear(h, wd)
    got = Q.mlp_forward(x, wg, wu, wd)
    assert torch.equal(got, want)
    # and it tracks the bf16 MLP the way the reference demands (tests/test_quant.py:157-178)
    wgf, wuf, wdf = (w.data.float() * w.scale for w in (wg, wu, wd))
    ref = F.linear(F.silu(F.linear(x.float(), wgf)) * F.linear(x.float(), wuf), wdf)
    assert F.cosine_similarity(got.float().flatten(), ref.flatten(), dim=0) > 0.99


def test_gated_output_projection(Q):
    B, T, H, D = 4, 1, 16, 256
    qg = randn_cpu((B, T, H * 2 * D), seed=27, scale=2.0).cuda()
    o = randn_cpu((B, T, H * D), seed=28).cuda()
    wo = Q.quantize_weight(randn_cpu((4096, H * D), seed=29, scale=0.02).cuda())
    _, gate = qg.view(B, T, H, 2 * D).chunk(2, dim=-1)
    want = Q.linear(o * torch.sigmoid(gate.reshape(B, T, H * D)), wo)
    assert torch.equal(Q.gated_output_projection(o, gate, wo), want)


def test_eager_equals_graph_replay(Q):
    """tests/test_graph_quant.py:48-87 in miniature: capture quantize + grouped GEMM + fused MLP,
    replay with new contents in the static input, compare with eager bit for bit."""
    M, H, I = 16, 1024, 2048
    wq_ = Q.quantize_weight(randn_cpu((2048, H), seed=30, scale=0.02).cuda())
    wk_ = Q.quantize_weight(randn_cpu((256, H), seed=31, scale=0.02).cuda())
    wg = Q.quantize_weight(randn_cpu((I, H), seed=32, scale=0.02).cuda())
    wu = Q.quantize_weight(randn_cpu((I, H), seed=33, scale=0.02).cuda())
    wd = Q.quantize_weight(randn_cpu((H, I), seed=34, scale=0.02).cuda())

    def step(x):
        q, k = Q.project(x, wq_, wk_)
        return q[:, :H] + Q.mlp_forward(x + k.sum(dim=1, keepdim=True) * 0, wg, wu, wd)

    static_x = randn_cpu((M, H), seed=35).cuda()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        for _ in range(3):
            step(static_x)
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        static_y = step(static_x)
    for seed in (36, 37):
        new = randn_cpu((M, H), seed=seed, scale=float(seed - 34)).cuda()
        eager = step(new).clone()
        static_x.copy_(new)
        graph.replay()
        assert torch.equal(static_y, eager)
    assert Q.device_status() == 0


def test_shape_guards(Q):
    with pytest.raises(ValueError, match="multiples of 16"):
        Q.quantize_weight(torch.randn(30, 256, device="cuda", dtype=torch.bfloat16))
    w = torch.randn(512, 250, device="cuda", dtype=torch.bfloat16)
    assert Q.maybe_quantize(w, True) is w
    _, _, xq, sx, fw = _operands(Q, 4, 64, 128, seed=40)
    bad = Q.FP8Weight(data=fw.data[:, :64].contiguous(), scale=fw.scale, shape=(64, 64))
    with pytest.raises(ValueError):
        Q.fp8_matmul(xq, sx, bad)
    assert Q.device_status() == 0


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16, torch.float32], ids=["bf16", "fp16", "fp32"])
@pytest.mark.parametrize("K,N", [(4096, 4096), (1040, 1024), (16, 16), (272, 144), (512, 40000), (12288, 1024)])
def test_linear_of_few_rows_as_one_launch(Q, dt, K, N):
    """Up to 16 rows and 64 KB every CTA quantizes the activation for itself: the bits of quantizer and GEMM
    apart, K tails, 1, 2 and 4 K slices, several clusters, a residual, both sides of both limits, NaN."""
    fw = Q.quantize_weight(randn_cpu((N, K), seed=1, scale=0.02).cuda())
    for M in (1, 2, 7, 8, 9, 16, 17):
        x = randn_cpu((M, K), seed=M, dtype=dt).cuda()
        x[0, 3] = 50.0
        res = randn_cpu((M, N), seed=2, dtype=dt).cuda()
        small = M <= 16 and M * K * x.element_size() <= 65536
        for r in (None, res):
            n0 = Q.launch_count()
            got = Q.linear(x, fw, residual=r)
            assert Q._NATIVE is None or Q.launch_count() - n0 == (1 if small else 2)
            xq, sx = Q.quantize_act(x)
            assert torch.equal(got, Q.fp8_matmul(xq, sx, fw, out_dtype=dt, residual=r)), (M, r is not None)
        assert torch.equal(Q.linear(x.view(M, 1, K), fw), Q.linear(x, fw).view(M, 1, N))
        x[M - 1, K - 1] = float("nan")
        assert torch.isnan(Q.linear(x, fw)).all()
    assert Q.device_status() == 0


# -- residual add in the epilogue ---------------------------------------------------------------
@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16, torch.float32], ids=["bf16", "fp16", "fp32"])
@pytest.mark.parametrize("M", [1, 8, 37, 128, 256, 512])
@pytest.mark.parametrize("N,K", [(4096, 4096), (4096, 12288), (1024, 4096), (272, 256), (16, 16)])
def test_residual_epilogue_equals_gemm_then_add(Q, dt, M, N, K):
    """`residual + fp8_matmul(...)` as torch evaluates it (GEMM output rounded to the output type,
    then the add rounds again) against the add done in the GEMM epilogue: bit-equal for every K
    split (1, 2, 4), ragged M, and the prefill sizes that fall back to a separate add."""
    if dt is not torch.bfloat16 and (N, K) not in ((4096, 4096), (272, 256)):
        pytest.skip("dtype variants on two shapes")
    _, _, xq, sx, fw = _operands(Q, M, N, K, seed=M + N)
    res = randn_cpu((M, N), seed=7, dtype=dt, scale=0.5).cuda()
    want = res + Q.fp8_matmul(xq, sx, fw, out_dtype=dt)
    got = Q.fp8_matmul(xq, sx, fw, out_dtype=dt, residual=res)
    assert got.dtype is dt and got.shape == (M, N)
    assert torch.equal(got, want), f"{int((got != want).sum())} of {got.numel()} differ"


def test_linear_of_few_rows_over_several_weights(Q):
    """The entry point takes several weights, of one and of four K slices: each output has the bits of its own
    launch."""
    import ctypes
    from braid_b200 import _lib
    M, K, Ns = 5, 1024, (12288, 272, 16)
    ws = [Q.quantize_weight(randn_cpu((n, K), seed=n, scale=0.02).cuda()) for n in Ns]
    x = randn_cpu((M, K), seed=1).cuda()
    ys = [torch.empty(M, n, device="cuda", dtype=x.dtype) for n in Ns]
    ptrs = lambda ts: (ctypes.c_void_p * 3)(*[t.data_ptr() for t in ts])  # noqa: E731
    n = (ctypes.c_int64 * 3)(*Ns)
    _lib.check(_lib.load().bq_linear_w8a8(x.data_ptr(), 1, M, K, 3, ptrs([w.data for w in ws]), ptrs([w.scale for w in ws]),
                                          None, 0, ptrs(ys), n, n, Q._take_slot(x.device), 16, Q._stream_ptr(x.device)),
               "linear")
    xq, sx = Q.quantize_act(x)
    assert all(torch.equal(y, Q.fp8_matmul(xq, sx, w)) for y, w in zip(ys, ws))
    assert Q.device_status() == 0


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16, torch.float32], ids=["bf16", "fp16", "fp32"])
@pytest.mark.parametrize("M,K,N,split", [(8, 2048, 4096, 0), (4, 4112, 4096, 0), (9, 2064, 8192, 0), (16, 2048, 5008, 2),
                                         (16, 4096, 8192, 0), (15, 6160, 1024, 0), (13, 4096, 2048, 8)])
def test_linear_whose_slices_look_at_their_own_columns(Q, dt, M, K, N, split):
    """Above 32 KB (16 bits: 40 KB) and over sliced weights a CTA looks for the maximum of its own K slice and the slices exchange
    theirs: the bits of quantizer and GEMM apart, on both sides of that line, K tails, 2, 4 and 8 slices, slices that fit the
    registers and that do not (from 40 KB), the largest value and a NaN in any slice, a residual, a replay."""
    fw = Q.quantize_weight(randn_cpu((N, K), seed=1, scale=0.02).cuda())
    res = randn_cpu((M, N), seed=2, dtype=dt).cuda()
    try:
        Q.set_option("decode_quant_inside", 262144)
        Q.set_option("decode_split_k", split)
        for at in (0, K // 2 - 1, K - 1):
            x = randn_cpu((M, K), seed=at, dtype=dt).cuda()
            x[M - 1, at] = -40.0
            xq, sx = Q.quantize_act(x)
            n0 = Q.launch_count()
            got = Q.linear(x, fw, residual=res)
            assert Q._NATIVE is None or Q.launch_count() - n0 == (1 if x.nbytes <= 262144 else 2)
            assert torch.equal(got, Q.fp8_matmul(xq, sx, fw, out_dtype=dt, residual=res)), at
            x[0, K - 1 - at] = float("nan")
            assert torch.isnan(Q.linear(x, fw)).all(), at
        graph, ins = torch.cuda.CUDAGraph(), randn_cpu((M, K), seed=5, dtype=dt).cuda()
        with torch.cuda.graph(graph):
            out = Q.linear(ins, fw)
        for seed in (6, 7):
            ins.copy_(randn_cpu((M, K), seed=seed, dtype=dt, scale=float(seed)))
            graph.replay()
            assert torch.equal(out, Q.fp8_matmul(*Q.quantize_act(ins), fw, out_dtype=dt))
    finally:
        Q.set_option("decode_quant_inside", -1)
        Q.set_option("decode_split_k", 0)
    assert Q.device_status() == 0


@pytest.mark.parametrize("dt,M,K,N,own", [
    (torch.bfloat16, 5, 4096, 8192, False), (torch.float16, 2, 9728, 5760, False), (torch.bfloat16, 4, 5136, 1024, True),
    (torch.bfloat16, 4, 4096, 9728, False), (torch.float16, 4, 4112, 9728, True), (torch.float32, 2, 4096, 4096, False),
    (torch.float32, 2, 4112, 8192, True), (torch.bfloat16, 6, 4096, 14336, False)])
def test_own_slices_only_where_they_pay(Q, dt, M, K, N, own):
    """Both sides of the lines at 32 KB (fp32, and 16 bits where two CTAs share an SM) and at 40 KB: which kernel is launched, and
    the same bits.  A weight that is not sliced has no slices to look at."""
    fw = Q.quantize_weight(randn_cpu((N, K), seed=1, scale=0.02).cuda())
    x = randn_cpu((M, K), seed=M, dtype=dt).cuda()
    try:
        Q.set_option("decode_quant_inside", 262144)
        assert torch.equal(Q.linear(x, fw), Q.fp8_matmul(*Q.quantize_act(x), fw, out_dtype=dt))
        torch.cuda.synchronize()
        (kernel,), _ = captured_kernels(lambda: Q.linear(x, fw))
    finally:
        Q.set_option("decode_quant_inside", -1)
    # the kernel's last template argument: 1 looks at all of x, 3 at its own slice
    assert ("Li3EEEv" if own else "Li1EEEv") in kernel["name"], kernel["name"]
    assert Q.device_status() == 0


def test_linear_whose_weights_have_unlike_slices(Q):
    """Weights of 4, 2 and 4 K slices in one launch, and one that is not sliced beside them (no exchange then)."""
    import ctypes
    from braid_b200 import _lib
    M, K = 8, 2560
    x = randn_cpu((M, K), seed=1).cuda()
    xq, sx = Q.quantize_act(x)
    for Ns in ((4096, 8192, 272), (4096, 12288)):
        ws = [Q.quantize_weight(randn_cpu((n, K), seed=n, scale=0.02).cuda()) for n in Ns]
        ys = [torch.empty(M, n, device="cuda", dtype=x.dtype) for n in Ns]
        ptrs = lambda ts: (ctypes.c_void_p * len(ts))(*[t.data_ptr() for t in ts])  # noqa: E731
        n = (ctypes.c_int64 * len(Ns))(*Ns)
        try:
            Q.set_option("decode_quant_inside", 262144)
            _lib.check(_lib.load().bq_linear_w8a8(x.data_ptr(), 1, M, K, len(Ns), ptrs([w.data for w in ws]),
                                                  ptrs([w.scale for w in ws]), None, 0, ptrs(ys), n, n,
                                                  Q._take_slot(x.device), 16, Q._stream_ptr(x.device)), "linear")
        finally:
            Q.set_option("decode_quant_inside", -1)
        assert all(torch.equal(y, Q.fp8_matmul(xq, sx, w)) for y, w in zip(ys, ws))
    assert Q.device_status() == 0


@pytest.mark.parametrize("M,K,N,eager,captured", [(6, 4096, 4096, 1, 1), (8, 4096, 4096, 1, 2), (8, 4096, 2048, 1, 1),
                                                  (5, 4096, 8192, 1, 1), (6, 4096, 8192, 1, 2), (6, 2048, 12288, 1, 1),
                                                  (8, 2048, 12288, 1, 2), (8, 4096, 6144, 2, 2), (16, 2048, 12288, 2, 2),
                                                  (1, 20480, 8192, 2, 2)])
def test_linear_of_few_rows_in_one_launch_only_where_that_is_faster(Q, M, K, N, eager, captured):
    """Both sides of each line of the rule, by 1, 2 and 4 K slices, eager and captured: the launches, and the
    same bits either way."""
    x = randn_cpu((M, K), seed=M).cuda()
    g = torch.Generator(device="cuda").manual_seed(N)
    codes = torch.randint(0, 120, (N, K), generator=g, device="cuda", dtype=torch.uint8).view(Q.FP8)
    fw = Q.FP8Weight(codes, torch.full((1, 1), 1e-3, device="cuda"), (N, K))
    want = Q.fp8_matmul(*Q.quantize_act(x), fw)
    n0 = Q.launch_count()
    assert torch.equal(Q.linear(x, fw), want)
    assert Q._NATIVE is None or Q.launch_count() - n0 == eager
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    n0 = Q.launch_count()
    with torch.cuda.graph(graph):
        y = Q.linear(x, fw)
    assert Q._NATIVE is None or Q.launch_count() - n0 == captured
    graph.replay()
    assert torch.equal(y, want)
    assert Q.device_status() == 0


@pytest.mark.parametrize("M,K,N,dt,eager,captured", [
    (1, 5760, 9600, torch.bfloat16, 1, 1), (3, 5888, 10240, torch.bfloat16, 1, 2), (5, 5760, 9600, torch.bfloat16, 2, 2),
    (1, 5760, 9984, torch.float32, 1, 1), (1, 11392, 4864, torch.float16, 1, 1), (2, 11776, 5120, torch.bfloat16, 1, 2),
    (1, 14336, 8192, torch.bfloat16, 1, 1), (1, 14208, 5248, torch.bfloat16, 1, 1), (2, 14336, 8192, torch.bfloat16, 2, 2),
    (1, 28672, 2048, torch.bfloat16, 2, 2), (1, 14464, 8192, torch.bfloat16, 2, 2)])
def test_linear_of_few_rows_whose_slices_leave_no_room_to_be_handed_over(Q, M, K, N, dt, eager, captured):
    """Slices as long as they can be: the launch fetches the partial sums, where that is still faster than two
    launches; the bits of quantizer and GEMM apart either way."""
    fw = Q.quantize_weight(randn_cpu((N, K), seed=1, scale=0.02).cuda())
    x, r = randn_cpu((M, K), seed=M, dtype=dt).cuda(), randn_cpu((M, N), seed=2, dtype=dt).cuda()
    n0 = Q.launch_count()
    got = Q.linear(x, fw, residual=r)
    assert Q._NATIVE is None or (Q.launch_count() - n0 == eager and Q.last_gemm_launch()["quantizes"] == (eager == 1))
    xq, sx = Q.quantize_act(x)
    want = Q.fp8_matmul(xq, sx, fw, out_dtype=dt, residual=r)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        n0 = Q.launch_count()
        again = Q.linear(x, fw, residual=r)
        assert Q._NATIVE is None or Q.launch_count() - n0 == captured
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(got, want) and torch.equal(again, want)
    assert Q.device_status() == 0


@pytest.mark.parametrize("key,value,back", [("stream_max_m", 8, 256), ("decode_wide", 1, -1), ("decode_stages", 2, 0),
                                            ("decode_b_stages", 1, 0)])
def test_linear_of_few_rows_leaves_forced_kernels_to_two_launches(Q, key, value, back):
    """An option that sends the batch to another kernel or forces a ring's depth: quantizer and that GEMM,
    bit for bit (another kernel sums K in another order: one rounding of the output away from the one
    launch)."""
    fw = Q.quantize_weight(randn_cpu((1024, 512), seed=1, scale=0.02).cuda())
    x = randn_cpu((16, 512), seed=2).cuda()
    n0 = Q.launch_count()
    want = Q.linear(x, fw)
    assert Q._NATIVE is None or Q.launch_count() - n0 == 1
    try:
        Q.set_option(key, value)
        n0 = Q.launch_count()
        got = Q.linear(x, fw)
        assert Q.launch_count() - n0 == 2
        assert torch.equal(got, Q.fp8_matmul(*Q.quantize_act(x), fw))
        assert key != "decode_stages" or Q.last_gemm_launch()["stages"] <= value
    finally:
        Q.set_option(key, back)
    assert max_rel(got, want) <= 2 ** -8
    assert Q.device_status() == 0


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float32], ids=["bf16", "fp32"])
@pytest.mark.parametrize("M,N,K", [(257, 4096, 512), (300, 272, 256), (413, 1040, 1040), (512, 16, 16), (1000, 4112, 2048)])
def test_prefill_residual_epilogue_over_row_pitches(Q, dt, M, N, K):
    """M > 256: ragged rows and columns, residual rows that start on 16 bytes or only on 8 (16-bit types),
    one that is a column block of a wider buffer; bit-equal to the separate add.  What records gradients
    stays a torch addition."""
    _, _, xq, sx, fw = _operands(Q, M, N, K, seed=M + N)
    y = Q.fp8_matmul(xq, sx, fw, out_dtype=dt)
    for off, pitch in ((0, N), (4, N + 20), (8, N + 16), (3, N + 8)):
        res = randn_cpu((M, pitch), seed=off, dtype=dt, scale=0.5).cuda()[:, off:off + N]
        assert torch.equal(Q.fp8_matmul(xq, sx, fw, out_dtype=dt, residual=res), res + y)
    res = randn_cpu((M, N), seed=9, dtype=dt).cuda().requires_grad_()
    assert Q.fp8_matmul(xq, sx, fw, out_dtype=dt, residual=res).requires_grad
    assert Q.device_status() == 0


def test_residual_strided_scoped_and_through_the_sublayers(Q):
    H, I, M = 4096, 12288, 16
    x = randn_cpu((M, 1, H), seed=1).cuda()
    mk = lambda n, k, s: Q.quantize_weight(randn_cpu((n, k), seed=s, scale=0.02).cuda())  # noqa: E731
    w_out, wg, wu, wd = mk(H, H, 2), mk(I, H, 3), mk(I, H, 4), mk(H, I, 5)
    wide = randn_cpu((M, 2 * H), seed=6).cuda()
    res = wide[:, H:]                                           # row stride 2H
    xq, sx = Q.quantize_act(x.reshape(M, H))
    assert torch.equal(Q.fp8_matmul(xq, sx, w_out, residual=res), res + Q.fp8_matmul(xq, sx, w_out))
    r3 = randn_cpu((M, 1, H), seed=8).cuda()
    assert torch.equal(Q.linear(x, w_out, residual=r3), r3 + Q.linear(x, w_out))
    assert torch.equal(Q.mlp_forward(x, wg, wu, wd, residual=r3), r3 + Q.mlp_forward(x, wg, wu, wd))
    # the scoped form: only the named weight takes the residual, and only once
    with Q.residual_into(w_out, r3) as slot:
        a = Q.linear(x, wd_t := mk(H, H, 9))                    # another weight: untouched
        assert not slot.taken
        b = Q.linear(x, w_out)
        assert slot.taken
        c = Q.linear(x, w_out)                                  # second call: plain again
    assert torch.equal(a, Q.linear(x, wd_t))
    assert torch.equal(b, r3 + Q.linear(x, w_out)) and torch.equal(c, Q.linear(x, w_out))
    with Q.residual_into(None, r3) as slot:
        assert torch.equal(Q.linear(x, w_out), c) and not slot.taken
    with pytest.raises(ValueError):
        Q.fp8_matmul(xq, sx, w_out, residual=r3.reshape(M, H)[:, :128])


# -- gate and up as one paired GEMM with SiLU*mul + quantization in the epilogue -----------------------
@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16, torch.float32], ids=["bf16", "fp16", "fp32"])
@pytest.mark.parametrize("M", [1, 8, 37, 128, 200, 256])
@pytest.mark.parametrize("I,K", [(12288, 4096), (9216, 2560), (1024, 512), (64, 128), (2048, 4096)],
                         ids=["9B", "4B", "small", "one_tile", "split4"])
def test_paired_gate_up_epilogue_equals_the_separate_kernels(Q, dt, M, I, K):
    """Codes and scale of h from the one-launch form against grouped GEMM + `silu_mul_quant`:
    every K split the shape rule produces (1, 2, 4), ragged M, three activation types."""
    if dt is not torch.bfloat16 and (I, K) not in ((9216, 2560), (1024, 512)):
        pytest.skip("dtype variants on two shapes")
    x = randn_cpu((M, K), seed=M + I, dtype=dt).cuda()
    gate = Q.quantize_weight(randn_cpu((I, K), seed=1, scale=0.02).cuda())
    up = Q.quantize_weight(randn_cpu((I, K), seed=2, scale=0.05).cuda())      # a different scale
    xq, sx = Q.quantize_act(x)
    g, u = Q.fp8_matmul_grouped(xq, sx, (gate, up), out_dtype=dt)
    hq_ref, sh_ref = Q.silu_mul_quant(g, u)
    got = Q.gate_up_silu_quant(xq, sx, gate, up, dt)
    if got is None:
        # the exchange needs the whole grid resident: with M > 128 the staging buffer allows one
        # CTA per SM, which tiles x K slices of the larger shapes exceed (192 for the 9B MLP,
        # 288 for the 4B one) -- the caller then runs 4 launches
        assert M > 128 and 2 * I // 128 > 74, "paired form refused a launch that fits"
        pytest.skip("grid not co-resident at this M: four-launch path")
    hq, sh = got
    assert torch.equal(sh, sh_ref), f"scale {sh.item():.9e} vs {sh_ref.item():.9e}"
    bad = int((hq.view(torch.uint8) != hq_ref.view(torch.uint8)).sum())
    assert bad == 0, f"{bad} of {hq.numel()} codes differ"
    assert Q.device_status() == 0


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16, torch.float32], ids=["bf16", "fp16", "fp32"])
@pytest.mark.parametrize("M,I,K", [(300, 1024, 512), (1000, 12288, 4096), (2048, 1536, 4096),
                                   (4100, 272, 1040)],
                         ids=["small", "9B", "shard_of_8", "ragged"])
def test_prefill_gate_up_silu_equals_the_separate_kernels(Q, dt, M, I, K):
    """M > 256: h = silu(gate) * up and its scale written by the CTA-pair GEMM's epilogue, then
    `cast_act`, against the grouped GEMM + torch's SiLU*mul + the quantizer: h, scale and codes
    bit for bit (three activation types, I off the tile grid, ragged M)."""
    if dt is not torch.bfloat16 and (M, I) not in ((300, 1024), (4100, 272)):
        pytest.skip("dtype variants on two shapes")
    x = randn_cpu((M, K), seed=M + I, dtype=dt).cuda()
    gate = Q.quantize_weight(randn_cpu((I, K), seed=1, scale=0.02).cuda())
    up = Q.quantize_weight(randn_cpu((I, K), seed=2, scale=0.05).cuda())
    xq, sx = Q.quantize_act(x)
    g, u = Q.fp8_matmul_grouped(xq, sx, (gate, up), out_dtype=dt)
    h_ref = F.silu(g) * u
    hq_ref, sh_ref = Q.quantize_act(h_ref)
    got = Q.gate_up_silu(xq, sx, gate, up, dt)
    assert got is not None and Q.last_gemm_launch()["kernel"] == "pair"
    h, sh = got
    assert torch.equal(h, h_ref), f"{int((h != h_ref).sum())} of {h.numel()} h values differ"
    assert torch.equal(sh, sh_ref), f"scale {sh.item():.9e} vs {sh_ref.item():.9e}"
    assert torch.equal(Q.cast_act(h, sh).view(torch.uint8), hq_ref.view(torch.uint8))
    h2, sh2 = Q.gate_up_silu(xq, sx, gate, up, dt)          # the scratch words were returned to zero
    assert torch.equal(h2, h) and torch.equal(sh2, sh)
    assert Q.device_status() == 0


@pytest.mark.parametrize("M", [1, 2, 3, 5, 15, 16, 17, 31, 33, 47, 48, 49])
def test_slices_handed_over_add_up_to_the_fetched_sum(Q, M):
    """Up to 48 rows the K slices of a tile are written into the CTA that sums them, beyond they are fetched: a row's
    bits do not depend on which, for 2 and 4 slices, weights that end inside a tile and rows that no CTA owns."""
    K = 4096
    x = randn_cpu((60, K), seed=5).cuda()
    xq, sx = Q.quantize_act(x)
    ws = [Q.quantize_weight(randn_cpu((n, K), seed=n, scale=0.02).cuda()) for n in (8192, 4096, 1040, 16)]
    r = randn_cpu((60, 4096), seed=6).cuda()
    Q.set_option("decode_wide", 0)
    try:
        far = Q.fp8_matmul_grouped(xq, sx, ws)                       # 60 rows: fetched
        near = Q.fp8_matmul_grouped(xq[:M].contiguous(), sx, ws)
        assert not Q.last_gemm_launch()["wide"]
        for a, b in zip(near, far):
            assert torch.equal(a, b[:M])
        assert torch.equal(Q.fp8_matmul(xq[:M].contiguous(), sx, ws[1], residual=r[:M]),
                           Q.fp8_matmul(xq, sx, ws[1], residual=r)[:M])
    finally:
        Q.set_option("decode_wide", -1)
    assert Q.device_status() == 0


@pytest.mark.parametrize("M", [44, 45, 48])
@pytest.mark.parametrize("N,K", [(9728, 5760), (10240, 2048), (5120, 2560)])
def test_slices_of_halves_are_handed_over_only_beside_four_stages(Q, M, N, K):
    """Two CTAs per SM: the area for the slices is not bought with the weight ring, where slices are long; the bits of
    the fetched sum."""
    x = randn_cpu((60, K), seed=5).cuda()
    xq, sx = Q.quantize_act(x)
    w = Q.quantize_weight(randn_cpu((N, K), seed=N, scale=0.02).cuda())
    Q.set_option("decode_wide", 0)
    try:
        far = Q.fp8_matmul(xq, sx, w)
        near = Q.fp8_matmul(xq[:M].contiguous(), sx, w)
        launch = Q.last_gemm_launch()
        assert not launch["wide"] and (launch["split"] != 2 or launch["stages"] >= 4)
        assert torch.equal(near, far[:M])
    finally:
        Q.set_option("decode_wide", -1)
    assert Q.device_status() == 0


@pytest.mark.parametrize("M,I,dt", [(1, 12288, torch.bfloat16), (6, 12288, torch.bfloat16), (7, 12288, torch.bfloat16),
                                    (5, 12288, torch.float16), (3, 12288, torch.float32), (4, 12288, torch.float32),
                                    (6, 8256, torch.bfloat16), (2, 8128, torch.bfloat16)])
def test_mlp_of_few_rows_casts_h_in_the_down_projection(Q, M, I, dt):
    """Up to 6 rows (3 of fp32) and from a down weight of 32 Mi values on, h is cast by the CTAs of the down projection:
    the bits of the separate launches at either side of both lines (seen in the last launch), with a last K block that is
    half full, with an infinity and a NaN in h, and again with the scratch that the calls before returned to zero."""
    H = 4096
    takes = Q._NATIVE is not None and M <= (3 if dt is torch.float32 else 6) and I * H >= 32 << 20
    mk = lambda n, k, s: Q.quantize_weight(randn_cpu((n, k), seed=s, scale=0.02).cuda())  # noqa: E731
    wg, wu, wd = mk(I, H, 3), mk(I, H, 4), mk(H, I, 5)
    r = randn_cpu((M, H), seed=M + 1, dtype=dt).cuda()
    big = torch.finfo(torch.float16).max if dt is torch.float16 else torch.finfo(dt).max
    for case in ("plain", "zeros", "inf", "nan"):
        x = randn_cpu((M, H), seed=M, dtype=dt).cuda()
        if case == "zeros":
            x.zero_()
        xq, sx = Q.quantize_act(x)
        if case in ("inf", "nan"):
            sx = torch.full_like(sx, big if case == "inf" else float("nan"))
        h = Q.QuantizedActivation(xq, sx, x.shape, dt)
        Q.set_paired_mlp(False)
        want, want_r = Q.mlp_forward(h, wg, wu, wd), Q.mlp_forward(h, wg, wu, wd, residual=r)
        Q.set_paired_mlp(True)
        for _ in range(2):
            n0 = Q.launch_count()
            got = Q.mlp_forward(h, wg, wu, wd)
            assert Q.launch_count() - n0 == 2 and Q.last_gemm_launch()["quantizes"] == takes
            got_r = Q.mlp_forward(h, wg, wu, wd, residual=r)
            for a, b in ((got, want), (got_r, want_r)):
                assert torch.equal(a.isnan(), b.isnan()) and torch.equal(a.nan_to_num(), b.nan_to_num()), case
    assert Q.device_status() == 0


@pytest.mark.parametrize("M,H,I,takes", [(4, 5120, 11264, 1), (5, 5120, 11264, 0), (6, 5120, 10752, 1), (6, 4096, 14336, 1),
                                         (1, 4736, 28160, 1), (3, 9216, 4096, 1), (2, 9216, 14144, 0), (2, 10368, 3328, 1),
                                         (2, 10368, 7232, 0)])
def test_mlp_of_few_rows_at_other_widths(Q, M, H, I, takes):
    """1, 2 and 4 slices of h, one and two CTAs per SM, slices that take two rounds of loads, either side of what fits:
    the bits of the separate launches, and which form ran."""
    from braid_b200 import _lib
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("what fits is a matter of the SMs")
    g = torch.Generator(device="cuda").manual_seed(H + I)

    def weight(n, k):
        codes = torch.randint(0, 0x60, (n, k), generator=g, device="cuda", dtype=torch.uint8)
        codes |= torch.randint(0, 2, (n, k), generator=g, device="cuda", dtype=torch.uint8) << 7
        return Q.FP8Weight(codes.view(Q.FP8), torch.full((1, 1), 1e-3, device="cuda"), (n, k))

    wg, wu, wd = weight(I, H), weight(I, H), weight(H, I)
    x, r = randn_cpu((M, H), seed=M).cuda(), randn_cpu((M, H), seed=M + 1).cuda()
    h = Q.QuantizedActivation(*Q.quantize_act(x), x.shape, x.dtype)
    assert _lib.load().bq_mlp_w8a8_takes(M, I, H, 1) == takes
    got = Q.mlp_forward(h, wg, wu, wd, residual=r)
    assert Q.last_gemm_launch()["quantizes"] == (takes == 1 and Q._NATIVE is not None)
    Q.set_paired_mlp(False)
    try:
        assert torch.equal(got, Q.mlp_forward(h, wg, wu, wd, residual=r))
    finally:
        Q.set_paired_mlp(True)
    assert Q.device_status() == 0


@pytest.mark.parametrize("M,H,I,dt,takes", [(2, 4096, 8192, torch.bfloat16, 1), (4, 4096, 8192, torch.float32, 0),
                                            (2, 5120, 11328, torch.bfloat16, 0)])
def test_mlp_of_few_rows_that_is_refused_allocates_nothing_for_it(Q, M, H, I, dt, takes):
    """h and y where both products are one call, else codes, scale and y: what is refused by its rows or its width is
    known to be before any of them is made."""
    if Q._NATIVE is None:
        pytest.skip("the native calls are not loaded")
    from braid_b200 import _lib
    codes = lambda n, k: Q.FP8Weight(torch.zeros(n, k, device="cuda", dtype=torch.uint8).view(Q.FP8),  # noqa: E731
                                     torch.ones(1, 1, device="cuda"), (n, k))
    wg, wu, wd = codes(I, H), codes(I, H), codes(H, I)
    assert _lib.load().bq_mlp_w8a8_takes(M, I, H, {torch.bfloat16: 1, torch.float32: 0}[dt]) == takes
    x = Q.QuantizedActivation(*Q.quantize_act(randn_cpu((M, H), seed=1, dtype=dt).cuda()), (M, H), dt)
    before = torch.cuda.memory_stats()["allocation.all.allocated"]
    Q.mlp_forward(x, wg, wu, wd)
    assert torch.cuda.memory_stats()["allocation.all.allocated"] - before == (2 if takes else 3)
    assert Q.device_status() == 0


def test_mlp_of_few_rows_leaves_its_scratch_clean_when_the_second_launch_fails(Q):
    """The maximum of h stays in the scratch between the two launches: a second one that cannot be made (injected on the
    host) returns it to zero, and the call is made again by the separate launches."""
    from braid_b200 import _lib
    H, I = 4096, 8192
    mk = lambda n, k, s: Q.quantize_weight(randn_cpu((n, k), seed=s, scale=0.02).cuda())  # noqa: E731
    wg, wu, wd = mk(I, H, 3), mk(I, H, 4), mk(H, I, 5)
    x = randn_cpu((2, H), seed=1).cuda()
    xq, sx = Q.quantize_act(x)
    want = Q.mlp_forward(x, wg, wu, wd)
    lib, h, y = _lib.load(), torch.empty(2, I, device="cuda", dtype=x.dtype), torch.empty_like(x)
    slot = torch.zeros(4, device="cuda", dtype=torch.int32)
    call = lambda: lib.bq_mlp_w8a8(  # noqa: E731
        xq.data_ptr(), sx.data_ptr(), *[w.data.data_ptr() for w in (wg, wu, wd)], *[w.scale.data_ptr() for w in (wg, wu, wd)],
        None, 0, 2, H, I, H, 1, h.data_ptr(), y.data_ptr(), H, slot.data_ptr(), 16, Q._stream_ptr(x.device))
    try:
        Q.set_option("fail_stream_launch", 2)
        assert call() == _lib.BQ_ERR_LAUNCH
        assert slot.tolist() == [0, 0, 0, 0] and h.abs().max() > 0         # the first launch ran
        assert call() == _lib.BQ_OK and torch.equal(y, want) and slot.tolist() == [0, 0, 0, 0]
        Q.set_option("fail_stream_launch", 2)
        assert torch.equal(Q.mlp_forward(x, wg, wu, wd), want)
    finally:
        Q.set_option("fail_stream_launch", 0)
    assert Q.device_status() == 0


@pytest.mark.parametrize("M", [129, 144, 200, 256])
def test_mlps_of_more_than_128_rows_back_to_back(Q, M):
    """More than 128 rows take half of an SM's tensor memory, and gate/up waits for the whole grid: launches of small
    weights, of which three CTAs would fit an SM, take the shared memory that keeps the third out.  MLPs without a launch
    between them, captured and replayed, have the bits of the four-launch form, and no wait runs out."""
    H, I = 1024, 3072
    ws = [[Q.quantize_weight(randn_cpu((n, k), seed=s + j, scale=0.02).cuda()) for j, (n, k) in enumerate(((I, H), (I, H), (H, I)))]
          for s in (1, 11, 21)]
    x = randn_cpu((M, H), seed=M).cuda()
    h = Q.QuantizedActivation(*Q.quantize_act(x), x.shape, x.dtype)
    Q.set_paired_mlp(False)
    want = [Q.mlp_forward(h, *w) for w in ws]
    Q.set_paired_mlp(True)
    Q.set_option("decode_wide", 0)
    try:
        got = [Q.mlp_forward(h, *w) for w in ws]
        launch = Q.last_gemm_launch()
        assert launch["kernel"] == "stream" and not launch["wide"] and 3 * (launch["smem"] + 1024) > 233472
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            again = [Q.mlp_forward(h, *w) for w in ws for _ in range(2)]
        graph.replay()
        graph.replay()
        torch.cuda.synchronize()
        assert Q.device_status() == 0
        for a, b in zip(got, want):
            assert torch.equal(a, b)
        for a, b in zip(again, [b for b in want for _ in range(2)]):
            assert torch.equal(a, b)
    finally:
        Q.set_option("decode_wide", -1)


def test_paired_mlp_equals_the_four_launch_mlp_and_replays(Q):
    H, I = 4096, 12288
    mk = lambda n, k, s: Q.quantize_weight(randn_cpu((n, k), seed=s, scale=0.02).cuda())  # noqa: E731
    wg, wu, wd = mk(I, H, 3), mk(I, H, 4), mk(H, I, 5)
    for M in (1, 16, 128, 300):
        x = randn_cpu((M, H), seed=M).cuda()
        r = randn_cpu((M, H), seed=M + 1).cuda()
        Q.set_paired_mlp(False)
        want, want_r = Q.mlp_forward(x, wg, wu, wd), Q.mlp_forward(x, wg, wu, wd, residual=r)
        Q.set_paired_mlp(True)
        n0 = Q.launch_count()
        got = Q.mlp_forward(x, wg, wu, wd)
        assert Q.launch_count() - n0 == (3 if M <= 128 else 4)
        assert torch.equal(got, want) and torch.equal(Q.mlp_forward(x, wg, wu, wd, residual=r), want_r)
    # the one-launch form reads the two weights in place: no copy of either is made or kept
    free0 = torch.cuda.mem_get_info()[0]
    Q.mlp_forward(randn_cpu((16, H), seed=2).cuda(), wg, wu, wd)
    torch.cuda.synchronize()
    assert free0 - torch.cuda.mem_get_info()[0] < 32 << 20
    # capture + replay
    x = randn_cpu((128, H), seed=9).cuda()
    eager = Q.mlp_forward(x, wg, wu, wd).clone()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        for _ in range(3):
            Q.mlp_forward(x, wg, wu, wd)
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = Q.mlp_forward(x, wg, wu, wd)
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, eager) and Q.device_status() == 0


def _pitched(Q, xq, sx, w, M, n):
    buf = torch.full((M, n + 4), 7.0, dtype=torch.bfloat16, device="cuda")
    Q.fp8_matmul_grouped(xq, sx, [w], out=[buf[:, :n]])
    return buf


@pytest.fixture
def wide(Q):
    Q.set_option("decode_wide", 1)
    yield
    Q.set_option("decode_wide", -1)


@pytest.mark.parametrize("M,ns,K", [(1, (48,), 256), (33, (16,), 128), (40, (48, 1040), 4096), (64, (4096, 1024), 1040),
                                    (65, (272,), 2560), (127, (4096,), 16), (128, (8192, 1024, 1024), 4096),
                                    (129, (4736,), 512), (200, (1040, 32), 2064), (256, (12288, 4096), 1024)])
def test_wide_batches_on_cta_pairs_agree_with_the_k_sliced_kernel(Q, M, ns, K):
    """Wide decode batches run on CTA pairs (one round of units over the whole of K); the option selects
    that kernel or the K-sliced one for any batch.  Edges: one unit, the last unit short, K below and beyond a 128-byte block,
    batches that fill half of a pair's rows, all of them, and one row more."""
    x = randn_cpu((M, K), seed=M + K).cuda()
    xq, sx = Q.quantize_act(x)
    ws = [Q.quantize_weight((randn_cpu((n, K), seed=n) * 0.02).cuda()) for n in ns]
    a = xq.float().double() * sx.double()

    def both(fn):
        out = []
        try:
            for wide in (1, 0):
                Q.set_option("decode_wide", wide)
                out.append(fn())
                assert Q.last_gemm_launch()["wide"] == bool(wide)
        finally:
            Q.set_option("decode_wide", -1)
        return out

    got, want = both(lambda: Q.fp8_matmul_grouped(xq, sx, ws, out_dtype=torch.float32))
    for y, z, w in zip(got, want, ws):
        assert torch.equal(y, z)      # the same sums in the same order: the choice of a kernel shows in no result
        b = w.data.float().double() * w.scale.double()
        # an fp32 sum of K products, 32 of them per step of the accumulator, each step off by at most
        # two units of the last place of the sum of magnitudes; the scaling adds two more
        bound = (K / 32 + 2) * 2.0 ** -22 * (a.abs() @ b.abs().t()) + 1e-30
        for t in (y, z):
            assert ((t.double() - a @ b.t()).abs() <= bound).all()
        for t, alone in zip((y, z), both(lambda: Q.fp8_matmul(xq, sx, w, out_dtype=torch.float32))):
            assert torch.equal(t, alone)
    # a residual, and an output row pitch that allows 8-byte accesses only
    n = ns[0]
    res = randn_cpu((M, n), seed=9).cuda()
    got, want = both(lambda: Q.linear(x, ws[0], residual=res))
    assert max_rel(got, want.double()) <= TOL_BF16
    for buf, plain in zip(both(lambda: _pitched(Q, xq, sx, ws[0], M, n)), both(lambda: Q.fp8_matmul(xq, sx, ws[0]))):
        assert torch.equal(buf[:, :n], plain) and bool((buf[:, n:] == 7.0).all())
    assert Q.device_status() == 0


def test_forced_ring_depths_leave_the_flags_of_the_wide_kernel_alone(Q, wide):
    """The deepest rings that options can ask for: 40 weight stages and as many activation stages as
    the barrier area has room for (its last bytes hold the tensor-memory address)."""
    M, n, K = 8, 48, 41 * 128 + 16
    x = randn_cpu((M, K), seed=1).cuda()
    xq, sx = Q.quantize_act(x)
    w = Q.quantize_weight((randn_cpu((n, K), seed=2) * 0.02).cuda())
    base = Q.fp8_matmul(xq, sx, w, out_dtype=torch.float32)
    try:
        for depth in (28, 29, 40, 1000):
            Q.set_option("decode_b_stages", depth)
            assert torch.equal(base, Q.fp8_matmul(xq, sx, w, out_dtype=torch.float32))
            assert Q.last_gemm_launch()["stages"] == 40 and Q.last_gemm_launch()["wide"]
    finally:
        Q.set_option("decode_b_stages", 0)
    assert Q.device_status() == 0


@pytest.mark.parametrize("M,I,K,dt", [(33, 64, 128, torch.bfloat16), (64, 4736, 1040, torch.float16),
                                      (96, 1024, 2048, torch.float32), (130, 192, 256, torch.bfloat16),
                                      (256, 12288, 1024, torch.bfloat16)])
def test_wide_gate_up_codes_equal_the_separate_kernels(Q, wide, M, I, K, dt):
    x = randn_cpu((M, K), seed=1, dtype=dt).cuda()
    xq, sx = Q.quantize_act(x)
    g, u = (Q.quantize_weight((randn_cpu((I, K), seed=s) * 0.05).cuda()) for s in (2, 3))
    got = Q.gate_up_silu_quant(xq, sx, g, u, dt)
    assert Q.last_gemm_launch()["wide"]
    gate, up = Q.fp8_matmul_grouped(xq, sx, (g, u), out_dtype=dt)
    q, s = Q.silu_mul_quant(gate, up)
    assert got is not None and torch.equal(got[1], s) and torch.equal(u8(got[0]), u8(q))
    assert Q.device_status() == 0


@pytest.mark.parametrize("M", [33, 64, 129])
def test_wide_greedy_pick_over_several_rounds(Q, wide, M):
    V, K = 60016, 256
    w = Q.quantize_weight((randn_cpu((V, K), seed=3) * 0.02).cuda())
    w.data.view(torch.uint8)[V - 16:] = w.data.view(torch.uint8)[:16]      # equal logits: the lower index wins
    x = randn_cpu((M, K), seed=M).cuda()
    idx, logits = Q.lm_head_argmax(x, w, return_logits=True)
    assert Q.last_gemm_launch()["wide"]
    assert torch.equal(idx.flatten(), logits.argmax(-1).flatten())
    xq, sx = Q.quantize_act(x)
    assert torch.equal(logits, Q.fp8_matmul(xq, sx, w))
    assert Q.device_status() == 0


@pytest.mark.parametrize("n,k,on,off", [
    (4096, 4096, (49, 128, 161, 256), (48, 129, 160)),        # one round
    (9472, 1024, (65,), (49, 64)), (9472, 2048, (49,), ()), (18944, 1024, (49, 176), (177, 256)),  # all pairs, short K
    (1024, 8192, (161,), ()), (1024, 12288, (225,), (161, 224)),                                  # long K, few rows
    (20480, 1024, (209,), (65, 208)), (32000, 1536, (65, 161), (64, 129)),                        # two rounds
    (32000, 2048, (97, 161), (96, 129)), (24576, 2048, (33, 129), (32,)), (49152, 2048, (33, 129), (32,))])
def test_which_decode_batches_run_on_cta_pairs(Q, n, k, on, off):
    """Both sides of every line of the dispatch.  Both kernels give the same bits, so that a grouped launch
    and per-weight calls agree although the lines may part them."""
    g = torch.Generator(device="cuda").manual_seed(n + k)
    data = torch.randint(0, 120, (n, k), generator=g, device="cuda", dtype=torch.uint8)
    w = Q.FP8Weight(data=data.view(Q.FP8), scale=torch.full((1, 1), 1e-3, device="cuda"), shape=(n, k))
    torch.cuda.synchronize()
    for M, wide in [(m, True) for m in on] + [(m, False) for m in off]:
        xq, sx = Q.quantize_act(randn_cpu((M, k), seed=M).cuda())
        y = Q.fp8_matmul(xq, sx, w, out_dtype=torch.float32)
        assert Q.last_gemm_launch()["wide"] == wide, f"{M} x {n} x {k}"
        try:
            Q.set_option("decode_wide", int(not wide))
            assert torch.equal(y, Q.fp8_matmul(xq, sx, w, out_dtype=torch.float32))
        finally:
            Q.set_option("decode_wide", -1)
    assert Q.device_status() == 0


@pytest.mark.parametrize("M,I,wide", [(48, 16384, False), (49, 16384, True), (160, 9472, False), (161, 9472, True)])
def test_which_gate_up_batches_run_on_cta_pairs(Q, M, I, wide):
    xq, sx = Q.quantize_act(randn_cpu((M, 256), seed=M).cuda())
    g, u = (Q.quantize_weight((randn_cpu((I, 256), seed=s) * 0.05).cuda()) for s in (1, 2))
    assert Q.gate_up_silu_quant(xq, sx, g, u, torch.bfloat16) is not None
    assert Q.last_gemm_launch()["wide"] == wide
    assert Q.device_status() == 0


def test_what_the_wide_kernel_has_no_layout_for_runs_on_the_k_sliced_one(Q, wide):
    """A vocabulary so small that the picks of the unit walkers do not fit the caller's scratch (a pair
    per row and 128 vocabulary rows), with the option that asks for the wide kernel."""
    x = randn_cpu((64, 256), seed=1).cuda()
    w = Q.quantize_weight((randn_cpu((1024, 256), seed=2) * 0.02).cuda())
    idx, logits = Q.lm_head_argmax(x, w, return_logits=True)
    assert not Q.last_gemm_launch()["wide"]
    assert torch.equal(idx.flatten(), logits.argmax(-1).flatten())
    # gate and up of more rows than one round of units holds: refused, as without the option
    xq, sx = Q.quantize_act(x)
    g, u = (Q.quantize_weight((randn_cpu((20480, 256), seed=s) * 0.05).cuda()) for s in (3, 4))
    assert Q.gate_up_silu_quant(xq, sx, g, u, torch.bfloat16) is None
    assert Q.device_status() == 0


@pytest.mark.parametrize("M", [33, 64, 200])
@pytest.mark.parametrize("K", [192, 1040, 4096])
def test_wide_16_bit_segments_over_several_rounds(Q, wide, M, K):
    """Segments of 16-bit weights beside FP8 ones in a launch of more units than are resident: both kinds
    share one ring layout, the first and the last unit of a walker may be of either kind."""
    dt = torch.bfloat16
    x = randn_cpu((M, K), seed=M + K, dtype=dt).cuda()
    a, b = (randn_cpu((n, K), seed=n, dtype=dt, scale=0.02).cuda() for n in (32, 272))
    w = Q.quantize_weight(randn_cpu((40960, K), seed=1, dtype=dt, scale=0.02).cuda())
    ya, yw, yb = Q.project(x, a, w, b)
    launch = Q.last_gemm_launch()
    assert launch["wide"] and launch["grid"] % 2 == 0 and 40960 // 256 > launch["grid"] // 2   # several rounds
    xq, sx = Q.quantize_act(x)
    assert torch.equal(yw, Q.fp8_matmul(xq, sx, w, out_dtype=dt))
    for y, d in ((ya, a), (yb, b)):
        # products of 16-bit values are exact in fp32; what is left is one rounding to the output type
        # and fp32 sums of K products
        ref = x.double() @ d.double().t()
        bound = 2.0 ** -8 * ref.abs() + K * 2.0 ** -22 * (x.double().abs() @ d.double().abs().t())
        assert ((y.double() - ref).abs() <= bound).all()
    assert Q.device_status() == 0


@pytest.mark.parametrize("n,k", [(272, 1040), (1024, 512), (12288, 4096)])
def test_a_fresh_weight_is_complete_before_a_queued_gemm_reads_it(Q, n, k):
    """The GEMMs fetch weights ahead of the kernels before them.  With the host far ahead of the device,
    quantize_weight -> GEMM -- directly, and with a quantizer or a norm in between -- must still see
    whole weights: eagerly, where a weight's memory held another one's codes, and in a graph whose
    source weights change between replays."""
    srcs = [(randn_cpu((n, k), seed=10 + i) * 0.02).cuda() for i in range(4)]
    x = randn_cpu((64, k), seed=1).cuda()
    gamma = torch.ones(k, device="cuda")
    xq, sx = Q.quantize_act(x)
    busy = torch.randn(4096, 4096, device="cuda")

    def chain(src, wait=lambda: None):
        out = []
        for rows in (8, 64):
            q8, xr = xq[:rows], x[:rows]
            w = Q.quantize_weight(src)
            wait()
            out.append(Q.fp8_matmul(q8, sx, w))
            w = Q.quantize_weight(src)
            wait()
            out.append(Q.linear(xr, w))                                  # a quantizer in between
            w = Q.quantize_weight(src)
            wait()
            out.append(Q.linear(Q.rms_norm_quant(xr, gamma, 1e-6), w))   # a norm in between
            w = Q.quantize_weight(src)
            wait()
            out.append(Q.lm_head_argmax(xr, w))
            g, u = Q.quantize_weight(src), Q.quantize_weight(src.neg())
            wait()
            if n % 64 == 0:
                out.extend(Q.gate_up_silu_quant(q8, sx, g, u, torch.bfloat16) or ())
        return out

    want = [chain(s, torch.cuda.synchronize) for s in srcs]
    torch.cuda.synchronize()
    for _ in range(3):
        for src, ref in zip(srcs, want):
            for _ in range(8):
                busy = (busy @ busy).clamp(-1, 1)                        # the device falls behind
            for a, b in zip(chain(src), ref, strict=True):
                assert torch.equal(u8(a), u8(b))
    src = srcs[0].clone()
    with torch.cuda.stream(torch.cuda.Stream()):
        chain(src)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = chain(src)
    for s, ref in zip(srcs, want):
        src.copy_(s)
        graph.replay()
        for a, b in zip(out, ref, strict=True):
            assert torch.equal(u8(a), u8(b))
    assert Q.device_status() == 0
