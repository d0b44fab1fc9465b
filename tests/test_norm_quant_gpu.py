"""RMSNorm fused into the quantizer, against the reference's torch spelling on the same device.

A sum of squares depends on the order of the additions, so bit identity with `F.rms_norm` is a
property of THIS torch build's CUDA kernel that the fused kernels restate; these tests are the
pin.  Every comparison is `torch.equal` on the dense activation, the scale and the code bytes.
Spec: braid/model/norm.py:31-45 (`rms_norm`), :48-71 (`rms_norm_gated`), consumed at
braid/model/layer.py:49,59 and braid/model/gdn.py:373-387.
"""
from __future__ import annotations

import pytest
import torch
import torch.nn.functional as F

from oracle import torch_spelling as TS
from _util import captured_kernels, randn_cpu, u8

pytestmark = pytest.mark.gpu

EPS = 1e-6


def _gamma(n, seed, spread=0.02):
    g = torch.Generator().manual_seed(seed)
    return (1.0 + spread * torch.randn(n, generator=g)).cuda()


def _same(qa, h_ref, what):
    qr, sr = TS.quantize_act(h_ref.reshape(-1, h_ref.shape[-1]))
    assert torch.equal(qa.scale, sr), f"{what}: scale {qa.scale.item():.9e} vs {sr.item():.9e}"
    diff = int((u8(qa.q) != u8(qr)).sum())
    assert diff == 0, f"{what}: {diff} of {qr.numel()} fp8 bytes differ"


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float32, torch.float16], ids=["bf16", "fp32", "fp16"])
@pytest.mark.parametrize("shape", [(1, 4096), (8, 4096), (37, 4096), (128, 4096), (128, 2560),
                                   (16, 8192), (5, 512), (3, 64), (256, 4096), (1024, 4096)])
def test_rms_norm_quant_is_bit_identical(Q, dt, shape):
    for seed in range(3):
        x = randn_cpu(shape, seed=seed * 101 + shape[0], dtype=dt, scale=(0.05, 1.0, 30.0)[seed]).cuda()
        gamma = _gamma(shape[1], seed, spread=(0.02, 0.3, 1.0)[seed])
        ref = TS.rms_norm(x, gamma, EPS)
        qa = Q.rms_norm_quant(x, gamma, EPS, keep_dense=True)
        assert qa.shape == x.shape and qa.dtype is dt
        bad = int((u8(qa.dense) != u8(ref)).sum())
        assert bad == 0, f"{dt} {shape} seed {seed}: {bad} bytes of the normalised activation differ"
        _same(qa, ref, f"{dt} {shape} seed {seed}")
        assert Q.rms_norm_quant(x, gamma, EPS).dense is None


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float32], ids=["bf16", "fp32"])
@pytest.mark.parametrize("rows,cols", [(768, 4096), (769, 4096), (770, 64), (803, 5120), (1777, 4096), (2366, 4096), (1003, 8192),
                                       (899, 516), (2369, 1024), (3552, 64), (3553, 1024), (1776, 2048), (1777, 2048),
                                       (2369, 2048), (1184, 4096), (1185, 4096), (2369, 4096), (1185, 8192)])
def test_rms_norm_quant_with_several_rows_per_block(Q, dt, rows, cols):
    """Beyond 768 rows a block normalises four or eight rows, as long as all of them are resident at once: both counts of
    each type, either side of each limit (seen in the launches), blocks with rows left over, vectors that end inside a
    thread's share, strided rows, and a NaN in the last row."""
    x = randn_cpu((rows, 2 * cols), seed=rows, dtype=dt, scale=2.0).cuda()[:, :cols]
    gamma = _gamma(cols, 7)
    ref = TS.rms_norm(x, gamma, EPS)
    per_sm = {torch.bfloat16: ((2048, 24), (4096, 16), (8192, 8)), torch.float32: ((1024, 24), (2048, 16), (4096, 8))}[dt]
    room = next((n for c, n in per_sm if cols <= c), 0) * torch.cuda.get_device_properties(0).multi_processor_count
    for keep in (True, False):
        n0 = Q.launch_count()
        qa = Q.rms_norm_quant(x, gamma, EPS, keep_dense=keep)
        assert rows <= 768 or Q.launch_count() - n0 == (1 if rows <= room else 2)
        if keep:
            assert int((u8(qa.dense) != u8(ref)).sum()) == 0
        _same(qa, ref, f"{rows} x {cols}")
    x[-1, -1] = float("nan")
    assert Q.rms_norm_quant(x, gamma, EPS).scale.isnan().all()
    assert not Q.rms_norm_quant(x[:-1], gamma, EPS).scale.isnan().any()
    assert Q.device_status() == 0


@pytest.mark.parametrize("dt", [torch.float16, torch.float32], ids=["fp16", "fp32"])
@pytest.mark.parametrize("rows,cols", [(256, 2048), (257, 2048), (259, 64), (384, 4096), (385, 4096), (387, 2052), (511, 1028)])
def test_rms_norm_quant_from_where_rows_share_a_block(Q, dt, rows, cols):
    """Rows of up to 2048 columns share a block from 257 rows on, of up to 4096 from 385: either side of both lines, rows
    left over in the last block, vectors that end inside a thread's share, strided rows, with and without the dense output."""
    x = randn_cpu((rows, 2 * cols), seed=rows, dtype=dt, scale=2.0).cuda()[:, cols:]
    gamma = _gamma(cols, 9)
    ref = TS.rms_norm(x, gamma, EPS)
    for keep in (True, False):
        n0 = Q.launch_count()
        qa = Q.rms_norm_quant(x, gamma, EPS, keep_dense=keep)
        assert Q.launch_count() - n0 == 1
        if keep:
            assert int((u8(qa.dense) != u8(ref)).sum()) == 0
        _same(qa, ref, f"{rows} x {cols}")
    x[-1, 0] = float("nan")
    assert Q.rms_norm_quant(x, gamma, EPS).scale.isnan().all()
    assert Q.device_status() == 0


def test_rms_norm_quant_many_rows_of_real_width(Q):
    """2048 independent rows x 3 magnitudes: a reduction-order mismatch shows up as a last-bit
    difference in a few percent of rows, so this is the statistical net under the exact cases."""
    for seed, scale in enumerate((1e-3, 1.0, 200.0)):
        x = randn_cpu((2048, 4096), seed=40 + seed, scale=scale).cuda()
        x[::7] *= 16.0          # rows of very different energy
        gamma = _gamma(4096, seed)
        ref = TS.rms_norm(x, gamma, EPS)
        qa = Q.rms_norm_quant(x, gamma, EPS, keep_dense=True)
        rows_bad = int((qa.dense != ref).any(dim=1).sum())
        assert rows_bad == 0, f"{rows_bad} of 2048 rows differ at scale {scale}"
        _same(qa, ref, f"scale {scale}")


def test_rms_norm_quant_strided_rows_leading_dims_and_fallback(Q):
    gamma = _gamma(4096, 1)
    wide = randn_cpu((16, 8192), seed=2).cuda()
    x = wide[:, :4096]                                  # row stride 8192
    qa = Q.rms_norm_quant(x, gamma, EPS, keep_dense=True)
    ref = TS.rms_norm(x, gamma, EPS)
    assert torch.equal(qa.dense, ref)
    _same(qa, ref, "strided")
    x3 = randn_cpu((4, 3, 4096), seed=3).cuda()         # [B, T, H] as the layer sees it
    qa = Q.rms_norm_quant(x3, gamma, EPS, keep_dense=True)
    assert qa.shape == x3.shape and qa.dense.shape == x3.shape and qa.q.shape == (12, 4096)
    _same(qa, TS.rms_norm(x3, gamma, EPS), "3-d")
    big = randn_cpu((4096, 4096), seed=4).cuda()        # more rows than fit at once: two steps
    qa = Q.rms_norm_quant(big, gamma, EPS, keep_dense=True)
    ref = TS.rms_norm(big, gamma, EPS)
    assert torch.equal(qa.dense, ref)
    _same(qa, ref, "4096 rows")


@pytest.mark.parametrize("dt,shape", [(torch.bfloat16, (8192, 4096)), (torch.bfloat16, (2500, 2560)),
                                      (torch.float32, (3000, 4096)), (torch.float16, (4100, 512))],
                         ids=["bf16-8192x4096", "bf16-2500x2560", "fp32-3000x4096", "fp16-4100x512"])
def test_rms_norm_quant_at_prefill_sizes(Q, dt, shape):
    """More rows than one co-resident grid has CTAs: the norm loops rows per CTA and leaves h and
    its scale without a grid-wide wait (`bq_rmsnorm_scale`), the cast pass writes the codes;
    bit-identical to the torch spelling, with and without the dense output, NaN included."""
    x = randn_cpu(shape, seed=shape[0], dtype=dt, scale=3.0).cuda()
    x[::5] *= 9.0
    gamma = _gamma(shape[1], 2, spread=0.3)
    ref = TS.rms_norm(x, gamma, EPS)
    calls = Q.launch_count()
    qa = Q.rms_norm_quant(x, gamma, EPS, keep_dense=True)
    assert Q.launch_count() - calls == 2        # the norm (which also leaves the scale), the cast
    assert torch.equal(qa.dense, ref)
    _same(qa, ref, f"{dt} {shape}")
    qb = Q.rms_norm_quant(x, gamma, EPS)
    assert qb.dense is None and torch.equal(u8(qb.q), u8(qa.q)) and torch.equal(qb.scale, qa.scale)
    x[shape[0] // 2, 7] = float("nan")
    qa = Q.rms_norm_quant(x, gamma, EPS, keep_dense=True)
    ref = TS.rms_norm(x, gamma, EPS)
    assert torch.isnan(qa.scale).all() and torch.equal(torch.isnan(qa.dense), torch.isnan(ref))
    assert Q.device_status() == 0


def test_rms_norm_quant_degenerate_values(Q):
    gamma = _gamma(4096, 5)
    zeros = torch.zeros(4, 4096, dtype=torch.bfloat16, device="cuda")
    qa = Q.rms_norm_quant(zeros, gamma, EPS, keep_dense=True)
    assert float(qa.dense.float().abs().max()) == 0.0 and qa.scale.item() == pytest.approx(1e-12)
    x = randn_cpu((4, 4096), seed=6).cuda()
    x[2, 100] = float("nan")
    qa = Q.rms_norm_quant(x, gamma, EPS, keep_dense=True)
    ref = TS.rms_norm(x, gamma, EPS)
    assert torch.isnan(qa.scale).all()
    assert torch.equal(torch.isnan(qa.dense), torch.isnan(ref))
    qr, sr = TS.quantize_act(ref)
    assert int((u8(qa.q) != u8(qr)).sum()) == 0
    huge = torch.full((2, 4096), 60000.0, dtype=torch.bfloat16, device="cuda")
    qa = Q.rms_norm_quant(huge, gamma, EPS, keep_dense=True)
    ref = TS.rms_norm(huge, gamma, EPS)
    assert torch.equal(qa.dense, ref)
    _same(qa, ref, "huge")


@pytest.mark.parametrize("ydt", [torch.float32, torch.bfloat16], ids=["y_fp32", "y_bf16"])
@pytest.mark.parametrize("rows,heads", [(1, 32), (8, 32), (37, 32), (128, 32), (16, 16), (5, 48), (3, 64)])
def test_gated_rms_norm_quant_is_bit_identical(Q, ydt, rows, heads):
    D = 128
    for seed in range(3):
        scale = (0.01, 1.0, 50.0)[seed]
        y = randn_cpu((rows, heads, D), seed=seed * 17 + rows, dtype=ydt, scale=scale).cuda()
        z = randn_cpu((rows, heads * D), seed=seed * 19 + rows + 1, scale=(1.0, 3.0, 8.0)[seed]).cuda()
        gamma = _gamma(D, seed, spread=(0.02, 0.3, 1.0)[seed])
        core = y.to(torch.bfloat16).reshape(-1, D)            # braid/model/gdn.py:383
        ref = TS.rms_norm_gated(core, z.reshape(-1, D), gamma, EPS).reshape(rows, heads * D)
        qa = Q.gated_rms_norm_quant(y, z, gamma, EPS, D)
        assert qa.shape == (rows, heads * D) and qa.dtype is torch.bfloat16
        _same(qa, ref, f"{ydt} rows {rows} heads {heads} seed {seed}")


def test_gated_rms_norm_quant_many_rows_and_nan(Q):
    D, heads = 128, 32
    y = randn_cpu((1024, heads, D), seed=3, dtype=torch.float32, scale=2.0).cuda()
    y[::5] *= 40.0
    z = randn_cpu((1024, heads * D), seed=4, scale=2.0).cuda()
    gamma = _gamma(D, 9)
    ref = TS.rms_norm_gated(y.to(torch.bfloat16).reshape(-1, D), z.reshape(-1, D), gamma,
                                 EPS).reshape(1024, heads * D)
    _same(Q.gated_rms_norm_quant(y, z, gamma, EPS, D), ref, "1024 rows")
    z[7, 300] = float("nan")
    ref = TS.rms_norm_gated(y.to(torch.bfloat16).reshape(-1, D), z.reshape(-1, D), gamma,
                                 EPS).reshape(1024, heads * D)
    qa = Q.gated_rms_norm_quant(y, z, gamma, EPS, D)
    assert torch.isnan(qa.scale).all()
    qr, _ = TS.quantize_act(ref)
    assert int((u8(qa.q) != u8(qr)).sum()) == 0


@pytest.mark.parametrize("ydt,rows,heads", [(torch.float32, 8192, 32), (torch.bfloat16, 3000, 32),
                                            (torch.float32, 2500, 16)],
                         ids=["f32-scan-8192x32", "bf16-3000x32", "f32-scan-2500x16"])
def test_gated_rms_norm_quant_at_prefill_sizes(Q, ydt, rows, heads):
    """More rows than one co-resident grid has CTAs: warps stride over all (row, head) pairs
    (`bq_gated_rmsnorm_scale`), then the cast pass; bit-identical to the torch spelling."""
    width = heads * 128
    y = randn_cpu((rows, heads, 128), seed=rows, dtype=ydt, scale=2.0).cuda()
    z = randn_cpu((rows, width), seed=rows + 1, scale=1.5).cuda()
    gamma = _gamma(128, 3, spread=0.3)
    ref = TS.rms_norm_gated(y.to(z.dtype).reshape(-1, 128), z.reshape(-1, 128), gamma, EPS).reshape(rows, width)
    calls = Q.launch_count()
    qa = Q.gated_rms_norm_quant(y, z, gamma, EPS, 128)
    assert Q.launch_count() - calls == 2
    _same(qa, ref, f"{ydt} {rows}x{heads}")
    assert Q.device_status() == 0


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16, torch.float32], ids=["bf16", "fp16", "fp32"])
@pytest.mark.parametrize("rows", [1, 33, 256, 257])
def test_norms_on_both_sides_of_the_wide_rows(Q, dt, rows):
    """Up to 256 rows a row has four times the threads (rms) or twice the warps (gated): widths at the
    edges of what a thread holds, heads that leave warps without one, on both sides of the line."""
    for cols in (4, 516, 1028, 2052, 4100, 8192):
        x = randn_cpu((rows, cols + 8), seed=cols, dtype=dt, scale=3.0).cuda()[:, 4:4 + cols]
        gamma = _gamma(cols, 2, spread=0.3)
        ref = TS.rms_norm(x, gamma, EPS)
        qa = Q.rms_norm_quant(x, gamma, EPS, keep_dense=True)
        assert torch.equal(u8(qa.dense), u8(ref)), f"{dt} {rows}x{cols}"
        _same(qa, ref, f"{dt} {rows}x{cols}")
    gamma = _gamma(128, 3, spread=0.3)
    for heads in (8, 9, 16, 17, 32, 33):
        y = randn_cpu((rows, heads * 128), seed=heads, dtype=torch.float32, scale=2.0).cuda()
        z = randn_cpu((rows, heads * 128), seed=heads + 1, dtype=dt, scale=2.0).cuda()
        ref = TS.rms_norm_gated(y.to(dt).reshape(-1, 128), z.reshape(-1, 128), gamma, EPS).reshape(rows, heads * 128)
        _same(Q.gated_rms_norm_quant(y, z, gamma, EPS, 128), ref, f"{dt} {rows} rows, {heads} heads")
    assert Q.device_status() == 0


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float32], ids=["bf16", "fp32"])
@pytest.mark.parametrize("heads", [1, 3, 4, 5, 33])
def test_gated_rms_norm_quant_with_heads_left_over(Q, dt, heads):
    """A warp takes four heads of a row at a time: rows whose heads do not divide by four, an infinite
    gamma (which a head that is not there must not see), rows of very different energy."""
    rows = 20000 // heads + 2400
    y = randn_cpu((rows, heads * 128), seed=heads, dtype=dt, scale=2.0).cuda()
    y[::7] *= 2.0 ** -12
    z = randn_cpu((rows, heads * 128), seed=heads + 1, dtype=dt, scale=4.0).cuda()
    gamma = _gamma(128, 3, spread=0.3)
    ref = TS.rms_norm_gated(y.reshape(-1, 128), z.reshape(-1, 128), gamma, EPS).reshape(rows, heads * 128)
    _same(Q.gated_rms_norm_quant(y, z, gamma, EPS, 128), ref, f"{dt} {heads}")
    gamma[5] = float("inf")
    ref = TS.rms_norm_gated(y.reshape(-1, 128), z.reshape(-1, 128), gamma, EPS).reshape(rows, heads * 128)
    qa = Q.gated_rms_norm_quant(y, z, gamma, EPS, 128)
    sr = TS.quantize_act(ref)[1]
    assert torch.equal(torch.isnan(qa.scale), torch.isnan(sr)) and torch.equal(qa.scale[~torch.isnan(sr)], sr[~torch.isnan(sr)])
    assert Q.device_status() == 0


def test_consumers_take_the_quantized_activation(Q):
    """`project`, `linear` and the MLP on a pre-quantized activation equal the reference order of
    operations (norm, then the consumer quantizes) bit for bit, bf16 weights in the mix included."""
    H, I = 4096, 12288
    x = randn_cpu((16, 1, H), seed=11).cuda()
    gamma = _gamma(H, 12)
    mk = lambda n, k, s: Q.quantize_weight((randn_cpu((n, k), seed=s, scale=0.02)).cuda())  # noqa: E731
    w_qkv, w_z, w_out = mk(8192, H, 13), mk(4096, H, 14), mk(H, 4096, 15)
    w_a = randn_cpu((32, H), seed=16, scale=0.02).cuda()
    h = TS.rms_norm(x, gamma, EPS)
    want = Q.project(h, w_qkv, w_z, w_a)
    got = Q.project(Q.rms_norm_quant(x, gamma, EPS, keep_dense=True), w_qkv, w_z, w_a)
    for a, b in zip(got, want):
        assert a.shape == b.shape and torch.equal(a, b)
    with pytest.raises(ValueError):
        Q.project(Q.rms_norm_quant(x, gamma, EPS), w_qkv, w_a)       # bf16 weight needs the dense form
    assert torch.equal(Q.linear(Q.rms_norm_quant(x, gamma, EPS), w_z), Q.linear(h, w_z))
    wg, wu, wd = mk(I, H, 17), mk(I, H, 18), mk(H, I, 19)
    assert torch.equal(Q.mlp_forward(Q.rms_norm_quant(x, gamma, EPS), wg, wu, wd),
                       Q.mlp_forward(h, wg, wu, wd))
    # GDN readout: gated norm feeding out_proj
    y = randn_cpu((16, 32, 128), seed=20, dtype=torch.float32).cuda()
    z = randn_cpu((16, 1, 4096), seed=21).cuda()
    g128 = _gamma(128, 22)
    core = TS.rms_norm_gated(y.to(torch.bfloat16).reshape(-1, 128), z.reshape(-1, 128), g128, EPS)
    want = Q.linear(core.reshape(16, 1, 4096), w_out)
    got = Q.linear(Q.gated_rms_norm_quant(y, z, g128, EPS, 128), w_out)
    assert got.shape == want.shape and torch.equal(got, want)


def test_norm_quant_survives_capture_and_replays_identically(Q):
    x = randn_cpu((128, 4096), seed=30).cuda()
    gamma = _gamma(4096, 31)
    y = randn_cpu((128, 32, 128), seed=32, dtype=torch.float32).cuda()
    z = randn_cpu((128, 4096), seed=33).cuda()
    g128 = _gamma(128, 34)

    def step():
        a = Q.rms_norm_quant(x, gamma, EPS, keep_dense=True)
        b = Q.gated_rms_norm_quant(y, z, g128, EPS, 128)
        return a.q, a.scale, a.dense, b.q, b.scale

    eager = [t.clone() for t in step()]
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        for _ in range(3):
            step()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        outs = step()
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    for e, r in zip(eager, outs):
        assert torch.equal(u8(e), u8(r))
    assert Q.device_status() == 0


@pytest.mark.parametrize("rows,dt", [(1, torch.bfloat16), (27, torch.float16), (128, torch.bfloat16)],
                         ids=["1", "27-fp16", "128"])
def test_norms_behind_a_running_gemm_read_its_output(Q, rows, dt):
    """Launched back to back from a graph, the norm kernels start before the kernel that writes their
    input has finished: they must see its output, not what the buffer held before."""
    hidden = 2048
    w1, w2 = (Q.quantize_weight((randn_cpu((hidden, hidden), seed=s, dtype=torch.bfloat16) * 0.05).cuda())
              for s in (1, 2))
    gamma, gamma_h = _gamma(hidden, 3), _gamma(128, 4)
    x0 = randn_cpu((rows, hidden), seed=5, dtype=dt).cuda()
    y = randn_cpu((rows, hidden), seed=6).cuda().float()

    def chain(wait=lambda t: t):
        x = x0
        for _ in range(6):
            z = wait(Q.linear(wait(Q.rms_norm_quant(x, gamma, EPS)), w1))
            x = wait(Q.linear(wait(Q.gated_rms_norm_quant(y, z, gamma_h, EPS, 128)), w2, residual=x))
        return z, x

    def one_at_a_time(t):
        torch.cuda.synchronize()
        return t

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        chain()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = chain()
    ref = chain(one_at_a_time)
    for _ in range(10):
        for t in out:
            t.zero_()
        graph.replay()
        graph.replay()
        for got, want in zip(out, ref):
            assert torch.equal(u8(got), u8(want))
    assert Q.device_status() == 0


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16], ids=["bf16", "fp16"])
def test_silu_of_the_looped_gated_norm_is_the_ieee_quotient(Q, lib, dt):
    """The looped kernel multiplies the fp32 quotient z / (1 + exp(-z)) by gamma before it rounds to 16
    bits, and takes that quotient without the division instruction up to |z| = 80.  For every such z a
    gamma is chosen whose product lands one fp32 step below a rounding boundary of the 16-bit type,
    and one that lands on it: a quotient one step too large or too small changes the output."""
    z = torch.arange(65536, dtype=torch.int32).to(torch.uint16).view(dt)
    z = z[z.float().abs() <= 80]
    s = F.silu(z.cuda().float()).cpu()                 # fp32, expf, an IEEE division
    keep = s.abs() >= 2.0 ** -120                      # gamma stays finite
    z, s = z[keep], s[keep].double()
    ulp = 2.0 ** -7 if dt is torch.bfloat16 else 2.0 ** -10
    for above in (False, True):
        wrong = torch.nextafter(s.float(), torch.zeros(()) if above else torch.full((), torch.inf).copysign(s.float()))
        gamma, want = torch.zeros(len(s)), torch.zeros(len(s))
        sharp = torch.zeros(len(s), dtype=torch.bool)
        for i in range(16):
            upper = 1.9375 - 2 * i * ulp               # even: the boundary itself rounds to it
            tie = upper - ulp / 2
            target = tie if above else tie - 2.0 ** -23
            for step in range(-3, 4):
                g = ((target / s) * (1 + step * 2.0 ** -24)).float()
                hit = (g.double() * s).float() == target           # exact products, one rounding
                hit &= ((g.double() * wrong.double()).float() >= tie) != above
                gamma = torch.where(hit & ~sharp, g, gamma)
                want = torch.where(hit & ~sharp, upper if above else upper - ulp, want)
                sharp |= hit
        assert sharp.float().mean() > 0.99             # (a few quotients have no such gamma)
        zs, gs, want = z[sharp], gamma[sharp], want[sharp]
        whole = torch.arange(-(-len(zs) // 128) * 128) % len(zs)   # the last row filled from the front
        zs, gs, want = zs[whole].cuda().reshape(-1, 128), gs[whole].cuda().reshape(-1, 128), want[whole]
        y = torch.ones(1, 128, device="cuda", dtype=dt)
        h, scale = torch.empty_like(zs), torch.empty(1, device="cuda")
        ws = torch.zeros(16, dtype=torch.uint8, device="cuda")
        stream = torch.cuda.current_stream().cuda_stream
        code = {torch.bfloat16: 1, torch.float16: 2}[dt]
        for i in range(len(zs)):
            assert lib.bq_gated_rmsnorm_scale(y.data_ptr(), code, 128, zs[i].data_ptr(), code, 128, gs[i].data_ptr(), 0.0,
                                              1, 1, 128, h[i].data_ptr(), 128, scale.data_ptr(), ws.data_ptr(), 16,
                                              stream) == 0
        assert torch.equal(h.float().cpu().flatten(), want)


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float32], ids=["bf16", "fp32"])
@pytest.mark.parametrize("cols", [128, 1000, 1024, 4096, 5120, 8192])
def test_exchange_inside_a_cluster_equals_the_grid_wide_one(Q, dt, cols):
    """Up to 64 rows the CTAs of a norm or quantizer are one cluster that exchanges the maximum in shared memory (option
    `quant_cluster`), with one to four rows per CTA: either side of every count, rows left over, the largest value in the
    first, a middle and the last row, and a NaN there.  The same bits as through the grid-wide exchange."""
    heads = max(1, cols // 128)
    gamma, g128 = _gamma(cols, 3, spread=0.3), _gamma(128, 4)
    for rows in (2, 3, 16, 17, 31, 32, 33, 47, 48, 49, 63, 64, 65):
        for peak in (0, rows // 2, rows - 1):
            for value in (300.0, float("nan")):
                x = randn_cpu((rows, cols), seed=rows, dtype=dt).cuda()
                x[peak, -1] = value
                y, z = x[:, :heads * 128 if cols >= 128 else cols].float(), torch.randn(rows, heads * 128, device="cuda").to(dt)
                got = []
                for on in (0, 1):
                    Q.set_option("quant_cluster", on)
                    try:
                        a = Q.rms_norm_quant(x, gamma, EPS, keep_dense=True)
                        b = Q.gated_rms_norm_quant(y, z, g128, EPS, 128) if cols % 128 == 0 and heads <= 64 else a
                        c = Q.quantize_act(x)
                        d = Q.sigmoid_gate_quant(x, x)
                    finally:
                        Q.set_option("quant_cluster", 1)
                    got.append([u8(a.dense), u8(a.q), u8(a.scale), u8(b.q), u8(b.scale), u8(c[0]), u8(c[1]), u8(d[0]), u8(d[1])])
                for i, (p, q) in enumerate(zip(*got)):
                    assert torch.equal(p, q), f"{rows} x {cols}, peak {peak} {value}: output {i}"
    assert Q.device_status() == 0


@pytest.mark.parametrize("call,dt,rows,cols,ctas", [
    ("norm", torch.bfloat16, 1, 4096, 0), ("norm", torch.bfloat16, 2, 4096, 2), ("norm", torch.bfloat16, 16, 8192, 16),
    ("norm", torch.bfloat16, 17, 4096, 9), ("norm", torch.bfloat16, 27, 8192, 14), ("norm", torch.bfloat16, 33, 4096, 11),
    ("norm", torch.float16, 48, 1024, 16), ("norm", torch.bfloat16, 49, 4096, 13), ("norm", torch.float16, 64, 512, 16),
    ("norm", torch.bfloat16, 65, 4096, 0), ("norm", torch.bfloat16, 33, 5120, 0), ("norm", torch.float32, 16, 8192, 16),
    ("norm", torch.float32, 17, 8192, 0), ("norm", torch.float32, 32, 4096, 16), ("norm", torch.float32, 33, 4096, 0),
    ("norm", torch.float32, 64, 2048, 16), ("gated", torch.bfloat16, 16, 4096, 16), ("gated", torch.bfloat16, 32, 4096, 16),
    ("gated", torch.float32, 17, 1024, 9), ("gated", torch.bfloat16, 33, 4096, 0), ("quantizer", torch.bfloat16, 1, 2048, 0),
    ("quantizer", torch.bfloat16, 1, 2056, 2), ("quantizer", torch.bfloat16, 32, 4096, 16), ("quantizer", torch.bfloat16, 33, 4096, 0),
    ("product", torch.float32, 27, 4096, 14), ("product", torch.bfloat16, 48, 4096, 0)])
def test_where_the_exchange_stays_inside_a_cluster(Q, call, dt, rows, cols, ctas):
    """The launch that a decode batch takes: one cluster of so many CTAs, or (0) a grid without one; by rows, width and type."""
    x, z = (torch.randn(rows, cols, device="cuda").to(dt) for _ in range(2))
    y, gamma, g128 = x.float(), _gamma(cols, 3), _gamma(128, 4)
    run = {"norm": lambda: Q.rms_norm_quant(x, gamma, EPS), "gated": lambda: Q.gated_rms_norm_quant(y, z, g128, EPS, 128),
           "quantizer": lambda: Q.quantize_act(x), "product": lambda: Q.sigmoid_gate_quant(x, z)}[call]
    run()
    torch.cuda.synchronize()
    (kernel,), _ = captured_kernels(run)
    assert kernel["cluster"] == ctas and (ctas == 0 or kernel["ctas"] == ctas), kernel
    assert Q.device_status() == 0


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float32], ids=["bf16", "fp32"])
@pytest.mark.parametrize("rows,cols", [(4000, 512), (4001, 504), (3999, 500), (3000, 2560), (2500, 4096), (2371, 4088), (1500, 5120), (1300, 8192)])
def test_rms_norm_quant_that_reads_its_rows_twice(Q, dt, rows, cols):
    """Beyond the rows that are resident at once: rows of whole and of partial vectors per thread, rows that are no whole
    16-byte pieces (through h), strided rows, more column blocks than one, with and without the dense form."""
    x = randn_cpu((rows, cols + 16), seed=rows, dtype=dt, scale=2.0).cuda()[:, :cols]
    x[::7] *= 20.0
    gamma = _gamma(cols, 9, spread=0.3)
    ref = TS.rms_norm(x, gamma, EPS)
    for keep in (False, True):
        qa = Q.rms_norm_quant(x, gamma, EPS, keep_dense=keep)
        if keep:
            assert torch.equal(u8(qa.dense), u8(ref))
        _same(qa, ref, f"{rows} x {cols}")
    x[rows - 1, cols - 1] = float("nan")
    assert Q.rms_norm_quant(x, gamma, EPS).scale.isnan().all()
    assert Q.device_status() == 0


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float32], ids=["bf16", "fp32"])
@pytest.mark.parametrize("rows,cols", [(3553, 8), (9001, 16), (30001, 24), (7105, 88), (40007, 64), (20003, 344), (6001, 1024), (6001, 1032)])
def test_narrow_rows_cast_next_to_one_another(Q, dt, rows, cols):
    """Rows of up to 128 groups of 8 lie next to one another in a CTA of the second launch, as many as put all rows on the device
    at once and at most what fits its 256 threads: counts that leave threads over, rows left over, one group per row, and the
    widest such row and the first that is not."""
    x = randn_cpu((rows, cols + 8), seed=rows, dtype=dt, scale=2.0).cuda()[:, :cols]
    x[::7] *= 20.0
    gamma = _gamma(cols, 9, spread=0.3)
    n0 = Q.launch_count()
    qa = Q.rms_norm_quant(x, gamma, EPS)
    assert Q.launch_count() - n0 == 2
    _same(qa, TS.rms_norm(x, gamma, EPS), f"{rows} x {cols}")
    assert Q.device_status() == 0


@pytest.mark.parametrize("dt,rows,cols,threads", [(torch.bfloat16, 3601, 1032, 160), (torch.float32, 1301, 2056, 160), (torch.float32, 1500, 2112, 160),
                                                  (torch.float16, 2603, 4096, 256), (torch.float32, 1201, 4104, 192), (torch.bfloat16, 1301, 5120, 224),
                                                  (torch.bfloat16, 1300, 6152, 224), (torch.float16, 1300, 8192, 256)])
def test_wide_rows_cast_by_as_many_threads_as_their_columns_need(Q, dt, rows, cols, threads):
    """One to four blocks of columns of a row, with threads for them in whole warps: the launch, and the bits, the last columns
    included."""
    x = randn_cpu((rows, cols), seed=rows, dtype=dt, scale=2.0).cuda()
    gamma = _gamma(cols, 9, spread=0.3)
    _same(Q.rms_norm_quant(x, gamma, EPS), TS.rms_norm(x, gamma, EPS), f"{rows} x {cols}")
    torch.cuda.synchronize()
    kernels, _ = captured_kernels(lambda: Q.rms_norm_quant(x, gamma, EPS))
    (cast,) = [k for k in kernels if "rmsnorm_cast_kernel" in k["name"]]
    assert cast["threads"] == threads
    assert Q.device_status() == 0


@pytest.mark.parametrize("rows,cols,vpt,whole", [(1301, 3072, 8, "Li0"), (1301, 4096, 8, "Li1"), (601, 4608, 16, None), (1777, 5120, 16, None),
                                                 (601, 8192, 16, "Li1"), (601, 8188, 16, None)])
def test_long_rows_of_fp32_take_the_kernel_of_their_width(Q, rows, cols, vpt, whole):
    """Rows of as many vectors as a thread has room for, and shorter ones: which kernel finds the scale, with and without the dense
    output, and the bits.  (None: the partial loop alone where h is not written, beside the whole one where it is.)"""
    x = randn_cpu((rows, cols), seed=rows, dtype=torch.float32, scale=2.0).cuda()
    gamma = _gamma(cols, 9, spread=0.3)
    ref = TS.rms_norm(x, gamma, EPS)
    for keep in (False, True):
        qa = Q.rms_norm_quant(x, gamma, EPS, keep_dense=keep)
        _same(qa, ref, f"{rows} x {cols}")
        assert not keep or torch.equal(u8(qa.dense), u8(ref))
        torch.cuda.synchronize()
        kernels, _ = captured_kernels(lambda: Q.rms_norm_quant(x, gamma, EPS, keep_dense=keep))
        dense = keep or cols % 8 != 0           # rows that are no whole 16-byte pieces of both types go through h
        form = whole or ("Lin1" if dense else "Li0")
        assert any(f"rmsnorm_scale_kernelIfLi{vpt}ELb{int(dense)}E{form}E" in k["name"] for k in kernels), kernels
    assert Q.device_status() == 0
