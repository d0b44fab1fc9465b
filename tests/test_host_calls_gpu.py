"""The native calls (`csrc/host_calls.cpp`) against the Python code they stand in for: same bits, same
shapes, no more launches, and whatever they do not take is decided by that code."""
from __future__ import annotations

import pytest
import torch
import torch.autograd.forward_ad as fwad
import torch.nn.functional as F

from _util import randn_cpu, u8

pytestmark = pytest.mark.gpu


def _flat(out):
    if isinstance(out, torch.Tensor):
        return [out]
    if out is None:
        return []
    if isinstance(out, (list, tuple)):
        return [t for o in out for t in _flat(o)]
    return _flat([out.q, out.scale, out.dense])          # QuantizedActivation


def _both(Q, monkeypatch, fn):
    """`fn()` through the native calls and through the Python code alone, with the launches of each."""
    assert Q._NATIVE is not None, "the native calls are not built for this torch"
    n0 = Q.launch_count()
    native = _flat(fn())
    n1 = Q.launch_count()
    with monkeypatch.context() as m:
        m.setattr(Q, "_NATIVE", None)
        python = _flat(fn())
    assert n1 - n0 <= Q.launch_count() - n1        # few rows: `linear` is one launch there
    assert len(native) == len(python)
    for a, b in zip(native, python):
        assert a.shape == b.shape and a.dtype is b.dtype and a.stride() == b.stride()
        assert torch.equal(u8(a), u8(b))
    return native


@pytest.fixture(scope="module")
def weights(request):
    from braid_b200 import quant as Q
    Q.warm_fused(True)
    mk = lambda n, k, s: Q.quantize_weight(randn_cpu((n, k), seed=s, scale=0.02).cuda())  # noqa: E731
    H = 512
    return {"a": mk(H, H, 1), "b": mk(1024, H, 2), "gate": mk(1536, H, 3), "up": mk(1536, H, 4), "down": mk(H, 1536, 5),
            "odd_gate": mk(1040, H, 6), "odd_up": mk(1040, H, 7), "odd_down": mk(H, 1040, 8)}


@pytest.mark.parametrize("dt", [torch.bfloat16, torch.float16, torch.float32], ids=["bf16", "fp16", "fp32"])
@pytest.mark.parametrize("M", [1, 17, 256, 257, 2500])
def test_native_calls_give_the_bits_of_the_python_code(Q, monkeypatch, weights, dt, M):
    H, w = 512, weights
    x = randn_cpu((M, H), seed=M, dtype=dt).cuda()
    x3 = x.view(M, 1, H)
    res = randn_cpu((M, H), seed=1, dtype=dt).cuda()
    strided = randn_cpu((M, 2 * H), seed=2, dtype=dt).cuda()[:, H:]
    gates = [randn_cpu((16, H), seed=s, dtype=dt, scale=0.02).cuda() for s in (3, 4)]
    gamma = 1 + 0.1 * randn_cpu((H,), seed=5, dtype=torch.float32).cuda()
    gamma_h = 1 + 0.1 * randn_cpu((128,), seed=6, dtype=torch.float32).cuda()
    scan = randn_cpu((M, H), seed=7, dtype=torch.float32).cuda()
    both = lambda fn: _both(Q, monkeypatch, fn)  # noqa: E731
    both(lambda: Q.quantize_act(x3))
    both(lambda: Q.quantize_act(strided))                               # the torch spelling, either way
    both(lambda: Q.linear(x, w["a"]))
    both(lambda: Q.linear(x3, w["a"], residual=res.view(M, 1, H)))
    both(lambda: Q.linear(x, w["a"], residual=strided))
    both(lambda: Q.linear(strided, w["a"]))
    both(lambda: Q.project(x, w["a"], w["b"]))
    both(lambda: Q.project(x3, w["a"], *gates, w["b"]))
    h = Q.rms_norm_quant(x, gamma, 1e-6, keep_dense=True)
    both(lambda: Q.rms_norm_quant(x3, gamma, 1e-6, keep_dense=True))
    both(lambda: Q.rms_norm_quant(strided, gamma, 1e-6))
    both(lambda: Q.project(h, w["a"], *gates))
    both(lambda: Q.gated_rms_norm_quant(scan.view(M, H // 128, 128), x, gamma_h, 1e-6, 128))
    both(lambda: Q.gated_rms_norm_quant(x, strided, gamma_h, 1e-6, 128))
    qg = randn_cpu((M, 2 * H), seed=8, dtype=dt).cuda().view(M, 2, H)
    both(lambda: Q.sigmoid_gate_quant(x, qg[..., H // 2:]))
    both(lambda: Q.sigmoid_gate_quant(x, res))
    both(lambda: Q.gated_output_projection(x, qg[..., H // 2:], w["a"]))
    both(lambda: Q.mlp_forward(x3, w["gate"], w["up"], w["down"], residual=res.view(M, 1, H)))
    both(lambda: Q.mlp_forward(h, w["gate"], w["up"], w["down"], residual=strided))
    both(lambda: Q.mlp_forward(x, w["odd_gate"], w["odd_up"], w["odd_down"]))
    both(lambda: Q.lm_head_argmax(h, w["b"], return_logits=True))
    both(lambda: [Q.lm_head_argmax(x3, w["b"])])
    assert Q.device_status() == 0


def test_what_the_python_code_refuses_stays_refused(Q, weights):
    w = weights
    x = randn_cpu((8, 512), seed=1).cuda()
    for bad in (lambda: Q.linear(x.cpu(), w["a"]), lambda: Q.quantize_act(x.cpu())):
        with pytest.raises(RuntimeError):
            bad()
    for bad in (lambda: Q.linear(x.double(), w["a"]), lambda: Q.quantize_act(x[:0]),
                lambda: Q.linear(x, w["a"], residual=x.float()), lambda: Q.linear(x, w["a"], residual=x[:4]),
                lambda: Q.rms_norm_quant(x, torch.ones(4, device="cuda"), 1e-6),
                lambda: Q.rms_norm_quant(x, torch.ones(512, device="cuda").half(), 1e-6),
                lambda: Q.project(x[:, :256].contiguous(), w["a"], w["b"])):
        with pytest.raises(ValueError):
            bad()


class _Tagged(torch.Tensor):
    """A subclass without a dispatch of its own: only its Python type tells it from a tensor."""


def test_what_torch_follows_above_256_rows_stays_a_torch_operation(Q, weights):
    """The residual add and the 16-bit gates of a prompt are torch operations where torch follows them:
    forward-mode tangents are carried, subclasses keep their type, a tracer sees the addition."""
    M, H, w = 300, 512, weights
    x, res, t = (randn_cpu((M, H), seed=s).cuda() for s in (1, 2, 3))
    gate, tg = (randn_cpu((16, H), seed=s, scale=0.02).cuda() for s in (4, 5))
    xq, sx = Q.quantize_act(x)
    adds = {"matmul": lambda r: Q.fp8_matmul(xq, sx, w["a"], residual=r), "linear": lambda r: Q.linear(x, w["a"], residual=r),
            "mlp": lambda r: Q.mlp_forward(x, w["gate"], w["up"], w["down"], residual=r)}
    for name, add in adds.items():
        with fwad.dual_level():
            out = fwad.unpack_dual(add(fwad.make_dual(res, t)))
            assert out.tangent is not None and torch.equal(out.tangent, t), name
            assert torch.equal(out.primal, add(res)), name
        assert type(add(res.as_subclass(_Tagged))) is _Tagged, name
        traced = torch.jit.trace(add, (res,), check_trace=False)
        assert torch.equal(traced(t), add(t)), name
    with fwad.dual_level():
        for got, want in ((Q.project(fwad.make_dual(x, t), w["a"], gate)[1], F.linear(t, gate)),
                          (Q.project(x, w["a"], fwad.make_dual(gate, tg))[1], F.linear(x, tg))):
            tangent = fwad.unpack_dual(got).tangent
            assert tangent is not None and torch.equal(tangent, want)
    assert type(Q.project(x.as_subclass(_Tagged), w["a"], gate)[1]) is _Tagged
    assert type(Q.project(x, w["a"], gate.as_subclass(_Tagged))[1]) is _Tagged
    assert Q.device_status() == 0


def test_mlp_of_two_launches_holds_a_slot_of_its_own(Q):
    """Between its launches the maximum of h lies in its scratch: not in one that a call of another thread may be handed
    meanwhile.  The common slots are not touched, the one it held is zero again, and threads that share a stream get
    the bits of a lone call.  A captured call keeps a common slot, which no call outside a graph holds."""
    import threading
    mk = lambda n, k, s: Q.quantize_weight(randn_cpu((n, k), seed=s, scale=0.02).cuda())  # noqa: E731
    wg, wu, wd = mk(8192, 4096, 1), mk(8192, 4096, 2), mk(4096, 8192, 3)
    xs = [randn_cpu((2, 4096), seed=i).cuda() * (1 + 3 * i) for i in range(4)]
    hs = [Q.QuantizedActivation(*Q.quantize_act(x), x.shape, x.dtype) for x in xs]
    want = [Q.mlp_forward(h, wg, wu, wd) for h in hs]
    n0, taken = Q.launch_count(), Q._next_slot[0]
    Q.mlp_forward(hs[0], wg, wu, wd)
    assert Q.last_gemm_launch()["quantizes"] and Q.launch_count() - n0 == 2 and Q._next_slot[0] == taken
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        again = Q.mlp_forward(hs[1], wg, wu, wd)
    assert Q._next_slot[0] == (taken + 1) % 256
    graph.replay()
    assert torch.equal(again, want[1])
    wrong = []

    def work(i):
        for _ in range(60):
            got = [Q.mlp_forward(hs[i], wg, wu, wd) for _ in range(3)]
            for _ in range(6):
                Q.linear(xs[i], wg)
            wrong.extend(1 for y in got if not torch.equal(y, want[i]))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
    torch.cuda.synchronize()
    assert not Q._scratch[0].view(torch.int32).any() and Q.device_status() == 0


def test_native_calls_from_threads_and_streams(Q, weights):
    """Slots are counted in one place whichever way a call takes; threads on their own streams get the
    bits of a lone call.  Small projections alone: their launches do not wait for one another's CTAs.  Launches
    that do (norms, larger quantizers, gate/up) are for one stream per device, and at most 256 launches may be in
    flight before a slot is taken again."""
    import threading
    w, x = weights, randn_cpu((4, 512), seed=1).cuda()
    want = Q.mlp_forward(x, w["gate"], w["up"], w["down"])
    torch.cuda.synchronize()
    wrong = []

    def work():
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(200):
                got = Q.linear(x, w["a"])
            out = [Q.fp8_matmul(*Q.quantize_act(x), w["a"]) for _ in range(20)]
            torch.cuda.current_stream().synchronize()
            wrong.extend(i for i, o in enumerate(out) if not torch.equal(o, got))

    threads = [threading.Thread(target=work) for _ in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
    assert torch.equal(want, Q.mlp_forward(x, w["gate"], w["up"], w["down"]))
    assert Q.device_status() == 0


@pytest.mark.parametrize("M,K,I", [(1, 256, 512), (16, 256, 512), (300, 256, 512), (16, 256, 28160), (16, 256, 576)])
def test_mlp_quantizes_its_input_once(Q, M, K, I):
    """A plain activation is quantized inside the native MLP call; where that call is refused behind the quantizer (28160 columns:
    more CTAs than are resident at once) the codes are used, not made again.  Same bits and one launch more than from codes."""
    g = torch.Generator(device="cuda").manual_seed(I + M)
    gate, up, down = (Q.quantize_weight((torch.randn(n, k, generator=g, device="cuda") * 0.05).bfloat16())
                      for n, k in ((I, K), (I, K), (K, I)))
    x, res = (torch.randn(M, K, generator=g, device="cuda").bfloat16() for _ in range(2))
    n0 = Q.launch_count()
    y = Q.mlp_forward(x, gate, up, down, residual=res)
    n1 = Q.launch_count()
    qa = Q.QuantizedActivation(*Q.quantize_act(x), x.shape, x.dtype)
    n2 = Q.launch_count()
    want = Q.mlp_forward(qa, gate, up, down, residual=res)
    assert torch.equal(y, want) and n1 - n0 == Q.launch_count() - n2 + 1
    assert torch.equal(Q.mlp_forward(x.view(1, M, K), gate, up, down, residual=res.view(1, M, K)), want.view(1, M, K))
    assert Q.device_status() == 0


def test_native_weight_quantizer_gives_the_same_weight(Q):
    """`quantize_weight` as a native call and from Python: same codes and scale; what torch would follow, strided weights
    and odd types go the other ways they went."""
    for dt in (torch.bfloat16, torch.float16, torch.float32):
        w = torch.randn(272, 1040, device="cuda").to(dt)
        a, b = Q.quantize_weight(w), Q._quantize_weight_fused(w)
        assert torch.equal(a.data.view(torch.uint8), b[0].view(torch.uint8)) and torch.equal(a.scale, b[1])
        assert a.shape == (272, 1040) and a.data.shape == (272, 1040) and a.scale.shape == (1, 1)
        p = torch.nn.Parameter(w)
        with torch.no_grad():
            assert torch.equal(Q.quantize_weight(p).scale, a.scale)
        t = w.t().contiguous().t()
        assert torch.equal(Q.quantize_weight(t).data.view(torch.uint8), a.data.view(torch.uint8))
    with pytest.raises(ValueError):
        Q.quantize_weight(torch.randn(8, 16, device="cuda"))


@pytest.mark.parametrize("H,I", [(1792, 5376), (2048, 6144), (3072, 9216), (3648, 9216)])
def test_mlp_that_asks_the_down_weight_into_l2_gives_the_same_bits(Q, monkeypatch, H, I):
    """The native MLP names the down weight to its gate/up launch, which asks 8 MB of it into L2 from 12 MB on, by the last warp and
    from 32 MB on by the first; the Python code names nothing."""
    g = torch.Generator(device="cuda").manual_seed(H)
    gate, up, down = (Q.quantize_weight((torch.randn(n, k, generator=g, device="cuda") * 0.02).bfloat16())
                      for n, k in ((I, H), (I, H), (H, I)))
    for M in (1, 16, 48):
        x = randn_cpu((M, H), seed=M).cuda()
        _both(Q, monkeypatch, lambda: Q.mlp_forward(x, gate, up, down, residual=x))
    assert Q.device_status() == 0
