"""The kernels of one composed call overlap on the device (programmatic serialization).  Many calls in a row, each on
other inputs and all in the same recycled memory, equal the separate steps, which are launched one after the other, bit
for bit; so does a replayed graph, and so do calls whose operands the kernels right in front of them write."""
import pytest
import torch

pytestmark = pytest.mark.gpu

if torch.cuda.is_available():
    from triton_int8_b200 import linear as LN
    from triton_int8_b200.linear import Int8Config

DEV = "cuda"
SHAPES = [(128, 128, 128), (128, 2048, 384), (1920, 640, 1408), (3968, 1152, 2176)]


def _separate(x, w, dy, bias, cfg):
    """Every kernel through its own entry point."""
    from triton_int8_b200 import _lib as L
    from triton_int8_b200 import kernels as K
    if cfg.whole_k:
        xq, xs = K.quant_row(x[None], L.QMODE_ROWRCP, cfg.hadamard)
        wq, ws = K.quant_row(w, L.QMODE_ROWRCP, cfg.hadamard)
        xt = LN._dc_transposed(x, cfg)
        y = K.gemm_rowcol(xq, wq, xs, ws, bias, cfg.post_for(x.shape[1]))[0]
    else:
        xq, xs, xqt, xst = K.quant_tile(x[None], cfg.gran, cfg.qmode, cfg.hadamard, natural=True, transposed=True)
        wq, ws = K.quant_row(w, cfg.qmode, cfg.hadamard)
        xt = (xqt, xst)
        y = K.gemm_block(xq, wq, xs, ws, cfg.a_kind, L.BSCALE_CHANNEL, bias, cfg.post, cfg.flags)[0]
    dy_op, dyt_op = LN.quantize_grad_output(dy, cfg)
    return y, LN.grad_input(dy_op, w, cfg), LN.grad_weight(dyt_op, xt, cfg)


def _composed(x, w, dy, bias, cfg):
    y, saved = LN.linear_forward(x, w, bias, cfg)
    dx, dw = LN.linear_backward(dy, w, saved, cfg)
    return y, dx, dw


def _inputs(shape, n):
    M, N, K = shape
    g = torch.Generator(device=DEV).manual_seed(M + N)
    r = lambda *s: torch.randn(*s, generator=g, device=DEV).to(torch.bfloat16)
    return [(r(M, K), r(N, K), r(M, N), r(N)) for _ in range(n)]


@pytest.mark.parametrize("scaling,rnd,had", [("tile128", "half_up", 0), ("tile128", "half_up", 128), ("row128", "rne", 0),
                                             ("row128", "rne", 128), ("double_channel", "half_up", 0),
                                             ("double_channel", "half_up", 128)])
@pytest.mark.parametrize("shape", SHAPES)
def test_calls_in_a_row_equal_separate_steps(shape, scaling, rnd, had):
    cfg = Int8Config(scaling=scaling, round=rnd, hadamard=had)
    ins = _inputs(shape, 4)
    refs = []
    for i in ins:
        refs.append([t.clone() for t in _separate(*i, cfg)])
        torch.cuda.synchronize()
    outs = [_composed(*ins[k % 4], cfg) for k in range(12)]   # nothing waits in between
    torch.cuda.synchronize()
    for k, out in enumerate(outs):
        for name, got, ref in zip(("y", "dx", "dw"), out, refs[k % 4]):
            assert torch.equal(got, ref), f"call {k}: {name}"


@pytest.mark.parametrize("scaling,rnd,had", [("tile128", "half_up", 0), ("tile128", "half_up", 128), ("row128", "rne", 0),
                                             ("double_channel", "half_up", 0)])
@pytest.mark.parametrize("shape", [(256, 4352, 256), (4224, 4352, 256), (1920, 640, 1408)])   # N, then M too, above 4096: maxima in memory
def test_training_steps_in_a_row_equal_separate_steps(shape, scaling, rnd, had):
    """With the bias gradient in the chain (from 1024 rows on several CTAs share its columns) and column maxima that are
    cleared in it."""
    from triton_int8_b200 import kernels as K
    from triton_int8_b200.linear import Int8Linear
    cfg = Int8Config(scaling=scaling, round=rnd, hadamard=had)
    M, N, Kd = shape
    ins = _inputs(shape, 3)
    lin = Int8Linear(Kd, N, device=DEV, config=cfg)
    refs = []
    for x, w, dy, bias in ins:
        refs.append([t.clone() for t in (*_separate(x, w, dy, bias, cfg), K.col_sum(dy))])
        torch.cuda.synchronize()

    def step(x, w, dy, bias):
        with torch.no_grad():
            lin.weight.copy_(w)
            lin.bias.copy_(bias)
        x = x.detach().requires_grad_(True)
        y = lin(x)
        return [y.detach(), *torch.autograd.grad(y, (x, lin.weight, lin.bias), dy)]

    outs = [step(*ins[k % 3]) for k in range(12)]   # nothing waits in between
    torch.cuda.synchronize()
    for k, out in enumerate(outs):
        for name, got, ref in zip(("y", "dx", "dw", "db"), out, refs[k % 3]):
            assert torch.equal(got, ref), f"call {k}: {name}"


def test_chain_in_a_graph_equals_separate_steps():
    cfg = Int8Config(hadamard=128)
    ins = _inputs((1920, 640, 1408), 3)
    static = [t.clone() for t in ins[0]]
    _composed(*static, cfg)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        out = _composed(*static, cfg)
    for i in ins:
        ref = _separate(*i, cfg)
        for s, t in zip(static, i):
            s.copy_(t)
        g.replay()
        torch.cuda.synchronize()
        for got, want in zip(out, ref):
            assert torch.equal(got, want)


@pytest.mark.parametrize("cfg", [dict(), dict(hadamard=128), dict(scaling="row128", round="rne"), dict(scaling="double_channel"),
                                 dict(scaling="double_channel", hadamard=-1)], ids=str)
@pytest.mark.parametrize("M", [128, 4096])
def test_operands_written_by_the_kernel_in_front(cfg, M):
    """An elementwise kernel writes the input, the weight or the output gradient right before the call, in place over the
    previous call's values, and one layer's output is the next one's input: the results are those of synchronised calls."""
    from triton_int8_b200.linear import Int8Linear
    torch.manual_seed(M)
    r = lambda *s: torch.randn(*s, device=DEV).to(torch.bfloat16)
    lins = [Int8Linear(a, b, device=DEV, config=Int8Config(**cfg)) for a, b in ((1024, 512), (512, 2048))]
    xs, dys, ws = [r(M, 1024) for _ in range(3)], [r(M, 2048) for _ in range(3)], [r(2048, 512) * 0.02 for _ in range(3)]
    x, dy = torch.zeros_like(xs[0]).requires_grad_(True), torch.zeros_like(dys[0])

    def step(k, sync):
        wait = torch.cuda.synchronize if sync else lambda: None
        with torch.no_grad():
            torch.mul(ws[k], 1, out=lins[1].weight)
            torch.mul(xs[k], 1, out=x)
        wait()
        h = lins[0](x)
        wait()
        y = lins[1](h)
        wait()
        torch.mul(dys[k], 1, out=dy)
        wait()
        grads = torch.autograd.grad(y, [x, *lins[0].parameters(), *lins[1].parameters()], dy)
        wait()
        return [y.detach(), *grads]

    refs = [step(k, True) for k in range(3)]
    outs = []
    for k in range(24):
        outs.append(step(k % 3, False))
        if len(outs) == 6:
            torch.cuda.synchronize()
            for j, out in enumerate(outs):
                assert all(torch.equal(got, ref) for got, ref in zip(out, refs[(k - 5 + j) % 3])), f"call {k - 5 + j}"
            outs = []


def test_a_cta_limit_keeps_sms_free_inside_a_call():
    """Under a limit the backward call's second GEMM does not sit on the free SMs while the first one runs: short kernels on
    another stream, one after the other, are done long before the first GEMM, half of the call's time."""
    from triton_int8_b200 import kernels as K
    x, w, dy, _ = _inputs((16384, 8192, 16384), 1)[0]
    saved = LN.linear_forward(x, w, None)[1]
    side = torch.cuda.Stream()
    ev = lambda: torch.cuda.Event(enable_timing=True)
    share = []
    for _ in range(3):
        start, others, end = ev(), ev(), ev()
        torch.cuda.synchronize()
        start.record()
        side.wait_event(start)
        with K.cta_limit(140):
            LN.linear_backward(dy, w, saved)
        end.record()
        with torch.cuda.stream(side):
            for _ in range(20):
                torch.cuda._sleep(50_000)   # 25 to 40 us each
            others.record()
        torch.cuda.synchronize()
        share.append(start.elapsed_time(others) / start.elapsed_time(end))
    K.check_status(DEV)
    assert min(share) < 0.4, share
