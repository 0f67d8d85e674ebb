"""The native host path (csrc/host.cpp) against the Python path of the same calls: the same bits, gradients and refusals, and
whatever it does not take goes to the Python path."""
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu

if torch.cuda.is_available():
    from triton_int8_b200 import _lib as L
    from triton_int8_b200 import kernels as K
    from triton_int8_b200.linear import Int8Config, Int8Linear, Int8LinearFn

DEV = "cuda"
CONFIGS = [dict(), dict(hadamard=128), dict(scaling="row128", round="rne"), dict(scaling="double_channel"),
           dict(scaling="double_channel", hadamard=128), dict(exact=True)]


def _layer(cfg, K_in=256, N=384, bias=True, seed=0):
    torch.manual_seed(seed)
    lin = Int8Linear(K_in, N, bias=bias, device=DEV, config=Int8Config(**cfg))
    if bias:
        with torch.no_grad():
            lin.bias.normal_()
    return lin


def _python(lin, x):
    return Int8LinearFn.apply(x, lin.weight, lin.bias, lin.config, torch.is_grad_enabled())


def _step(f, lin, x, dy):
    x = x.detach().requires_grad_(x.requires_grad)
    lin.zero_grad(set_to_none=True)
    y = f(lin, x)
    y.backward(dy)
    return [y.detach(), x.grad, *(p.grad for p in lin.parameters())]


@pytest.mark.parametrize("cfg", CONFIGS)
@pytest.mark.parametrize("bias", [True, False])
@pytest.mark.parametrize("x_grad,w_grad", [(True, True), (True, False), (False, True)])
def test_step_equals_python_path(cfg, bias, x_grad, w_grad):
    lin = _layer(cfg, bias=bias)
    lin.weight.requires_grad_(w_grad)
    x = torch.randn(2, 128, 256, device=DEV).to(torch.bfloat16).requires_grad_(x_grad)
    dy = torch.randn(2, 128, 384, device=DEV).to(torch.bfloat16)
    for d in (dy, dy[:, :1].expand_as(dy)):   # as backward may get it: dense, and with strides of its own
        native = _step(lambda m, t: K.host().linear(t, m.weight, m.bias, *m.config.native), lin, x, d)
        for got, ref in zip(native, _step(_python, lin, x, d)):
            assert (got is None and ref is None) or torch.equal(got, ref)
    with torch.no_grad():
        y = K.host().linear(x, lin.weight, lin.bias, *lin.config.native)
        assert not y.requires_grad and torch.equal(y, _python(lin, x))


def test_what_it_does_not_take_goes_to_the_python_path():
    lin = _layer({})
    h = lambda x, w=None, b=None, cfg=lin.config: K.host().linear(x, lin.weight if w is None else w, b, *cfg.native)
    x = torch.randn(128, 256, device=DEV).to(torch.bfloat16)
    assert h(x) is not None
    assert h(x.t().contiguous().t()) is None and h(x.float()) is None and h(x.cpu()) is None and h(x[:, :128]) is None
    assert h(x.as_subclass(type("T", (torch.Tensor,), {}))) is None
    assert h(x, cfg=Int8Config(scaling="double_channel", hadamard=-1)) is None
    assert h(x, b=lin.bias[:100]) is None and h(x, b=lin.bias.float()) is None
    assert torch.equal(lin(x.t().contiguous().t()), lin(x))
    with pytest.raises(TypeError):
        lin(x.float())
    with pytest.raises(ValueError):
        lin(x[:, :128].contiguous())
    with pytest.raises(L.I8LError, match="SHAPE"):
        lin(x[:100])
    with pytest.raises(RuntimeError):
        torch.func.vmap(lin)(x.view(2, 64, 256).repeat(1, 2, 1))
    with pytest.raises((RuntimeError, NotImplementedError)), torch.autograd.forward_ad.dual_level():
        lin(torch.autograd.forward_ad.make_dual(x, torch.ones_like(x)))
    with pytest.raises(RuntimeError):   # a view out of a custom function
        y = lin(x.requires_grad_(True))
        y += 1
    x = x.detach()
    a3, b2 = x[None], lin.weight.detach()
    assert K.host().quant_gemm(a3, b2, 0, 2, 0, 0, None, 1.0, 0, False) is not None
    assert K.host().quant_gemm(a3.float(), b2, 0, 2, 0, 0, None, 1.0, 0, False) is None
    assert K.host().quant_gemm(a3, b2[:, :128], 0, 2, 0, 0, None, 1.0, 0, False) is None


def test_saved_tensor_hooks_versions_and_graph_creation():
    lin = _layer({})
    x = torch.randn(128, 256, device=DEV).to(torch.bfloat16).requires_grad_(True)
    seen = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: (seen.append(t.shape), t.cpu())[1], lambda t: t.to(DEV)):
        y = lin(x)
    y.sum().backward()
    assert len(seen) == 3   # weight, int8 x^T, its scales
    g = lin.weight.grad.clone()
    lin.zero_grad()
    lin(x).sum().backward()
    assert torch.equal(lin.weight.grad, g)
    y = lin(x)
    with torch.no_grad():
        lin.weight.add_(1)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        y.sum().backward()
    y = lin(x)
    dy = torch.ones_like(y, requires_grad=True)
    dx, db = torch.autograd.grad(y, (x, lin.bias), dy, create_graph=True)
    assert not dx.requires_grad and db.requires_grad   # the bias gradient is torch's own sum


def test_a_gemm_that_gave_up_is_reported_by_the_next_forward():
    lin = _layer({})
    x = torch.randn(128, 256, device=DEV).to(torch.bfloat16)
    lin(x)
    torch.cuda.synchronize()
    lib = L.load()
    assert lib.i8l_test_set_wait_limit(256, 1) == 0
    try:
        lin(x)
        torch.cuda.synchronize()
    finally:
        assert lib.i8l_test_set_wait_limit(0, 0) == 0
    with pytest.raises(L.I8LError) as e:
        lin(x)
    assert e.value.code == L.TIMEOUT
    y = lin(x)
    K.check_status(DEV)
    assert torch.equal(y, _python(lin, x))


def _give_up(lin, x):
    lib = L.load()
    assert lib.i8l_test_set_wait_limit(256, 1) == 0
    try:
        lin(x)
        torch.cuda.synchronize()
    finally:
        assert lib.i8l_test_set_wait_limit(0, 0) == 0


def test_a_cleared_status_word_is_not_reported():
    lin = _layer({})
    x = torch.randn(128, 256, device=DEV).to(torch.bfloat16)
    y = lin(x)
    _give_up(lin, x)
    word = K.device_status(x.device)
    assert word.item() == L.TIMEOUT
    word.zero_()
    assert torch.equal(lin(x), y)
    _give_up(lin, x)
    with pytest.raises(L.I8LError):   # the next one is
        lin(x)
    K.check_status(DEV)


def test_a_timeout_waits_until_a_capture_is_over():
    lin = _layer({}).requires_grad_(False)
    x = torch.randn(128, 256, device=DEV).to(torch.bfloat16)
    ref = lin(x)
    _give_up(lin, x)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        y = lin(x)
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, ref)
    with pytest.raises(L.I8LError) as e:
        lin(x)
    assert e.value.code == L.TIMEOUT
    assert torch.equal(lin(x), ref)
    K.check_status(DEV)


def test_threads_with_streams_of_their_own():
    lin = _layer(dict(hadamard=128))
    xs = [torch.randn(256, 256, device=DEV).to(torch.bfloat16) for _ in range(4)]
    dy = torch.randn(256, 384, device=DEV).to(torch.bfloat16)
    refs = [_step(_python, lin, x.requires_grad_(True), dy) for x in xs]
    torch.cuda.synchronize()
    bad = []

    def work(i):
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            for _ in range(20):
                x = xs[i].detach().requires_grad_(True)
                y = lin(x)
                dx, = torch.autograd.grad(y, x, dy)
                s.synchronize()
                if not (torch.equal(y, refs[i][0]) and torch.equal(dx, refs[i][1])):
                    bad.append(i)

    ts = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert not bad


def test_outputs_without_gradients_are_views_as_in_the_python_path():
    """An in-place operation that would need gradients through the output is refused by both paths."""
    lin = _layer({}).requires_grad_(False)
    x = torch.randn(128, 256, device=DEV).to(torch.bfloat16)
    p = torch.ones(384, device=DEV, dtype=torch.bfloat16, requires_grad=True)
    for f in (lin, lambda t: _python(lin, t)):
        y = f(x)
        y.add_(1)
        with pytest.raises(RuntimeError):
            y.add_(p)
        with torch.no_grad():
            f(x).add_(1)


def test_traced_module_records_the_python_function():
    lin = _layer({})
    x = torch.randn(128, 256, device=DEV).to(torch.bfloat16)
    with torch.no_grad():
        graph = str(torch.jit.trace(lin, x, check_trace=False).graph)
    assert "Int8LinearFn" in graph


@pytest.mark.parametrize("path", ["native", "python"])
@pytest.mark.parametrize("off", [0, 1, 4])
def test_bias_gradient_alone_takes_any_contiguous_gradient(path, off):
    """With only the bias trainable no kernel but the sum reads the gradient: one that starts off a 16-byte boundary (a
    slice of a larger buffer) is taken.  One rounding to bf16, behind at most 256 fp32 sums."""
    lin = _layer({})
    lin.weight.requires_grad_(False)
    x = torch.randn(256, 256, device=DEV).to(torch.bfloat16)
    dy = torch.randn(off + 256 * 384, device=DEV).to(torch.bfloat16)[off:].view(256, 384)
    y = lin(x) if path == "native" else _python(lin, x)
    y.backward(dy)
    ref = dy.double().sum(0)
    bound = ref.abs() * 2.0 ** -8 + dy.double().abs().sum(0) * 2.0 ** -24 * 256
    assert ((lin.bias.grad.double() - ref).abs() <= bound).all()


@pytest.mark.parametrize("cfg,path", [({}, "native"), (dict(scaling="double_channel", hadamard=-1), "python")])
def test_bias_gradient_alone_of_a_batch_of_gradients(cfg, path):
    lin = _layer(cfg)
    lin.weight.requires_grad_(False)
    x = torch.randn(256, 256, device=DEV).to(torch.bfloat16)
    dys = torch.randn(3, 256, 384, device=DEV).to(torch.bfloat16)
    y = lin(x) if path == "native" else _python(lin, x)
    db, = torch.autograd.grad(y, lin.bias, dys, is_grads_batched=True)
    assert torch.equal(db, dys.sum(1))


FIRST_USE = """
import threading
import torch
from triton_int8_b200 import _lib as L, kernels as K
from triton_int8_b200.linear import Int8Linear
lin = Int8Linear(256, 384, device="cuda").requires_grad_(False)
x = torch.randn(128, 256, device="cuda").to(torch.bfloat16)
torch.cuda.synchronize()
start = threading.Barrier(8)
ts = [threading.Thread(target=lambda: (start.wait(), lin(x))) for _ in range(8)]
[t.start() for t in ts]
[t.join() for t in ts]
torch.cuda.synchronize()
lib = L.load()
lib.i8l_test_set_wait_limit(256, 1)
lin(x)
torch.cuda.synchronize()
lib.i8l_test_set_wait_limit(0, 0)
try:
    lin(x)
except L.I8LError as e:
    assert e.code == L.TIMEOUT
else:
    raise SystemExit("not reported")
lin(x)
K.check_status("cuda")
"""


def test_a_timeout_is_reported_once_after_a_first_use_by_several_threads():
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", FIRST_USE], cwd=root, capture_output=True, text=True, timeout=240)
    assert r.returncode == 0, r.stdout + r.stderr
