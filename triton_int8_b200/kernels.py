"""Tensor-level wrappers of the C ABI: allocate outputs with torch, pass raw pointers and the
current CUDA stream.  These are the building blocks of the fwd_32 / bwd_33 variants."""
from __future__ import annotations

import threading

import torch

from . import _lib as L


_current_device = torch._C._cuda_getDevice
_raw_stream = torch._C._cuda_getCurrentRawStream


def _ptr(t):
    return None if t is None else t.data_ptr()


def _call(name: str, dev: torch.device, *args, tensors=()) -> None:
    """Launch on `dev`: the C side takes the device, its SM count and the stream from the current CUDA
    context, so the tensors' device is made current for the call (the trailing stream argument is that
    device's current stream), and every operand must live on it."""
    for t in tensors:
        if t is not None and t.device != dev:
            raise ValueError(f"{name}: operands on different devices ({t.device} vs {dev})")
    index = dev.index
    if index == _current_device():   # the usual case, without the context manager (4 us of host time)
        L.call(name, *args, _raw_stream(index))
    else:
        with torch.cuda.device(dev):
            L.call(name, *args, _raw_stream(index))


# ---------------------------------------------------------------------------------------- status word
# The GEMM kernels bound every device-side wait; a wait that gives up makes the kernel return early and
# write I8L_ERR_TIMEOUT into a device int32.  One such word per device is passed to every GEMM launched
# from here.  check_status() reads it (synchronously); poll_status() is the cheap form for a training
# loop: it looks at a copy started by the previous poll and starts the next one, never blocking.
_STATUS: dict = {}
_STATUS_LOCK = threading.Lock()   # one word per device, also when several threads come first


class _StatusWord:
    def __init__(self, dev):
        self.dev = dev
        self.word = torch.zeros(1, dtype=torch.int32, device=dev)
        self.host = torch.zeros(1, dtype=torch.int32).pin_memory()
        if not torch.cuda.is_current_stream_capturing():
            torch.cuda.current_stream(dev).synchronize()   # polls copy the word on a stream of their own
        with torch.cuda.device(dev):
            self.poller = L.load().i8l_status_open(self.word.data_ptr(), self.host.data_ptr())
            if not self.poller:
                raise L.I8LError(-4, "i8l_status_open failed")
            self.mirror = torch.zeros(1, dtype=torch.int32).pin_memory()
            L.call("i8l_status_mirror", self.poller, self.mirror.data_ptr())


def _status_of(dev: torch.device) -> "_StatusWord":
    key = dev.index if dev.index is not None else torch.cuda.current_device()
    st = _STATUS.get(key)
    if st is None:
        with _STATUS_LOCK:
            st = _STATUS.get(key)
            if st is None:
                st = _STATUS[key] = _StatusWord(torch.device("cuda", key))
    return st


def device_status(dev) -> torch.Tensor:
    """The int32 status word that GEMMs on `dev` report into (0 = no wait has ever given up)."""
    return _status_of(dev if isinstance(dev, torch.device) else torch.device(dev)).word


def _raise_if_set(st: "_StatusWord", code: int) -> None:
    if code:
        st.word.zero_()
        # a copy started from now on, on whatever stream, must see the cleared word, and one started before is void
        torch.cuda.current_stream(st.dev).synchronize()
        L.call("i8l_status_reset", st.poller)
        raise L.I8LError(code, f"a GEMM on {st.dev} gave up a bounded device-side wait; its output is incomplete")


def check_status(dev=None) -> None:
    """Synchronous check: raises I8LError (code TIMEOUT) if a GEMM on `dev` gave up a wait since the
    last check, and clears the word."""
    st = _status_of(torch.device(dev if dev is not None else "cuda"))   # without an index: the current device
    _raise_if_set(st, int(st.word.item()))


def poll_status(dev) -> None:
    """Non-blocking check for hot loops: raises if the copy started by an earlier poll has completed and
    shows a timeout; then starts the next copy.  Does nothing while the stream is being captured."""
    st = _status_of(dev if isinstance(dev, torch.device) else torch.device(dev))
    index = st.dev.index
    if index == _current_device():
        rc = L.load().i8l_status_poll(st.poller, _raw_stream(index))
    else:
        with torch.cuda.device(st.dev):
            rc = L.load().i8l_status_poll(st.poller, _raw_stream(index))
    if rc:
        if rc == L.TIMEOUT:
            _raise_if_set(st, rc)
        raise L.I8LError(rc, L.load().i8l_last_error().decode())


# ---------------------------------------------------------------------------------------- native host path
# _host.so (csrc/host.cpp) runs the composed calls on plain tensors without the interpreter in between and returns None for
# anything else, which the Python code below then takes.
_host = None


def _on_error(name: str, code: int, index: int) -> None:
    raise L.I8LError(code, L.load().i8l_last_error().decode())


def _on_timeout(index: int) -> None:
    """The mirror of a status word is set.  Nothing happens while the stream is being captured, as in poll_status: a later call
    reports it.  A word that its owner has cleared since is not reported."""
    st = _status_of(torch.device("cuda", index))
    with torch.cuda.device(st.dev):
        if torch.cuda.is_current_stream_capturing():
            return
    code = int(st.word.item())
    _raise_if_set(st, code)
    L.call("i8l_status_reset", st.poller)


def _open_status(index: int):
    st = _status_of(torch.device("cuda", index))
    return st.word.data_ptr(), st.poller


def _backward_in_python(dy, w, xqt, xst, gran, qmode, hadamard, flags, whole_k, need_dx, need_dw):
    post = [1.0 / hadamard if hadamard else 1.0] * 2
    return linear_backward(dy, w, (xqt, xst), L.GRAN_ROW if whole_k else gran, L.QMODE_ROWRCP if whole_k else qmode, hadamard,
                           *post, 0 if whole_k else flags, bool(need_dx), bool(need_dw))


def host():
    """The native module, bound to the loaded library."""
    global _host
    if _host is None:
        L.load()
        try:
            from . import _host as mod
            from .build import host_abi
            if mod.abi != host_abi():
                raise ImportError(f"built for {mod.abi}, this is {host_abi()}")
        except ImportError as e:
            raise ImportError(f"triton_int8_b200/_host.so is missing or does not fit this torch: build it with "
                              f"`python -m triton_int8_b200.build` ({e})") from e
        mod.setup(L.address("i8l_quant_gemm"), L.address("i8l_linear_backward_bias"), L.address("i8l_status_peek"), _on_error,
                  _on_timeout, _open_status, _backward_in_python)
        _host = mod
    return _host


def _check_bf16(x: torch.Tensor, name: str) -> torch.Tensor:
    if not x.is_cuda:
        raise ValueError(f"{name} must be a CUDA tensor (no CPU path exists)")
    if x.dtype != torch.bfloat16:
        raise TypeError(f"{name} must be bfloat16, got {x.dtype}")
    return x.contiguous()


def _check_bias(bias, N: int):
    """The kernels read N consecutive bf16 values."""
    if bias is None:
        return None
    if bias.dtype != torch.bfloat16:
        raise TypeError(f"bias must be bfloat16, got {bias.dtype}")
    if bias.numel() < N:
        raise ValueError(f"bias has {bias.numel()} elements, {N} are needed")
    return bias.contiguous()


def _check_saved(xqt, xst, M: int, K: int, gran: int):
    """The operand that linear_backward takes over from quant_gemm: its scales must be those of the same grouping."""
    shape = {L.GRAN_TILE128: (1, K // 128, M // 128), L.GRAN_GROUP128: (1, K, M // 128)}.get(gran, (1, K))
    if xqt.dtype != torch.int8 or tuple(xqt.shape) != (1, K, M):
        raise ValueError(f"saved operand {xqt.dtype} {tuple(xqt.shape)}, expected int8 {(1, K, M)}")
    if xst.dtype != torch.float32 or tuple(xst.shape) != shape:
        raise ValueError(f"saved scales {xst.dtype} {tuple(xst.shape)}, expected float32 {shape} for this grouping")
    return xqt.contiguous(), xst.contiguous()


def quant_tile(x: torch.Tensor, gran: int = L.GRAN_TILE128, qmode: int = L.QMODE_TRITON, hadamard: int = 0,
               natural: bool = True, transposed: bool = False):
    """x bf16 [B, R, C] -> (q, scale, qt, scale_t); entries not requested are None."""
    x = _check_bf16(x, "x")
    B, R, C = x.shape
    q = s = qt = st = None
    if natural:
        q = torch.empty((B, R, C), dtype=torch.int8, device=x.device)
        s_shape = {L.GRAN_TILE128: (B, R // 128, C // 128), L.GRAN_TILE128X256: (B, R // 128, C // 256)}.get(gran, (B, R, C // 128))
        s = torch.empty(s_shape, dtype=torch.float32, device=x.device)
    if transposed:
        qt = torch.empty((B, C, R), dtype=torch.int8, device=x.device)
        st = torch.empty((B, C // 128, R // 128) if gran == L.GRAN_TILE128 else (B, C, R // 128),
                         dtype=torch.float32, device=x.device)
    _call("i8l_quant_tile", x.device, x.data_ptr(), B, R, C, gran, qmode, hadamard, _ptr(q), _ptr(s), _ptr(qt), _ptr(st))
    return q, s, qt, st


def quant_row(x: torch.Tensor, qmode: int = L.QMODE_TRITON, hadamard: int = 0):
    """x bf16 [..., C] -> int8 [..., C], fp32 scale [...]."""
    x = _check_bf16(x, "x")
    C = x.shape[-1]
    rows = x.numel() // C
    q = torch.empty(x.shape, dtype=torch.int8, device=x.device)
    s = torch.empty(x.shape[:-1], dtype=torch.float32, device=x.device)
    _call("i8l_quant_row", x.device, x.data_ptr(), rows, C, qmode, hadamard, q.data_ptr(), s.data_ptr())
    return q, s


def quant_col_t(x: torch.Tensor, qmode: int = L.QMODE_TRITON, hadamard: int = 0):
    """x bf16 [R, C] -> int8 x^T [C, R] with one scale per column of x, fp32 [C]; hadamard=128 rotates
    x^T in 128-wide groups along its contraction axis (the rows of x) first."""
    x = _check_bf16(x, "x")
    R, C = x.shape
    qt = torch.empty((C, R), dtype=torch.int8, device=x.device)
    st = torch.empty((C,), dtype=torch.float32, device=x.device)
    scratch = torch.empty((C,), dtype=torch.float32, device=x.device)
    if hadamard not in (0, 128):
        raise ValueError("quant_col_t: hadamard must be 0 or 128")
    _call("i8l_quant_col_t_rot" if hadamard else "i8l_quant_col_t", x.device, x.data_ptr(), R, C, qmode, qt.data_ptr(),
          st.data_ptr(), scratch.data_ptr())
    return qt, st


def _gemm_dims(aq: torch.Tensor, bq: torch.Tensor):
    if aq.dtype != torch.int8 or bq.dtype != torch.int8:
        raise TypeError("quantized operands must be int8")
    B, M, K = aq.shape
    b_batched = bq.dim() == 3
    N = bq.shape[-2]
    if bq.shape[-1] != K or (b_batched and bq.shape[0] != B):
        raise ValueError(f"operand shapes do not match: {tuple(aq.shape)} x {tuple(bq.shape)}")
    return B, M, N, K, b_batched


def gemm_block(aq, bq, a_s, b_s, a_kind=L.ASCALE_TILE, b_kind=L.BSCALE_CHANNEL, bias=None, post_scale=1.0,
               flags=0, status=None):
    """Block-scaled GEMM; returns bf16 (fp32 with GEMM_OUT_F32) [B, M, N]."""
    aq, bq = aq.contiguous(), bq.contiguous()
    B, M, N, K, bb = _gemm_dims(aq, bq)
    bias = _check_bias(bias, N)
    out = torch.empty((B, M, N), dtype=torch.float32 if flags & L.GEMM_OUT_F32 else torch.bfloat16, device=aq.device)
    a_s, b_s = a_s.contiguous(), b_s.contiguous()
    status = device_status(aq.device) if status is None else status
    _call("i8l_gemm_block", aq.device, aq.data_ptr(), bq.data_ptr(), a_s.data_ptr(), b_s.data_ptr(),
          a_kind, b_kind, int(bb), _ptr(bias), float(post_scale), out.data_ptr(), B, M, N, K, flags, _ptr(status),
          tensors=(bq, a_s, b_s, bias, status))
    return out


def gemm_rowcol(aq, bq, a_s, b_s, bias=None, post_scale=1.0, flags=0, status=None):
    aq, bq = aq.contiguous(), bq.contiguous()
    B, M, N, K, bb = _gemm_dims(aq, bq)
    bias = _check_bias(bias, N)
    out = torch.empty((B, M, N), dtype=torch.float32 if flags & L.GEMM_OUT_F32 else torch.bfloat16, device=aq.device)
    a_s, b_s = a_s.contiguous(), b_s.contiguous()
    status = device_status(aq.device) if status is None else status
    _call("i8l_gemm_rowcol", aq.device, aq.data_ptr(), bq.data_ptr(), a_s.data_ptr(), b_s.data_ptr(),
          int(bb), _ptr(bias), float(post_scale), out.data_ptr(), B, M, N, K, flags, _ptr(status),
          tensors=(bq, a_s, b_s, bias, status))
    return out


def fused_gemm(a_bf, b_bf, flags=0, status=None):
    """bf16 a [B, M, K] x bf16 b [N, K] or [B, N, K] -> bf16 (fp32 with GEMM_OUT_F32) [B, M, N] in ONE kernel:
    operand tiles are quantized on the fly per 128-wide K step inside the GEMM (nothing int8 reaches memory)."""
    a_bf, b_bf = _check_bf16(a_bf, "a"), _check_bf16(b_bf, "b")
    B, M, K = a_bf.shape
    bb = b_bf.dim() == 3
    N = b_bf.shape[-2]
    if b_bf.shape[-1] != K or (bb and b_bf.shape[0] != B):
        raise ValueError(f"operand shapes do not match: {tuple(a_bf.shape)} x {tuple(b_bf.shape)}")
    out = torch.empty((B, M, N), dtype=torch.float32 if flags & L.GEMM_OUT_F32 else torch.bfloat16, device=a_bf.device)
    status = device_status(a_bf.device) if status is None else status
    _call("i8l_fused_gemm", a_bf.device, a_bf.data_ptr(), b_bf.data_ptr(), out.data_ptr(), B, M, N, K, int(bb), flags,
          _ptr(status), tensors=(b_bf, status))
    return out


def _pad(n: int) -> int:
    return (n + 255) & -256


def _scale_count(gran: int, batch: int, rows: int, cols: int) -> int:
    if gran == L.GRAN_TILE128:
        return batch * (rows // 128) * (cols // 128)
    if gran == L.GRAN_TILE128X256:
        return batch * (rows // 128) * (cols // 256)
    return batch * rows * (cols // 128) if gran == L.GRAN_GROUP128 else batch * rows


def quant_gemm(a, b, a_gran, b_gran, qmode, hadamard=0, bias=None, post_scale=1.0, flags=0, want_at=False):
    """bf16 a [B, M, K] x bf16 b [N, K] or [B, N, K] -> ([B, M, N], at): both quantizations and the GEMM in one call
    of the library, the int8 operands in one workspace.  want_at (B = 1): at = (int8 a^T [1, K, M], its scales along M)
    for linear_backward, else (None, None)."""
    done = host().quant_gemm(a, b, a_gran, b_gran, qmode, hadamard, bias, post_scale, flags, want_at)
    if done is not None:
        return done
    a, b = _check_bf16(a, "a"), _check_bf16(b, "b")
    B, M, K = a.shape
    bb = b.dim() == 3
    N = b.shape[-2]
    if b.shape[-1] != K or (bb and b.shape[0] != B):
        raise ValueError(f"operand shapes do not match: {tuple(a.shape)} x {tuple(b.shape)}")
    bias = _check_bias(bias, N)
    dev = a.device
    out = torch.empty((B, M, N), dtype=torch.float32 if flags & L.GEMM_OUT_F32 else torch.bfloat16, device=dev)
    nb = B if bb else 1
    size = (_pad(B * M * K) + _pad(nb * N * K) + _pad(4 * _scale_count(a_gran, B, M, K)) +
            _pad(4 * _scale_count(b_gran, nb, N, K)) + (_pad(4 * K) if want_at else 0))
    ws = torch.empty(size, dtype=torch.int8, device=dev)
    qt = st = None
    if want_at:
        qt = torch.empty((B, K, M), dtype=torch.int8, device=dev)
        shape = (B, K // 128, M // 128) if a_gran == L.GRAN_TILE128 else ((B, K) if a_gran == L.GRAN_ROW else (B, K, M // 128))
        st = torch.empty(shape, dtype=torch.float32, device=dev)
    status = device_status(dev)
    _call("i8l_quant_gemm", dev, a.data_ptr(), b.data_ptr(), _ptr(bias), out.data_ptr(), _ptr(qt), _ptr(st), B, M, N, K,
          int(bb), a_gran, b_gran, qmode, hadamard, float(post_scale), flags, ws.data_ptr(), size, status.data_ptr(),
          tensors=(b, bias))
    return out, (qt, st)


def linear_backward(dy, w, xt, gran, qmode, hadamard=0, post_dx=1.0, post_dw=1.0, flags=0, need_dx=True, need_dw=True):
    """dy bf16 [M, N], w bf16 [N, K], xt from quant_gemm(want_at=True) -> (dx [M, K] or None, dw [N, K] or None), all
    quantizations and both GEMMs in one call of the library."""
    dy, w = _check_bf16(dy, "dy"), _check_bf16(w, "w")
    M, N = dy.shape
    K = w.shape[1]
    if w.shape[0] != N:
        raise ValueError(f"operand shapes do not match: {tuple(dy.shape)} x {tuple(w.shape)}")
    dev = dy.device
    dx = torch.empty((M, K), dtype=torch.bfloat16, device=dev) if need_dx else None
    dw = torch.empty((N, K), dtype=torch.bfloat16, device=dev) if need_dw else None
    xqt, xst = _check_saved(*xt, M, K, gran) if need_dw else (None, None)
    size = _pad(4 * max(K, N))
    if need_dx:
        size += _pad(M * N) + _pad(4 * _scale_count(gran, 1, M, N)) + _pad(4 * K)
        size += 0 if need_dw else _pad(K * N)   # with both gradients the int8 w^T lies in dw until dx is done
    if need_dw:
        size += _pad(N * M) + _pad(4 * _scale_count(gran, 1, N, M))
    ws = torch.empty(size, dtype=torch.int8, device=dev)
    status = device_status(dev)
    _call("i8l_linear_backward", dev, dy.data_ptr(), w.data_ptr(), _ptr(xqt), _ptr(xst), _ptr(dx), _ptr(dw), M, N, K, gran,
          qmode, hadamard, float(post_dx), float(post_dw), flags, ws.data_ptr(), size, status.data_ptr(),
          tensors=(w, xqt, xst))
    return dx, dw


def col_sum(x: torch.Tensor) -> torch.Tensor:
    """x bf16 [R, C] -> bf16 [C], the sum over the rows."""
    x = _check_bf16(x, "x")
    R, C = x.shape
    out = torch.empty((C,), dtype=torch.bfloat16, device=x.device)
    _call("i8l_col_sum", x.device, x.data_ptr(), R, C, out.data_ptr())
    return out


def gemm_dump_i32(aq, bq, per_block=False, status=None):
    aq, bq = aq.contiguous(), bq.contiguous()
    B, M, N, K, bb = _gemm_dims(aq, bq)
    shape = (B, K // 128, M, N) if per_block else (B, M, N)
    out = torch.empty(shape, dtype=torch.int32, device=aq.device)
    status = device_status(aq.device) if status is None else status
    _call("i8l_gemm_dump_i32", aq.device, aq.data_ptr(), bq.data_ptr(), int(bb), out.data_ptr(), B, M, N, K, int(per_block),
          _ptr(status), tensors=(bq, status))
    return out


def gemm_block_scatter(aq, bq, a_s, b_s, slot_ptrs, rank: int, b_kind=L.BSCALE_CHANNEL, post_scale=1.0, status=None):
    """Block-scaled GEMM [M, K] x [N, K]^T whose row block o goes to slot `rank` of the bf16
    [world, M/world, N] buffer at slot_ptrs[o] (device pointers, peers included).  Nothing is returned:
    the caller synchronises the ranks and sums its own buffer with sum_slots."""
    import ctypes
    aq, bq = aq.contiguous(), bq.contiguous()
    B, M, N, K, bb = _gemm_dims(aq, bq)
    if B != 1 or bb:
        raise ValueError("gemm_block_scatter: one batch, shared B operand")
    world = len(slot_ptrs)
    arr = (ctypes.c_void_p * world)(*[int(p) for p in slot_ptrs])
    a_s, b_s = a_s.contiguous(), b_s.contiguous()
    status = device_status(aq.device) if status is None else status
    _call("i8l_gemm_block_scatter", aq.device, aq.data_ptr(), bq.data_ptr(), a_s.data_ptr(),
          b_s.data_ptr(), b_kind, float(post_scale), ctypes.cast(arr, ctypes.c_void_p), world, int(rank),
          M, N, K, _ptr(status), tensors=(bq, a_s, b_s, status))


def sum_slots(slots: torch.Tensor, out: torch.Tensor | None = None) -> torch.Tensor:
    """slots bf16 [world, rows, cols] -> bf16 [rows, cols], summed in slot order in fp32."""
    if slots.dtype != torch.bfloat16 or slots.dim() != 3 or not slots.is_contiguous():
        raise TypeError("sum_slots: contiguous bf16 [world, rows, cols]")
    world, rows, cols = slots.shape
    if out is None:
        out = torch.empty((rows, cols), dtype=torch.bfloat16, device=slots.device)
    _call("i8l_sum_slots", slots.device, slots.data_ptr(), out.data_ptr(), world, rows, cols, tensors=(out,))
    return out


class cta_limit:
    """Context manager: GEMMs launched inside use at most `n` CTAs, leaving the other SMs to a kernel
    running beside them (a collective on another stream).  n <= 0 means no limit."""

    def __init__(self, n: int):
        self.n = max(0, int(n))

    def __enter__(self):
        L.call("i8l_set_cta_limit", self.n)
        return self

    def __exit__(self, *exc):
        L.call("i8l_set_cta_limit", 0)
        return False
