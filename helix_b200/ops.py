"""Operator front-end over the C ABI.  torch supplies device memory and streams only.

These calls replace what the reference does by spawning a per-configuration
executable and parsing its stdout (scripts/Ampere_FP16/Ampere_FP16_gemm.py
:432-441, scripts/Ampere_FP16/Ampere_FP16_conv.py:431-446,
scripts/Ampere_FP32/Ampere_FP32_gemm.py:101-107).  Layouts follow the reference
kernels: fp16 GEMM takes A[M,K] and B stored [N,K]; fp32 GEMM takes A[M,K] (or
K x M with ``trans_a``) and B[K,N].
"""
import ctypes
import warnings

import torch

from . import _lib
from ._lib import Cfg, DevInfo, Launch, OP_CONV_F16, OP_GEMM_F16, OP_GEMM_F32, OP_GEMV_F16, check

_status_words = {}
_workspaces = {}
_eager = None


class _PythonCalls:
    """In the place of the native module where that cannot be imported: it covers nothing, and launches through ctypes."""

    def __getattr__(self, name):
        return lambda *args: None

    @staticmethod
    def run(launch):
        dev = torch.cuda.current_device()
        check(_lib.load().helix_launch(ctypes.byref(launch), status_word(dev).data_ptr(), _stream(dev)), "helix_launch")


def _native():
    """The native form of the eager operators (csrc/eager_call.cpp): a call it does not cover returns None and goes through
    the Python implementation below.  Without it (not built, or built for another torch, which it checks itself) every call does:
    the same launches, some 8 us of host time more for each."""
    global _eager
    if _eager is None:
        lib = _lib.load()
        try:
            from . import _eager_call
        except ImportError as e:
            warnings.warn(f"helix_b200/_eager_call is not used ({e}): eager operators go through ctypes, which is slower.  Build it "
                          "with `python -m helix_b200.build`.", RuntimeWarning, stacklevel=3)
            _eager = _PythonCalls()
            return _eager
        _eager_call.connect(ctypes.cast(lib.helix_launch, ctypes.c_void_p).value,
                            ctypes.cast(lib.helix_workspace_bytes, ctypes.c_void_p).value,
                            _status_words, status_word, workspace, check)
        _eager = _eager_call
    return _eager


def _require_cuda(*tensors):
    """Operands of one launch: CUDA tensors of one device whose elements all have a place of their own (in the C ABI a leading
    dimension or batch stride of 0 stands for a contiguous operand, so an expanded one would be read past its end)."""
    for t in tensors:
        if not t.is_cuda:
            raise ValueError("helix_b200 operators take CUDA tensors only (there is no CPU path)")
        if t.get_device() != tensors[0].get_device():
            raise ValueError(f"operands on different devices: {tensors[0].device} and {t.device}")
        if 0 in t.stride() and any(n > 1 and st == 0 for n, st in zip(t.shape, t.stride())):
            raise ValueError("expanded operands (a stride of 0) are not supported: make them contiguous")


def _stream(dev=None):
    """Handle of torch's current stream.  torch.cuda.current_stream() builds a Stream object to hold it (3.4 us, as much as
    the launch itself); the raw getter returns the integer."""
    return torch._C._cuda_getCurrentRawStream(torch.cuda.current_device() if dev is None else dev)


def status_word(device=None):
    """Per-device int32 the kernels write HELIX_ERR_TIMEOUT into when a bounded wait runs out."""
    dev = device if isinstance(device, int) else torch.cuda.current_device() if device is None else torch.device(device).index
    word = _status_words.get(dev)
    if word is None:
        word = _status_words[dev] = torch.zeros(1, dtype=torch.int32, device=f"cuda:{dev}")
    return word


def check_status(device=None):
    """Synchronising read of the status word; raises HelixError if a kernel reported a failure."""
    w = status_word(device)
    v = int(w.item())
    if v != 0:
        w.zero_()
        raise _lib.HelixError(v, "device status word")


def workspace(nbytes, device=None, lane=0):
    """Grow-only scratch buffer per device (and per lane of concurrent launch chains), reused across
    calls that are ordered on one stream."""
    dev = torch.cuda.current_device() if device is None else torch.device(device).index
    cur = _workspaces.get((dev, lane))
    if cur is None or cur.numel() < nbytes:
        cur = torch.empty(max(int(nbytes), 1 << 20), dtype=torch.uint8, device=f"cuda:{dev}")
        _workspaces[(dev, lane)] = cur
    return cur


def limit_ctas(launch, max_ctas, lane=0):
    """Let `launch` spread over at most `max_ctas` SMs (so that independent launches on other streams can
    run beside it) and give it the scratch buffer of its lane; the library re-chooses its configuration
    for the smaller machine when cfg is left to it."""
    lib = _lib.load()
    launch.cfg.max_ctas = int(max_ctas)
    need = lib.helix_workspace_bytes(ctypes.byref(launch))
    if need:
        buf = workspace(need, lane=lane)
        launch.ws = buf.data_ptr()
        launch.ws_bytes = buf.numel() * buf.element_size()
        launch._ws_ref = buf
    else:
        launch.ws, launch.ws_bytes = None, 0
    return launch


def device_info(dev=-1):
    info = DevInfo()
    check(_lib.load().helix_device_info(dev, ctypes.byref(info)), "helix_device_info")
    return info


def configs(op):
    lib = _lib.load()
    out = []
    for i in range(lib.helix_num_configs(op)):
        c = Cfg()
        if lib.helix_get_config(op, i, ctypes.byref(c)) == 0:
            out.append(c)
    return out


def default_config(launch):
    """The configuration the library picks for `launch` when its cfg is left zero (helix_default_config)."""
    c = Cfg()
    check(_lib.load().helix_default_config(ctypes.byref(launch), ctypes.byref(c)), "helix_default_config")
    return c


def kernel_name(launch):
    """Name of the main kernel `launch` resolves to (its first template arguments).  GEMVs and products of up to 16 rows without
    a configuration are one family each, whose kernel the library picks by sizes (gemv_f16_streams, gemv_f16_stream_covers and
    gemv_f32_streams in csrc/)."""
    own = launch.cfg.tile_n or launch.cfg.tile_m
    c = launch.cfg if own else default_config(launch)
    if launch.op == _lib.OP_GEMV_F16:
        return "gemv_f16_kernel" if own else "gemv_f16"
    if launch.op == _lib.OP_GEMV_F32:
        return "gemv_f32_kernel" if own else "gemv_f32"
    if launch.op == OP_GEMM_F16 and not own and launch.batch <= 1 and launch.M <= 16 and launch.N >= 1024 and launch.K >= 512:
        return "gemm_f16_skinny"
    if launch.op == _lib.OP_GEMM_F32:
        return "%s<%d,%d>" % ("sgemm_f32_ring_kernel" if c.stages >= 3 else "sgemm_f32_kernel", c.tile_m, c.tile_n)
    if c.cta_group == 2:
        return "gemm_f16_tc2_kernel<%d>" % c.tile_n
    gathers = False
    if launch.op == OP_CONV_F16:
        n, h, w, ch, ko, r, s, stride, pad = list(launch.conv)
        if ch == 4:
            return "conv_f16_stem_kernel<%d>" % (4 if ko <= 64 else 2)
        rows_geom = ch == 64 and ko == 64 and r == 3 and s == 3 and stride == 1 and pad == 1 and w + 2 <= 64
        if rows_geom and c.conv_gather == 4:    # explicit, or the library's default for this geometry
            return "conv_f16_rows_kernel"
        as_gemm = r == 1 and s == 1 and stride == 1 and pad == 0
        if c.conv_gather >= 3 and not as_gemm:
            return "conv_f16_win_kernel" if c.conv_gather == 3 else "conv_f16_rows_kernel"
        gathers = not as_gemm and conv_pixel_channels(launch) == 0
    return "gemm_f16_tc_kernel<%d,%d>" % (c.tile_n, 1 if gathers else 0)


def conv_pixel_channels(launch):
    """Channels of a filter tap that an fp16 convolution's kernel fetches per pixel through the im2col tensor map (64, 32 or 16), or
    0 where warps gather its pixels (helix_conv_pixel_channels)."""
    n = _lib.load().helix_conv_pixel_channels(ctypes.byref(launch))
    if n < 0:
        check(n, "helix_conv_pixel_channels")
    return n


def conv_reads_tensor_map(n, h, w, ch, stride, ko=0, r=1, s=1, pad=0):
    """True where the implicit GEMM may fetch its input through the im2col tensor map in slabs of 64 channels (conv_im2col_eligible in
    csrc/gemm_f16_tc.cu; conv_pixel_channels says what a launch does): the channels a 64-channel block is filled up with must be few and, where ch is no multiple of 16,
    the layer small (`ko` output channels of an r x s filter)."""
    filled = (ch + 63) // 64 * 64
    few = filled * 3 <= ch * 4 if ch % 32 == 0 else filled * 5 <= ch * 6 and ch >= 96
    if ch % 16 != 0:
        ho, wo = conv_out_hw(h, w, r, s, stride, pad)
        macs = n * ho * wo * ko * r * s * ch
        few = few and (macs <= 4e9 or filled * 10 <= ch * 11 and macs <= 3e10)
    return ch % 8 == 0 and few and n * h * w * ch * 2 >= 131072 and stride <= 8


def make_cfg(op, tile_m=128, tile_n=128, tile_k=64, stages=0, cta_group=1, split_k=1, swap_ab=0, raster=8,
             thread_m=0, thread_n=0, load_group=0, stream_k=0, conv_gather=0, probe=0):
    c = Cfg()
    c.op, c.tile_m, c.tile_n, c.tile_k, c.stages = op, tile_m, tile_n, tile_k, stages
    c.cta_group, c.split_k, c.swap_ab, c.raster, c.thread_m, c.thread_n = cta_group, split_k, swap_ab, raster, thread_m, thread_n
    c.load_group = load_group
    c.stream_k = stream_k
    c.conv_gather = conv_gather
    c.probe = probe
    return c


# ----------------------------------------------------------------------------- launch builders
def _finish(launch, cfg, ws):
    lib = _lib.load()
    if cfg is not None:
        launch.cfg = cfg
    need = lib.helix_workspace_bytes(ctypes.byref(launch))
    if need:
        buf = ws if ws is not None else workspace(need, launch._refs[0].device)
        if buf.numel() * buf.element_size() < need:
            raise ValueError(f"workspace too small: need {need} bytes")
        launch.ws = buf.data_ptr()
        launch.ws_bytes = buf.numel() * buf.element_size()
        launch._ws_ref = buf
    return launch


def launch_gemm_f16(a, b_nk, out, cfg=None, ws=None):
    """A[M,K] (or [B,M,K]) x B[N,K] (or [B,N,K]) -> out[M,N] (or [B,M,N]), fp16."""
    _require_cuda(a, b_nk, out)
    assert a.dtype == b_nk.dtype == out.dtype == torch.float16
    l = Launch()
    l.op = OP_GEMM_F16
    if a.dim() == 3:
        assert a.stride(2) == 1 and b_nk.stride(2) == 1 and out.stride(2) == 1
        l.batch, l.M, l.K = a.shape
        l.N = b_nk.shape[1]
        assert b_nk.shape[0] == out.shape[0] == l.batch
        l.lda, l.ldb, l.ldc = a.stride(1), b_nk.stride(1), out.stride(1)
        l.stride_a, l.stride_b, l.stride_c = a.stride(0), b_nk.stride(0), out.stride(0)
    else:
        assert a.stride(1) == 1 and b_nk.stride(1) == 1 and out.stride(1) == 1
        l.batch = 1
        l.M, l.K = a.shape
        l.N = b_nk.shape[0]
        l.lda, l.ldb, l.ldc = a.stride(0), b_nk.stride(0), out.stride(0)
    assert b_nk.shape[-1] == l.K and tuple(out.shape[-2:]) == (l.M, l.N)
    l.a, l.b, l.c = a.data_ptr(), b_nk.data_ptr(), out.data_ptr()
    l._refs = (a, b_nk, out)
    return _finish(l, cfg, ws)


def launch_gemv_f16(w, x, out, cfg=None, ws=None, out_transposed=False):
    """W[rows,K], X[m,K] (m <= 8) -> out[m,rows]; or out[rows,m] when ``out_transposed``."""
    _require_cuda(w, x, out)
    assert w.dtype == x.dtype == out.dtype == torch.float16
    assert w.stride(1) == 1 and x.stride(1) == 1
    l = Launch()
    l.op = OP_GEMV_F16
    l.N, l.K = w.shape
    l.M = x.shape[0]
    assert x.shape[1] == l.K
    l.lda, l.ldb = w.stride(0), x.stride(0)
    if out_transposed:
        assert tuple(out.shape) == (l.N, l.M)
        l.ldc, l.ldc_inner = out.stride(1), out.stride(0)
    else:
        assert tuple(out.shape) == (l.M, l.N)
        l.ldc, l.ldc_inner = out.stride(0), out.stride(1)
    l.a, l.b, l.c = w.data_ptr(), x.data_ptr(), out.data_ptr()
    l._refs = (w, x, out)
    return _finish(l, cfg, ws)


def launch_gemv_f32(w, x, out, cfg=None, ws=None, out_transposed=False):
    """W[rows,K], X[m,K] (m <= 8), fp32 -> out[m,rows]; or out[rows,m] when ``out_transposed``."""
    _require_cuda(w, x, out)
    assert w.dtype == x.dtype == out.dtype == torch.float32
    assert w.stride(1) == 1 and x.stride(1) == 1
    l = Launch()
    l.op = _lib.OP_GEMV_F32
    l.N, l.K = w.shape
    l.M = x.shape[0]
    assert x.shape[1] == l.K
    l.lda, l.ldb = w.stride(0), x.stride(0)
    if out_transposed:
        assert tuple(out.shape) == (l.N, l.M)
        l.ldc, l.ldc_inner = out.stride(1), out.stride(0)
    else:
        assert tuple(out.shape) == (l.M, l.N)
        l.ldc, l.ldc_inner = out.stride(0), out.stride(1)
    l.a, l.b, l.c = w.data_ptr(), x.data_ptr(), out.data_ptr()
    l._refs = (w, x, out)
    return _finish(l, cfg, ws)


def gemv_f32(w, x, out=None, cfg=None):
    if cfg is None and (y := _native().gemv_f32(w, x, out)) is not None:
        return y
    if out is None:
        out = w.new_empty((x.shape[0], w.shape[0]))
    _run_eager(launch_gemv_f32(w, x, out, cfg))
    return out


def conv_out_hw(H, W, R, S, stride, pad):
    return (H + 2 * pad - R) // stride + 1, (W + 2 * pad - S) // stride + 1


def conv_stored_channels(IC, H, W, OC, kh, kw, stride, pad):
    """Channels an NHWC fp16 activation of IC logical channels is stored with (the rest are zeros).  Pixels are
    16 bytes or more (C a multiple of 8) for the tensor-map kernels; an input of up to 4 channels is stored as 4
    where the first-layer kernel covers the geometry (stride 2, filter up to 8 x 7, output rows of up to 128 pixels,
    64 or 128 output channels -- the conditions of conv_f16_stem_eligible in csrc/conv_f16_stem.cu)."""
    if IC <= 4 and stride == 2 and 2 <= kh <= 8 and pad < kh and W % 2 == 0 and OC in (64, 128):
        P = (pad + 1) & ~1
        Wo = (W + 2 * pad - kw) // 2 + 1
        Ho = (H + 2 * pad - kh) // 2 + 1
        if P - pad + kw <= 8 and 1 <= Wo <= 128 and Ho >= 1 and (P + W) * 8 <= 2176:
            return 4
    return (IC + 7) // 8 * 8


def conv_has_fixed_kernel(N, C, H, W, KO, R, S, stride, pad):
    """True where the library runs a convolution through a kernel without a tunable configuration (the 4-channel
    first-layer kernel, the 64 -> 64 channel row-pair kernel): nothing for a cost model to pick there."""
    if C == 4:
        return True
    l = Launch()
    l.op = OP_CONV_F16
    for i, v in enumerate((N, H, W, C, KO, R, S, stride, pad)):
        l.conv[i] = v
    return default_config(l).conv_gather == 4


def launch_conv2d_f16(x, w, out, stride, pad, cfg=None, ws=None):
    """x[N,H,W,C], w[KO,R,S,C] -> out[N,Ho,Wo,KO], all contiguous fp16."""
    _require_cuda(x, w, out)
    assert x.dtype == w.dtype == out.dtype == torch.float16
    assert x.is_contiguous() and w.is_contiguous() and out.is_contiguous()
    N, H, W, C = x.shape
    KO, R, S, C2 = w.shape
    assert C == C2
    Ho, Wo = conv_out_hw(H, W, R, S, stride, pad)
    assert tuple(out.shape) == (N, Ho, Wo, KO)
    l = Launch()
    l.op = OP_CONV_F16
    l.a, l.b, l.c = x.data_ptr(), w.data_ptr(), out.data_ptr()
    for i, v in enumerate((N, H, W, C, KO, R, S, stride, pad)):
        l.conv[i] = v
    l._refs = (x, w, out)
    return _finish(l, cfg, ws)


def launch_conv2d_f32(x, w, out, stride, pad, cfg=None, ws=None):
    """x[N,H,W,C], w[KO,R,S,C] -> out[N,Ho,Wo,KO], true fp32 (FFMA GEMM over the windows, see conv_f32.cu)."""
    _require_cuda(x, w, out)
    assert x.dtype == w.dtype == out.dtype == torch.float32
    assert x.is_contiguous() and w.is_contiguous() and out.is_contiguous()
    N, H, W, C = x.shape
    KO, R, S, C2 = w.shape
    assert C2 == C
    Ho, Wo = conv_out_hw(H, W, R, S, stride, pad)
    assert tuple(out.shape) == (N, Ho, Wo, KO)
    l = Launch()
    l.op = _lib.OP_CONV_F32
    for i, v in enumerate((N, H, W, C, KO, R, S, stride, pad)):
        l.conv[i] = v
    l.a, l.b, l.c = x.data_ptr(), w.data_ptr(), out.data_ptr()
    l._refs = (x, w, out)
    return _finish(l, cfg, ws)


def conv2d_f32_nhwc(x, w, stride=1, pad=0, out=None, cfg=None):
    if cfg is None and (y := _native().conv2d_f32(x, w, stride, pad, out)) is not None:
        return y
    N, H, W, _ = x.shape
    KO, R, S, _ = w.shape
    Ho, Wo = conv_out_hw(H, W, R, S, stride, pad)
    if out is None:
        out = x.new_empty((N, Ho, Wo, KO))
    _run_eager(launch_conv2d_f32(x, w, out, stride, pad, cfg))
    return out


def launch_gemm_f32(a, b, out, trans_a=False, cfg=None):
    """A[M,K] (or [K,M] with trans_a) x B[K,N] -> out[M,N], fp32 FFMA."""
    _require_cuda(a, b, out)
    assert a.dtype == b.dtype == out.dtype == torch.float32
    assert a.stride(1) == 1 and b.stride(1) == 1 and out.stride(1) == 1
    l = Launch()
    l.op = OP_GEMM_F32
    if trans_a:
        l.K, l.M = a.shape
    else:
        l.M, l.K = a.shape
    assert b.shape[0] == l.K
    l.N = b.shape[1]
    assert tuple(out.shape) == (l.M, l.N)
    l.lda, l.ldb, l.ldc = a.stride(0), b.stride(0), out.stride(0)
    l.trans_a = int(trans_a)
    l.a, l.b, l.c = a.data_ptr(), b.data_ptr(), out.data_ptr()
    l._refs = (a, b, out)
    return _finish(l, cfg, None)


def run(launch):
    """Queue a prepared launch on torch's current stream; its operands live on the current device."""
    _native().run(launch)


def _run_eager(launch):
    dev = launch._refs[0].device
    if dev.index != torch.cuda.current_device():
        raise ValueError(f"operands on {dev} while device {torch.cuda.current_device()} is current")
    run(launch)


# ----------------------------------------------------------------------------- eager operators
def gemm_f16(a, b_nk, out=None, cfg=None):
    if cfg is None and (y := _native().gemm_f16(a, b_nk, out)) is not None:
        return y
    shape = (*a.shape[:-1], b_nk.shape[-2])
    if out is None:
        out = a.new_empty(shape)
    _run_eager(launch_gemm_f16(a, b_nk, out, cfg))
    return out


def gemv_f16(w, x, out=None, cfg=None):
    if cfg is None and (y := _native().gemv_f16(w, x, out)) is not None:
        return y
    if out is None:
        out = w.new_empty((x.shape[0], w.shape[0]))
    _run_eager(launch_gemv_f16(w, x, out, cfg))
    return out


def conv2d_f16_nhwc(x, w, stride=1, pad=0, out=None, cfg=None):
    if cfg is None and (y := _native().conv2d_f16(x, w, stride, pad, out)) is not None:
        return y
    if out is None:
        Ho, Wo = conv_out_hw(x.shape[1], x.shape[2], w.shape[1], w.shape[2], stride, pad)
        out = x.new_empty((x.shape[0], Ho, Wo, w.shape[0]))
    _run_eager(launch_conv2d_f16(x, w, out, stride, pad, cfg))
    return out


def gemm_f32(a, b, trans_a=False, out=None, cfg=None):
    if cfg is None and (y := _native().gemm_f32(a, b, trans_a, out)) is not None:
        return y
    M = a.shape[1] if trans_a else a.shape[0]
    if out is None:
        out = a.new_empty((M, b.shape[1]))
    _run_eager(launch_gemm_f32(a, b, out, trans_a, cfg))
    return out


# ----------------------------------------------------------------------------- timing
def time_launches(launches, warmup=3, iters=20, use_graph=False):
    """Seconds per launch (average), plus (min, max) seconds per round over the list.

    The list is walked round-robin, so passing launches over distinct operand
    buffers whose total footprint exceeds the L2 gives HBM-resident timings.
    """
    arr = (Launch * len(launches))()
    for i, l in enumerate(launches):
        ctypes.memmove(ctypes.byref(arr[i]), ctypes.byref(l), ctypes.sizeof(Launch))
    avg, mn, mx = ctypes.c_double(), ctypes.c_double(), ctypes.c_double()
    torch.cuda.synchronize()
    check(_lib.load().helix_time_launches(arr, len(launches), warmup, iters, int(use_graph),
                                          ctypes.byref(avg), ctypes.byref(mn), ctypes.byref(mx)),
          "helix_time_launches")
    return avg.value, mn.value, mx.value


def capture_timeline(launch, warm=2):
    """Run `launch` (a one-CTA fp16 GEMM / convolution) with timeline capture on and return an int64
    array [CTAs, words] of the stamps described at helix_trace_buffer; rows of CTAs that did not run
    stay zero.  The stamps are those of the kernel's general variant: `launch` without capture may run a leaner one."""
    lib = _lib.load()
    words = lib.helix_trace_words_per_cta()
    ctas = device_info().sm_count
    buf = torch.zeros((ctas, words), dtype=torch.int64, device="cuda")
    for _ in range(warm):
        run(launch)
    torch.cuda.synchronize()
    check(lib.helix_trace_buffer(buf.data_ptr(), buf.numel() * 8), "helix_trace_buffer")
    try:
        run(launch)
        torch.cuda.synchronize()
    finally:
        lib.helix_trace_buffer(None, 0)
    check_status()
    return buf.cpu().numpy()


def selftest_bounded_wait(limit_ns=2_000_000):
    """Launch the library's wait self-test on the current stream: a wait nothing satisfies gives up after
    `limit_ns` and leaves HELIX_ERR_TIMEOUT in the status word (read it with check_status)."""
    check(_lib.load().helix_selftest_bounded_wait(int(limit_ns), ctypes.c_void_p(status_word().data_ptr()), _stream()),
          "helix_selftest_bounded_wait")


def launch_count():
    return int(_lib.load().helix_launch_count())
