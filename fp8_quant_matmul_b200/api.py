"""ctypes binding of libfp8bs.so and the Python mirror of the reference's operator surface.

Device memory, streams and (in the benchmark) torch.distributed come from PyTorch; all
arithmetic happens in the library's CUDA kernels.
"""
import ctypes
import itertools
import os
import threading

import numpy as np

_PKG_DIR = os.path.dirname(os.path.abspath(__file__))
_LIB_PATH = os.path.join(_PKG_DIR, "lib", "libfp8bs.so")

PATH_AUTO, PATH_MN_LARGE, PATH_MN_SMALL = 0, 1, 2
TILE_PAIR = 0x1000      # tile_n = 256 | TILE_PAIR: a 256 x 256 tile owned by a pair of CTAs
SPLIT_WORKSPACE = 0x2000  # OR into tile_n: reduce split-K partial sums through the workspace, not in a cluster
STREAM_K = 0x4000         # OR into tile_n: deal the K blocks of all tiles out evenly over the SMs (needs the workspace)
SMALL_M = 0x10000         # tile_n = SMALL_M: M <= 64, the kernel for few rows (select_path reports 128 | SMALL_M)
SHORT_K = 0x8000          # OR into tile_n (0 or 256): K <= 256, both K blocks of a tile stay in tensor memory

# The 18 benchmark shapes (M, N, K) of the reference's results table (README.md:15-25).
SHAPES_18 = [(m, n, k) for m in (1024, 6144)
             for (n, k) in ((1536, 7168), (3072, 1536), (576, 7168), (7168, 256), (7168, 2048),
                            (4608, 7168), (7168, 2304), (512, 7168), (4096, 512))]


class Fp8bsError(RuntimeError):
    def __init__(self, code, where):
        self.code = code
        super().__init__("%s failed: %d (%s)" % (where, code, status_string(code)))


_lib = None

_c = ctypes
_SIGS = {
    "fp8bs_gemm": (_c.c_int, [_c.c_void_p] * 5 + [_c.c_int] * 3 + [_c.c_void_p, _c.c_size_t, _c.c_void_p]),
    "fp8bs_gemm_mn_large": (_c.c_int, [_c.c_void_p] * 5 + [_c.c_int] * 3 + [_c.c_void_p]),
    "fp8bs_gemm_mn_small": (_c.c_int, [_c.c_void_p] * 5 + [_c.c_int] * 4 + [_c.c_void_p, _c.c_size_t, _c.c_void_p]),
    "fp8bs_gemm_mn_small_static": (_c.c_int, [_c.c_void_p] * 5 + [_c.c_int] * 4 + [_c.c_void_p]),
    "fp8bs_gemm_ex": (_c.c_int, [_c.c_void_p] * 5 + [_c.c_int] * 8 + [_c.c_void_p, _c.c_size_t, _c.c_void_p]),
    "fp8bs_gemm_scatter": (_c.c_int, [_c.c_void_p] * 4 + [_c.POINTER(_c.c_void_p)] + [_c.c_int] * 6 + [_c.c_void_p]),
    "fp8bs_gemm_ref": (_c.c_int, [_c.c_void_p] * 5 + [_c.c_int] * 3 + [_c.c_void_p]),
    "fp8bs_select_path": (_c.c_int, [_c.c_int] * 3 + [_c.POINTER(_c.c_int)] * 2),
    "fp8bs_select_path_sms": (_c.c_int, [_c.c_int] * 4 + [_c.POINTER(_c.c_int)] * 3),
    "fp8bs_workspace_bytes": (_c.c_size_t, [_c.c_int] * 3),
    "fp8bs_workspace_bytes_ex": (_c.c_size_t, [_c.c_int] * 6),
    "fp8bs_workspace_init": (_c.c_int, [_c.c_void_p, _c.c_size_t, _c.c_void_p]),
    "fp8bs_capture_id": (_c.c_int, [_c.c_void_p, _c.POINTER(_c.c_ulonglong)]),
    "fp8bs_capture_hold": (_c.c_int, [_c.c_void_p, _c.c_ulonglong]),
    "fp8bs_capture_released": (_c.c_int, [_c.POINTER(_c.c_ulonglong), _c.c_int]),
    "fp8bs_last_device_status": (_c.c_int, [_c.c_void_p, _c.POINTER(_c.c_uint)]),
    "fp8bs_selftest_wait_timeout": (_c.c_int, [_c.c_void_p]),
    "fp8bs_status_string": (_c.c_char_p, [_c.c_int]),
    "fp8bs_last_cuda_error": (_c.c_int, []),
    "fp8bs_launch_count": (_c.c_ulonglong, []),
    "fp8bs_gemmGPU": (_c.c_int, [_c.c_void_p] * 5 + [_c.c_size_t] * 3 + [_c.c_int]),
    "fp8bs_host_ctx_create": (_c.c_int, [_c.POINTER(_c.c_void_p)] + [_c.c_size_t] * 3),
    "fp8bs_host_ctx_destroy": (_c.c_int, [_c.c_void_p]),
    "fp8bs_host_ctx_buffer": (_c.c_void_p, [_c.c_void_p, _c.c_int]),
    "fp8bs_gemm_host": (_c.c_int, [_c.c_void_p] * 6 + [_c.c_int] * 5),
    "fp8bs_quantize_rowwise": (_c.c_int, [_c.c_void_p, _c.c_int, _c.c_void_p, _c.c_void_p, _c.c_int, _c.c_int, _c.c_float, _c.c_void_p]),
    "fp8bs_quantize_block": (_c.c_int, [_c.c_void_p, _c.c_int, _c.c_void_p, _c.c_void_p, _c.c_int, _c.c_int, _c.c_float, _c.c_void_p]),
    "fp8bs_gen_normal_e4m3": (_c.c_int, [_c.c_void_p, _c.c_size_t, _c.c_uint64]),
    "fp8bs_gen_uniform_f32": (_c.c_int, [_c.c_void_p, _c.c_size_t, _c.c_uint64, _c.c_float, _c.c_float]),
    "fp8bs_float_to_e4m3fn": (_c.c_uint8, [_c.c_float]),
    "fp8bs_e4m3fn_to_float": (_c.c_float, [_c.c_uint8]),
    "fp8bs_fnuz_to_fn_device": (_c.c_int, [_c.c_void_p, _c.c_void_p, _c.c_size_t, _c.c_void_p, _c.c_void_p]),
    "fp8bs_fnuz_to_fn_device_sync": (_c.c_int, [_c.c_void_p, _c.c_void_p, _c.c_size_t, _c.POINTER(_c.c_uint), _c.c_void_p]),
    "fp8bs_fnuz_to_fn": (_c.c_int, [_c.c_void_p, _c.c_void_p, _c.c_size_t, _c.POINTER(_c.c_size_t)]),
}


def load(path):
    """Load the library from `path` and make it the one every call of this module uses (e.g. the instrumented
    build lib/libfp8bs_prof.so).  Raises if the file is missing: there is no other code path."""
    global _lib
    if not os.path.exists(path):
        raise RuntimeError("libfp8bs.so is not built (%s); run `python -m fp8_quant_matmul_b200.build`. "
                           "There is no fallback implementation." % path)
    handle = ctypes.CDLL(path)
    for name, (res, args) in _SIGS.items():
        fn = getattr(handle, name)
        fn.restype = res
        fn.argtypes = args
    _lib = handle
    _set_up.clear()     # what one build answers about a shape says nothing about another's
    _needs.clear()
    return _lib


def lib():
    """The loaded library.  Raises if it has not been built: there is no other code path."""
    if _lib is None:
        load(_LIB_PATH)
    return _lib


def exported_symbols():
    """Names this binding expects the library to export (all of include/fp8bs.h)."""
    return sorted(_SIGS)


def status_string(code):
    try:
        return lib().fp8bs_status_string(int(code)).decode()
    except Exception:  # library absent: still give a usable message
        return "status %d" % code


def _check(code, where):
    if code != 0:
        raise Fp8bsError(code, where)


def launch_count():
    return int(lib().fp8bs_launch_count())


# ---------------------------------------------------------------- host-only helpers ----
def select_path(M, N, K):
    """(path, splits, tile_n) the run-time dispatch picks for a shape (pure host function)."""
    s, t = _c.c_int(0), _c.c_int(0)
    rc = lib().fp8bs_select_path(M, N, K, _c.byref(s), _c.byref(t))
    if rc < 0:
        raise Fp8bsError(rc, "fp8bs_select_path")
    return rc, s.value, t.value


def select_path_sms(M, N, K, sm_count):
    """(path, splits, tile_n, ctas that must be co-resident) for a GPU with sm_count SMs (pure host function)."""
    s, t, c = _c.c_int(0), _c.c_int(0), _c.c_int(0)
    rc = lib().fp8bs_select_path_sms(M, N, K, sm_count, _c.byref(s), _c.byref(t), _c.byref(c))
    if rc < 0:
        raise Fp8bsError(rc, "fp8bs_select_path_sms")
    return rc, s.value, t.value, c.value


def workspace_bytes(M, N, K, path=None, splits=0, tile_n=0):
    if path is None:
        return int(lib().fp8bs_workspace_bytes(M, N, K))
    return int(lib().fp8bs_workspace_bytes_ex(M, N, K, path, splits, tile_n))


def gen_normal_e4m3(n, seed):
    """n e4m3fn bytes: N(0,1) rounded to nearest even, |x| <= 240, |x| < 2^-6 -> +0."""
    out = np.empty(int(n), dtype=np.uint8)
    _check(lib().fp8bs_gen_normal_e4m3(out.ctypes.data, out.size, int(seed)), "fp8bs_gen_normal_e4m3")
    return out


def gen_uniform_f32(n, seed, lo, hi):
    out = np.empty(int(n), dtype=np.float32)
    _check(lib().fp8bs_gen_uniform_f32(out.ctypes.data, out.size, int(seed), float(lo), float(hi)),
           "fp8bs_gen_uniform_f32")
    return out


def float_to_e4m3fn(x):
    x = np.ascontiguousarray(x, dtype=np.float32)
    f = lib().fp8bs_float_to_e4m3fn
    return np.array([f(float(v)) for v in x.ravel()], dtype=np.uint8).reshape(x.shape)


def e4m3fn_to_float(b):
    b = np.ascontiguousarray(b, dtype=np.uint8)
    f = lib().fp8bs_e4m3fn_to_float
    table = np.array([f(i) for i in range(256)], dtype=np.float32)
    return table[b]


def fnuz_to_fn(src):
    """Re-encode e4m3fnuz bytes as e4m3fn bytes of equal value; raises on a byte that has none."""
    src = np.ascontiguousarray(src, dtype=np.uint8)
    dst = np.empty_like(src)
    bad = _c.c_size_t(0)
    rc = lib().fp8bs_fnuz_to_fn(dst.ctypes.data, src.ctypes.data, src.size, _c.byref(bad))
    if rc != 0:
        err = Fp8bsError(rc, "fp8bs_fnuz_to_fn")
        err.bad_index = bad.value
        raise err
    return dst


def fnuz_to_fn_device(src, dst=None):
    """Re-encode a CUDA uint8 tensor of e4m3fnuz bytes as e4m3fn bytes; returns (dst, number of inexact bytes)."""
    if not src.is_cuda or (dst is not None and (not dst.is_cuda or dst.get_device() != src.get_device())):
        raise ValueError("expected CUDA tensors on one device")
    if dst is None:
        dst = _torch().empty_like(src)
    count = _c.c_uint(0)
    _check(lib().fp8bs_fnuz_to_fn_device_sync(dst.data_ptr(), src.data_ptr(), src.numel(), _c.byref(count),
                                              _stream(src.get_device())), "fp8bs_fnuz_to_fn_device_sync")
    return dst, count.value


# ---------------------------------------------------------------- the operator ---------
_torch_module = None


def _torch():
    global _torch_module
    if _torch_module is None:
        import torch
        _torch_module = torch
    return _torch_module


def _stream(index):
    """Handle of the current stream of CUDA device `index`.  torch.cuda.current_stream(device).cuda_stream gives the same
    number but takes 2.2 us (it builds a Stream object), a third of what a small call costs."""
    return _torch()._C._cuda_getCurrentRawStream(index)


MAX_WORKSPACES = 16
_workspaces = {}        # (device index, stream handle) -> tensor, oldest first
_graph_workspaces = {}  # token -> (device index, stream handle, capture id, tensor)
_tokens = itertools.count(1)
_workspaces_lock = threading.Lock()


def _drop_graph_workspaces():
    """Gives up the workspaces of graphs that no longer exist."""
    gone = (_c.c_ulonglong * 64)()
    for i in range(lib().fp8bs_capture_released(gone, len(gone))):
        _graph_workspaces.pop(gone[i], None)


def _new_workspace(device, stream, nbytes):
    torch = _torch()
    _drop_graph_workspaces()
    ws = torch.empty(max(nbytes, 1 << 20), dtype=torch.uint8, device=device)
    _check(lib().fp8bs_workspace_init(ws.data_ptr(), ws.numel(), stream), "fp8bs_workspace_init")
    return ws


def _workspace(device, index, stream, nbytes):
    """A zero-initialised workspace for a call on the current stream of `device`: calls that may overlap on the GPU never get
    the same one.  One per stream, grown on demand and reused between calls; a captured graph has its own, see below.  Each is
    allocated on the stream that uses it, so one that is replaced or given up goes back to torch's allocator in stream order."""
    if _torch().cuda.is_current_stream_capturing():
        return _graph_workspace(device, index, stream, nbytes)
    ws = _workspaces.get((index, stream))
    if ws is None or ws.numel() < nbytes:
        ws = _new_workspace(device, stream, nbytes)
        with _workspaces_lock:
            _workspaces.pop((index, stream), None)
            while len(_workspaces) >= MAX_WORKSPACES:
                del _workspaces[next(iter(_workspaces))]
            _workspaces[(index, stream)] = ws
    return ws


def _graph_workspace(device, index, stream, nbytes):
    """The workspace of a call that is being captured: one per capture and stream, zeroed by the graph itself, as graphs may be
    replayed beside one another and beside eager calls.  Held until the graph and everything instantiated from it are gone."""
    capture = _c.c_ulonglong(0)
    _check(lib().fp8bs_capture_id(stream, _c.byref(capture)), "fp8bs_capture_id")
    for owner in list(_graph_workspaces.values()):
        if owner[:3] == (index, stream, capture.value) and owner[3].numel() >= nbytes:
            return owner[3]
    ws = _new_workspace(device, stream, nbytes)
    token = next(_tokens)
    _graph_workspaces[token] = (index, stream, capture.value, ws)
    rc = lib().fp8bs_capture_hold(stream, token)
    if rc != 0:
        del _graph_workspaces[token]
        _check(rc, "fp8bs_capture_hold")
    return ws


_needs = {}       # (device index, M, N, K, path, splits, tile_n) -> workspace bytes
_set_up = set()   # devices on which a call has succeeded: from then on the answer for a key no longer changes


def _workspace_need(key):
    need = _needs.get(key)
    if need is None:
        _, M, N, K, path, splits, tile_n = key
        need = workspace_bytes(M, N, K, path, splits, tile_n) if (path or splits or tile_n) else workspace_bytes(M, N, K)
        if key[0] in _set_up:
            if len(_needs) >= 4096:
                _needs.clear()
            _needs[key] = need
    return need


def gemm(A, B, a_scale, b_scale, C=None, M=None, N=None, K=None, path=PATH_AUTO, splits=0, tile_n=0,
         n0=0, n_total=None, workspace=None):
    """C = (A . a_scale) @ (B . b_scale)^T on the current CUDA stream.

    Arguments follow the kernel signature (A, B, As, Bs, C, M, N, K) of mn_large.hip:11:
      A        uint8/float8_e4m3fn CUDA tensor, M*K bytes, column-major  A[m + M*k]
      B        same, N*K bytes, column-major                             B[n + N*k]
      a_scale  float32 CUDA tensor [K/128, M] (memory order a_scale[m + M*kb])
      b_scale  float32 CUDA tensor [K/128, ceil(n_total/128)]
      C        bfloat16 CUDA tensor [M, N] (allocated if None)
    path / splits / tile_n force a kernel; n0 / n_total describe an N-shard.
    workspace is for split-K and stream-K; without one the call uses a workspace of the current stream, or of the graph that it
    is being captured into.  A workspace that is passed in must not be in use by another call on the GPU at the same time.
    """
    torch = _torch()
    if not A.is_cuda:
        raise RuntimeError("fp8bs.gemm needs CUDA tensors; there is no CPU implementation")
    if M is None or N is None or K is None:
        raise ValueError("M, N, K are required (operands are flat column-major buffers)")
    index = A.get_device()
    stream = _stream(index)
    if C is None:
        C = A.new_empty((M, N), dtype=torch.bfloat16)
    if n_total is None:
        n_total = N
    ws_ptr, ws_bytes = None, 0
    if workspace is not None:
        ws_ptr, ws_bytes = workspace.data_ptr(), workspace.numel() * workspace.element_size()
    else:
        need = _workspace_need((index, M, N, K, path, splits, tile_n))
        if need:
            ws = _workspace(A.device, index, stream, need)
            ws_ptr, ws_bytes = ws.data_ptr(), ws.numel()
    rc = lib().fp8bs_gemm_ex(A.data_ptr(), B.data_ptr(), a_scale.data_ptr(), b_scale.data_ptr(), C.data_ptr(),
                             M, N, K, n0, n_total, path, splits, tile_n, ws_ptr, ws_bytes, stream)
    if rc != 0:
        _check(rc, "fp8bs_gemm_ex")
    _set_up.add(index)
    return C


def gemm_scatter(A, B, a_scale, b_scale, dests, M, N, K, n0, n_total, stream=None):
    """N-sharded GEMM with the distribution of C fused into the epilogue: computes columns [n0, n0 + N) of an
    n_total-wide C and stores them into every buffer of `dests` (device pointers as ints, or torch tensors of shape
    [M, n_total] bf16): this GPU's own C and the peer-mapped C of the other GPUs."""
    import torch
    ptrs = [d.data_ptr() if hasattr(d, "data_ptr") else int(d) for d in dests]
    arr = (_c.c_void_p * len(ptrs))(*ptrs)
    if stream is None:
        stream = torch.cuda.current_stream(A.device).cuda_stream
    with torch.cuda.device(A.device):
        rc = lib().fp8bs_gemm_scatter(A.data_ptr(), B.data_ptr(), a_scale.data_ptr(), b_scale.data_ptr(), arr, len(ptrs),
                                      M, N, K, n0, n_total, stream)
    _check(rc, "fp8bs_gemm_scatter")


STATIC_SCRATCH_BYTES = (32 << 20) + 65536


def gemm_mn_small_static(A, B, a_scale, b_scale, M, N, K, splits=0, C=None):
    """Split-K GEMM on the library's built-in scratch array: nothing is allocated, no workspace is passed.

    For callers that cannot allocate device memory when they call.  Problems whose partial sums exceed
    STATIC_SCRATCH_BYTES raise Fp8bsError(-4).  Calls share the scratch: keep them ordered on the GPU.
    C must be given if the caller truly cannot allocate; it is created here only as a convenience.
    """
    torch = _torch()
    if C is None:
        C = torch.empty((M, N), dtype=torch.bfloat16, device=A.device)
    stream = torch.cuda.current_stream(A.device).cuda_stream
    _check(lib().fp8bs_gemm_mn_small_static(A.data_ptr(), B.data_ptr(), a_scale.data_ptr(), b_scale.data_ptr(),
                                            C.data_ptr(), M, N, K, splits, stream), "fp8bs_gemm_mn_small_static")
    return C


def gemm_ref(A, B, a_scale, b_scale, M, N, K, C=None):
    """The ground-truth kernel restated in CUDA (ref_kernel, check.cu:30-49)."""
    torch = _torch()
    if C is None:
        C = torch.empty((M, N), dtype=torch.bfloat16, device=A.device)
    stream = torch.cuda.current_stream(A.device).cuda_stream
    _check(lib().fp8bs_gemm_ref(A.data_ptr(), B.data_ptr(), a_scale.data_ptr(), b_scale.data_ptr(), C.data_ptr(),
                                M, N, K, stream), "fp8bs_gemm_ref")
    return C


def _quantize(fn_name, X, fp8_max):
    torch = _torch()
    if not X.is_cuda or X.dim() != 2 or not X.is_contiguous():
        raise ValueError("expected a contiguous 2-D CUDA tensor [rows, K]")
    if X.dtype not in (torch.float32, torch.bfloat16):
        raise ValueError("fp32 or bf16 input")
    rows, K = X.shape
    q = X.new_empty(rows * K, dtype=torch.uint8)
    block = fn_name.endswith("block")
    n_scales = (K // 128) * (((rows + 127) // 128) if block else rows)
    scales = X.new_empty(n_scales, dtype=torch.float32)
    _check(getattr(lib(), fn_name)(X.data_ptr(), int(X.dtype == torch.bfloat16), q.data_ptr(), scales.data_ptr(),
                                   rows, K, float(fp8_max), _stream(X.get_device())), fn_name)
    return q, scales


def quantize_rowwise(X, fp8_max=448.0):
    """A and a_scale of the GEMM from a row-major [M, K] activation matrix (quantize.py:43-67).
    Returns (A bytes column-major, flat; inverse scales laid out a_scale[m + M*kb])."""
    return _quantize("fp8bs_quantize_rowwise", X, fp8_max)


def quantize_block(W, fp8_max=448.0):
    """B and b_scale of the GEMM from a row-major [N, K] weight matrix (128 x 128 blocks, quantize.py:16-41).
    Returns (B bytes column-major, flat; inverse scales laid out b_scale[nb + ceil(N/128)*kb])."""
    return _quantize("fp8bs_quantize_block", W, fp8_max)


def last_device_status(stream=None):
    """Synchronises and raises if a kernel recorded a barrier timeout."""
    detail = _c.c_uint(0)
    rc = lib().fp8bs_last_device_status(stream, _c.byref(detail))
    if rc != 0:
        err = Fp8bsError(rc, "fp8bs_last_device_status")
        err.detail = detail.value
        raise err


def gemmGPU(A, B, a_scale, b_scale, M, N, K, option=0):
    """Mirror of the reference's gemmGPU (check.cu:51-130): HOST fp32 arrays in, HOST bf16 bits out.

    A is fp32 M x K column-major, B fp32 N x K column-major (flat numpy arrays); they are
    converted to fp8 on the device as the reference does.  option: 0 auto, 1 mn_small, 2 ref kernel.
    Returns a uint16 array [M, N] of bf16 bit patterns.
    """
    A = np.ascontiguousarray(A, dtype=np.float32)
    B = np.ascontiguousarray(B, dtype=np.float32)
    a_scale = np.ascontiguousarray(a_scale, dtype=np.float32)
    b_scale = np.ascontiguousarray(b_scale, dtype=np.float32)
    C = np.empty((M, N), dtype=np.uint16)
    _check(lib().fp8bs_gemmGPU(C.ctypes.data, A.ctypes.data, B.ctypes.data, a_scale.ctypes.data,
                               b_scale.ctypes.data, M, N, K, option), "fp8bs_gemmGPU")
    return C


class HostContext:
    """Reusable end-to-end context: pinned host staging + device buffers, no allocation per call."""

    def __init__(self, max_M, max_N, max_K):
        self._h = _c.c_void_p(None)
        _check(lib().fp8bs_host_ctx_create(_c.byref(self._h), max_M, max_N, max_K), "fp8bs_host_ctx_create")
        self.max = (max_M, max_N, max_K)

    def buffer(self, which, nbytes, dtype):
        """numpy view of pinned staging buffer `which` (0 A, 1 B, 2 a_scale, 3 b_scale, 4 C)."""
        ptr = lib().fp8bs_host_ctx_buffer(self._h, which)
        buf = (_c.c_uint8 * nbytes).from_address(ptr)
        return np.frombuffer(buf, dtype=dtype)

    def gemm(self, C, A, B, a_scale, b_scale, M, N, K, n0=0, n_total=None):
        """Host pointers (numpy arrays, ideally views of the pinned buffers) in and out; synchronous."""
        _check(lib().fp8bs_gemm_host(self._h, C.ctypes.data, A.ctypes.data, B.ctypes.data, a_scale.ctypes.data,
                                     b_scale.ctypes.data, M, N, K, n0, N if n_total is None else n_total),
               "fp8bs_gemm_host")
        return C

    def close(self):
        if self._h:
            lib().fp8bs_host_ctx_destroy(self._h)
            self._h = _c.c_void_p(None)

    def __del__(self):
        try:
            self.close()
        except Exception:
            pass
