"""Loader of ``libfe3d_gb300.so`` and device-buffer plumbing.

The library is a plain C ABI (``include/fe3d_gb300.h``) loaded with ctypes.
PyTorch only provides device memory and the current CUDA stream.  There is no
CPU fallback: every entry point raises if the library or a GPU is missing.
"""
import collections
import ctypes
import os
import threading

import numpy as np

HERE = os.path.dirname(os.path.abspath(__file__))
LIB_PATH = os.path.join(HERE, 'libfe3d_gb300.so')

FE3D_ERRORS = {
    -1: 'invalid argument',
    -2: 'kernel launch failed',
    -3: 'CUDA runtime error',
    -4: 'offset outside the caller\'s buffers',
    -5: 'device allocation failed',
    -6: 'object used in the wrong state',
    -7: 'size above the allocation-free maximum (FE3D_NOALLOC_MAX_ROWS rows)',
}

_lib = None
_err_words = {}

c_i64 = ctypes.c_int64
c_int = ctypes.c_int
c_dbl = ctypes.c_double
c_vp = ctypes.c_void_p

# argument signatures of the exported entry points (see include/fe3d_gb300.h)
_SIGS = {
    'fe3d_version': ([], c_int),
    'fe3d_stream_synchronize': ([c_vp], c_int),
    'fe3d_quad4_frame': ([c_i64, c_vp, c_vp, c_i64, c_vp, c_int, c_vp, c_vp, c_vp, c_vp, c_vp, c_vp], c_int),
    'fe3d_quad4_probe_xe': ([c_i64, c_vp, c_vp, c_i64, c_vp, c_vp, c_vp, c_vp, c_vp], c_int),
    'fe3d_quad4_probe_ue': ([c_i64, c_vp, c_vp, c_i64, c_vp, c_vp, c_vp, c_vp], c_int),
    'fe3d_quad4_kc0': ([c_i64, c_vp, c_vp, c_vp, c_i64, c_vp, c_int, c_vp, c_vp, c_vp, c_vp, c_vp, c_i64,
                        c_vp, c_vp, c_vp, c_vp, c_i64, c_int, c_vp, c_vp], c_int),
    'fe3d_quad4_kg': ([c_i64, c_vp, c_vp, c_vp, c_i64, c_vp, c_int, c_vp, c_i64, c_vp, c_vp, c_vp, c_vp,
                       c_vp, c_i64, c_vp, c_vp, c_vp, c_vp, c_i64, c_vp, c_vp], c_int),
    'fe3d_quad4_m': ([c_i64, c_vp, c_vp, c_vp, c_i64, c_vp, c_vp, c_vp, c_vp, c_i64, c_vp, c_vp, c_vp,
                      c_vp, c_i64, c_int, c_vp, c_vp], c_int),
    'fe3d_quad4_fint': ([c_i64, c_vp, c_vp, c_vp, c_vp, c_vp, c_vp, c_vp, c_i64, c_vp, c_vp, c_i64,
                         c_vp, c_vp], c_int),
    'fe3d_beamc_frame': ([c_i64, c_vp, c_vp, c_i64, c_vp, c_int, c_vp, c_vp, c_vp, c_vp, c_vp], c_int),
    'fe3d_beamc_probe_xe': ([c_i64, c_vp, c_vp, c_i64, c_vp, c_vp, c_vp, c_vp, c_vp], c_int),
    'fe3d_beamc_probe_ue': ([c_i64, c_vp, c_vp, c_i64, c_vp, c_vp, c_vp, c_vp], c_int),
    'fe3d_beamc_kc0': ([c_i64, c_vp, c_vp, c_vp, c_vp, c_vp, c_i64, c_vp, c_vp, c_vp, c_vp, c_i64, c_int,
                        c_vp, c_vp], c_int),
    'fe3d_beamc_kg': ([c_i64, c_vp, c_vp, c_vp, c_vp, c_vp, c_vp, c_i64, c_vp, c_vp, c_vp, c_vp, c_i64,
                       c_int, c_vp, c_vp], c_int),
    'fe3d_beamc_m': ([c_i64, c_vp, c_vp, c_vp, c_vp, c_vp, c_i64, c_vp, c_vp, c_vp, c_vp, c_i64, c_int,
                      c_vp, c_vp], c_int),
    'fe3d_quad4_finte': ([c_i64, c_vp, c_vp, c_vp, c_vp, c_vp, c_vp, c_vp, c_i64, c_vp, c_vp, c_i64, c_vp, c_vp,
                          c_vp], c_int),
    'fe3d_quad4_kg_given_stress': ([c_i64, c_vp, c_vp, c_vp, c_i64, c_vp, c_int, c_vp, c_vp, c_vp, c_int, c_vp,
                                    c_vp, c_vp, c_i64, c_vp, c_vp], c_int),
    'fe3d_tria3r_frame': ([c_i64, c_vp, c_vp, c_i64, c_vp, c_int, c_vp, c_vp, c_vp, c_vp, c_vp, c_vp], c_int),
    'fe3d_tria3r_probe_xe': ([c_i64, c_vp, c_vp, c_i64, c_vp, c_vp, c_vp, c_vp, c_vp], c_int),
    'fe3d_tria3r_probe_ue': ([c_i64, c_vp, c_vp, c_i64, c_vp, c_vp, c_vp, c_vp], c_int),
    'fe3d_tria3r_kc0': ([c_i64, c_vp, c_vp, c_vp, c_i64, c_vp, c_int, c_vp, c_vp, c_vp, c_vp, c_vp, c_i64,
                         c_vp, c_vp, c_int, c_vp, c_int, c_vp, c_vp, c_vp, c_i64, c_int, c_vp, c_vp], c_int),
    'fe3d_quad4r_kc0': ([c_i64, c_vp, c_vp, c_vp, c_i64, c_vp, c_int, c_vp, c_vp, c_vp, c_vp, c_vp, c_i64,
                         c_vp, c_vp, c_int, c_vp, c_int, c_vp, c_vp, c_vp, c_i64, c_int, c_vp, c_vp], c_int),
    'fe3d_tria3r_finte': ([c_i64, c_vp, c_vp, c_vp, c_vp, c_vp, c_vp, c_vp, c_i64, c_vp, c_vp, c_int, c_vp,
                           c_int, c_vp, c_i64, c_vp, c_vp, c_vp], c_int),
    'fe3d_quad4r_finte': ([c_i64, c_vp, c_vp, c_vp, c_vp, c_vp, c_vp, c_vp, c_i64, c_vp, c_vp, c_int, c_vp,
                           c_int, c_vp, c_i64, c_vp, c_vp, c_vp], c_int),
    'fe3d_tria3r_kg': ([c_i64, c_vp, c_vp, c_vp, c_i64, c_vp, c_int, c_vp, c_i64, c_vp, c_vp, c_vp, c_vp, c_vp,
                        c_vp, c_i64, c_vp, c_vp, c_vp, c_vp, c_i64, c_int, c_vp, c_vp], c_int),
    'fe3d_tria3r_kg_given_stress': ([c_i64, c_vp, c_vp, c_vp, c_i64, c_vp, c_vp, c_vp, c_vp, c_int, c_vp, c_vp,
                                     c_vp, c_i64, c_int, c_vp, c_vp], c_int),
    'fe3d_tria3r_m': ([c_i64, c_vp, c_vp, c_vp, c_i64, c_vp, c_vp, c_vp, c_i64, c_vp, c_vp, c_vp, c_vp, c_i64,
                       c_int, c_vp, c_vp], c_int),
    'fe3d_beamc_fint': ([c_i64, c_vp, c_vp, c_vp, c_vp, c_vp, c_i64, c_vp, c_vp, c_i64, c_vp, c_vp, c_vp], c_int),
    'fe3d_isotropic_plate_records': ([c_i64, c_vp, c_int, c_vp, c_int, c_vp, c_int, c_vp, c_int, c_vp, c_int,
                                      c_int, c_vp, c_vp], c_int),
    'fe3d_laminate_records': ([c_i64, c_int, c_vp, c_i64, c_vp, c_i64, c_vp, c_i64, c_vp, c_i64, c_vp, c_i64,
                               c_int, c_vp, c_vp], c_int),
    'fe3d_spmm': ([c_vp, c_vp, c_vp, c_vp, c_int, c_vp], c_int),
    'fe3d_solver_precond_multi': ([c_vp, c_vp, c_vp, c_int, c_vp], c_int),
    'fe3d_dense_gram_scratch': ([c_int, c_int], c_i64),
    'fe3d_dense_gram': ([c_i64, c_int, c_int, c_vp, c_vp, c_vp, c_vp, c_vp], c_int),
    'fe3d_dense_gemm_tall': ([c_i64, c_int, c_int, c_vp, c_vp, c_dbl, c_dbl, c_vp, c_vp], c_int),
    'fe3d_quad4_kc0_host': ([c_i64, c_vp, c_vp, c_vp, c_i64, c_vp, c_i64, c_vp, c_vp, c_vp, c_vp, c_i64, c_int,
                             c_i64, c_vp, c_vp], c_int),
    'fe3d_pattern_build': ([c_vp, c_vp, c_i64, c_i64, c_vp, c_vp, c_vp, c_vp], c_int),
    'fe3d_pattern_free': ([c_vp], c_int),
    'fe3d_pattern_info': ([c_vp, c_vp, c_vp, c_vp], c_int),
    'fe3d_pattern_arrays': ([c_vp, c_vp, c_vp, c_vp, c_vp], c_int),
    'fe3d_pattern_copy': ([c_vp, c_vp, c_vp, c_vp, c_vp], c_int),
    'fe3d_assemble': ([c_vp, c_vp, c_vp, c_vp], c_int),
    'fe3d_spmv': ([c_vp, c_vp, c_vp, c_vp, c_vp], c_int),
    'fe3d_solver_create': ([c_vp, c_int, c_vp], c_int),
    'fe3d_solver_setup': ([c_vp, c_vp, c_int, c_vp, c_vp], c_int),
    'fe3d_solver_solve': ([c_vp, c_vp, c_vp, c_vp, c_vp, c_vp], c_int),
    'fe3d_solver_free': ([c_vp], c_int),
    'fe3d_solver_set_blocks': ([c_vp, c_vp, c_vp, c_vp, c_vp], c_int),
    'fe3d_lpc_features': ([c_vp, c_vp, c_vp, c_vp], c_int),
    'fe3d_lpc_features_set': ([c_vp, c_int, c_vp, c_vp, c_vp], c_int),
    'fe3d_lpc_forward': ([c_i64, c_vp, c_vp, c_vp, c_vp, c_vp], c_int),
    'fe3d_lpc_blocks': ([c_vp, c_vp, c_vp, ctypes.c_float, c_vp, c_vp], c_int),
    'fe3d_lpc_apply': ([c_vp, c_vp, c_vp, c_vp], c_int),
    'fe3d_lpc_loss_grad': ([c_vp, c_vp, c_vp, c_vp, c_vp, c_vp, ctypes.c_double, ctypes.c_double,
                            ctypes.c_float, c_int, c_vp, c_vp, c_vp], c_int),
    'fe3d_lpc_backward': ([c_i64, c_vp, c_vp, c_vp, c_vp, c_vp, c_vp, c_vp], c_int),
    'fe3d_lpc_adam': ([c_i64, c_vp, c_vp, c_vp, c_vp, ctypes.c_float, ctypes.c_float, ctypes.c_float,
                       ctypes.c_float, c_int, c_vp], c_int),
    'fe3d_bsolver_create': ([c_vp, c_int, c_i64, c_vp, c_vp], c_int),
    'fe3d_bsolver_setup': ([c_vp, c_vp, c_int, c_vp, c_vp], c_int),
    'fe3d_bsolver_info': ([c_vp, c_vp, c_vp], c_int),
    'fe3d_bsolver_set_split': ([c_vp, c_i64, c_vp], c_int),
    'fe3d_bsolver_solve': ([c_vp, c_vp, c_vp, c_vp, c_vp, c_vp, c_vp, c_vp, c_vp], c_int),
    'fe3d_bsolver_free': ([c_vp], c_int),
    'fe3d_pattern_build_elements': ([c_vp, c_int, c_i64, c_vp, c_vp, c_vp, c_vp], c_int),
    'fe3d_fmap_build': ([c_vp, c_vp, c_int, c_vp, c_vp, c_vp], c_int),
    'fe3d_fmap_free': ([c_vp], c_int),
    'fe3d_fmap_info': ([c_vp, c_int, c_vp, c_vp], c_int),
    'fe3d_csr_scatter': ([c_vp, c_int, c_vp, c_vp, c_i64, c_vp, c_int, c_vp, c_vp], c_int),
    'fe3d_quad4_kc0_csr': ([c_vp, c_int, c_vp, c_i64, c_vp, c_int, c_vp, c_i64, c_vp, c_vp, c_int, c_vp, c_vp],
                           c_int),
    'fe3d_noalloc_max_rows': ([], c_i64),
    'fe3d_jacobi_pcg_noalloc': ([c_i64, c_vp, c_vp, c_vp, c_vp, c_vp, c_vp, c_vp, c_vp], c_int),
}


class Fe3dError(RuntimeError):
    """Error reported by the CUDA library (negative status or device error word)."""


def declared_symbols():
    return dict(_SIGS)


def load(path=LIB_PATH):
    """Load the shared library (without touching the GPU)."""
    global _lib
    if _lib is None:
        if not os.path.exists(path):
            raise Fe3dError('%s is not built: run `python -m pyfe3d_gb300.build`' % path)
        lib = ctypes.CDLL(path)
        for name, (args, res) in _SIGS.items():
            f = getattr(lib, name)
            f.argtypes = args
            f.restype = res
        _lib = lib
    return _lib


def register(name, args, res=c_int):
    """Declare the signature of an additional entry point."""
    _SIGS[name] = (args, res)
    if _lib is not None:
        f = getattr(_lib, name)
        f.argtypes = args
        f.restype = res


_torch = None
_available = False


def torch_mod():
    global _torch
    if _torch is None:
        import torch
        _torch = torch
    return _torch


def _device_index():
    """Index of the current CUDA device; raises when no GPU is available."""
    global _available
    torch = torch_mod()
    if not _available:
        if not torch.cuda.is_available():
            raise Fe3dError('pyfe3d_gb300 needs a CUDA device (GB300, sm_103a); none is available')
        _available = True
    return torch.cuda.current_device()


def device():
    """The current CUDA device; raises when no GPU is available."""
    return torch_mod().device('cuda', _device_index())


def _raw_stream():
    torch = torch_mod()
    raw = getattr(torch._C, '_cuda_getCurrentRawStream', None)
    return raw(torch.cuda.current_device()) if raw is not None else torch.cuda.current_stream().cuda_stream


def stream_ptr():
    return c_vp(_raw_stream())


def err_word():
    """Per-device int32 error word the kernels OR their error bits into: pinned
    host memory, which kernels touch only to report an error and the host
    reads without a copy once it has synchronised the stream."""
    torch = torch_mod()
    idx = _device_index()
    w = _err_words.get(idx)
    if w is None:
        w = torch.zeros(1, dtype=torch.int32).pin_memory()
        _err_words[idx] = w
    return w


class _Constants:
    """Small constant device tensors (a scalar, zero record indices) kept per
    device and stream, so that a call that needs one neither copies from the
    host nor fills.  A tensor is only ever used on the stream it was made on,
    which also orders its release; at most 64 tensors of 16 MB are kept, the
    least recently used released first.  Nothing is kept during a graph
    capture, whose memory belongs to the graph."""

    def __init__(self):
        self._kept = collections.OrderedDict()
        self._lock = threading.Lock()

    def get(self, kind, n, make):
        """make(m) returns a tensor of m equal entries; the result has n of them."""
        if n > (1 << 21) or torch_mod().cuda.is_current_stream_capturing():
            return make(n)
        key = (kind, _device_index(), _raw_stream())
        with self._lock:
            t = self._kept.get(key)
            if t is None or t.numel() < n:
                t = self._kept[key] = make(max(n, 1024))
                if len(self._kept) > 64:
                    self._kept.popitem(last=False)
            self._kept.move_to_end(key)
        return t[:n]


_constants = _Constants()


def scalar_f64(v):
    """A one-entry float64 device tensor holding v."""
    torch = torch_mod()
    v = float(v)
    return _constants.get(('f64', v.hex()), 1,
                          lambda m: torch.full((m,), v, dtype=torch.float64, device=device()))


def zeros_i32(n):
    """n int32 zeros on the device (not to be written)."""
    torch = torch_mod()
    return _constants.get('i32', n, lambda m: torch.zeros(m, dtype=torch.int32, device=device()))


def ptr(t):
    if t is None:
        return None
    return c_vp(t.data_ptr())


_kept = []


def keep(t):
    """Pointer of a temporary device tensor that must outlive the launch it
    is passed to: the tensor is held until the next ``check`` has
    synchronised the stream (otherwise the caching allocator could hand its
    memory to the next temporary before the kernel has run)."""
    _kept.append(t)
    return ptr(t)


def synchronize():
    """Wait for the current stream."""
    rc = load().fe3d_stream_synchronize(stream_ptr())
    if rc != 0:
        raise Fe3dError('%s (status %d)' % (FE3D_ERRORS.get(rc, 'unknown'), rc))


def check(rc, what='', err=None):
    """Raise on a negative status; with ``err``, synchronise and check the device word."""
    if _kept:
        synchronize()
        del _kept[:]
    if rc != 0:
        raise Fe3dError('%s: %s (status %d)' % (what, FE3D_ERRORS.get(rc, 'unknown'), rc))
    if err is not None:
        synchronize()
        if ctypes.c_int32.from_address(err.data_ptr()).value:
            v = int(err.item())
            err.zero_()
            raise Fe3dError('%s: device reported error bits 0x%x (an offset outside the '
                            'caller\'s buffers)' % (what, v))


_NP_TO_TORCH = None


def _torch_dtype(dtype):
    global _NP_TO_TORCH
    if _NP_TO_TORCH is None:
        torch = torch_mod()
        _NP_TO_TORCH = {np.float64: torch.float64, np.int64: torch.int64, np.int32: torch.int32,
                        np.float32: torch.float32, np.uint8: torch.uint8}
    return _NP_TO_TORCH[dtype] if dtype in _NP_TO_TORCH else _NP_TO_TORCH[np.dtype(dtype).type]


def to_device(a, dtype):
    """numpy array or torch tensor -> contiguous CUDA tensor of ``dtype`` (numpy dtype)."""
    torch = torch_mod()
    tdt = _torch_dtype(dtype)
    if isinstance(a, torch.Tensor):
        t = a
        if t.dtype != tdt:
            t = t.to(tdt)
        idx = _device_index()
        if not t.is_cuda or t.get_device() != idx:
            t = t.to(device())
        return t.contiguous()
    arr = np.ascontiguousarray(a, dtype=dtype)
    return torch.from_numpy(arr).to(device())


def is_cuda_tensor(a):
    try:
        torch = torch_mod()
    except ImportError:
        return False
    return isinstance(a, torch.Tensor) and a.is_cuda
