"""Device-buffer plumbing: numpy arrays are copied to CUDA tensors and back;
CUDA tensors are used in place (zero copy)."""
import ctypes

import numpy as np
import torch

from ._lib import call, lib

_NP2T = {np.float64: torch.float64, np.float32: torch.float32, np.int32: torch.int32,
         np.int64: torch.int64, np.uint8: torch.uint8}

UPLOAD_MAX = 16000      # NX_UPLOAD_MAX


def require_cuda():
    if not torch.cuda.is_available():
        raise RuntimeError("nixis_gb300 needs a CUDA GPU (sm_103a); none is available")


def stream_handle(stream=None):
    # (the current stream's handle without torch's stream object: 0.4 us, not 2.9)
    return ctypes.c_void_p(stream.cuda_stream if stream is not None
                           else torch._C._cuda_getCurrentRawStream(torch.cuda.current_device()))


def ctypes_void(v):
    return ctypes.c_void_p(int(v))


def ptr(t):
    return ctypes.c_void_p(t.data_ptr()) if t is not None else None


def is_host(a):
    return isinstance(a, np.ndarray)


def _in_memory(a):
    """Whether a numpy array's bytes are memory that numpy, or from_device,
    allocated: the base of everything it is a view of, through memoryviews as
    well.  Whatever else may lie behind an array (a mapped file, as np.memmap or
    np.frombuffer of one or a checkpoint loaded with mmap; memory of another
    process) is not told apart, and the GPU is not sent to it."""
    while True:
        if isinstance(a, np.ndarray):
            if a.base is None:
                return bool(a.flags.owndata)
            a = a.base
        elif isinstance(a, memoryview):
            a = a.obj
        else:
            return getattr(a, "_nx_host", False)


def from_device(t):
    """A CUDA tensor's values as a numpy array, in torch's memory: the driver
    program at 256,002 vertices takes 3.0 ms so and 4.8 ms with arrays made by
    numpy, whose pages cost more to make.  Where upload would ask, the array's
    base is marked as such."""
    a = (t.cpu() if t.is_cuda else t.clone()).numpy()
    if a.nbytes > UPLOAD_MAX:
        a.base._nx_host = True
    return a


def upload(arr, tdt):
    """A CUDA tensor with the bytes of a contiguous numpy array, which the
    caller may change as soon as this returns.

    Small tables go as kernel arguments (nothing waits).  The rest is copied
    straight out of the array: the GPU reads pageable memory here at
    110-180 GB/s, and staging through pinned memory copies it once more on one
    core (24 MB: 147 us against 195, 80 MB: 466 against 627).  That copy waits
    for the stream, so it is staged where the stream has work queued, under
    capture, and for memory that is not known (_in_memory)."""
    if arr.nbytes <= UPLOAD_MAX:
        t = torch.empty(arr.shape, dtype=tdt, device="cuda")
        if arr.nbytes:
            call("nx_upload", ptr(t), ctypes.c_void_p(arr.ctypes.data), arr.nbytes, stream_handle())
        return t
    t = torch.from_numpy(arr)
    if _in_memory(arr) and lib().nx_stream_idle(stream_handle()):
        return t.to("cuda")
    return t.pin_memory().to("cuda", non_blocking=True)


def put(dst, src, stream=None):
    """The bytes of a small numpy array (or ctypes structure) into the CUDA
    tensor dst, in stream order; src may change as soon as this returns."""
    a = np.frombuffer(src, np.uint8) if not isinstance(src, np.ndarray) else np.ascontiguousarray(src)
    call("nx_upload", ptr(dst), ctypes.c_void_p(a.ctypes.data), a.nbytes, stream_handle(stream))


def to_host(dst, src):
    """dst[...] = src for a numpy array and a CUDA tensor of its type; straight
    into a contiguous array (80 MB: 430 us; through a fresh array, whose pages
    have to be made first, 2,870)."""
    t = torch.empty(0, dtype=src.dtype).numpy().dtype
    if (dst.dtype == t and dst.flags.c_contiguous and dst.flags.writeable and tuple(dst.shape) == tuple(src.shape)
            and _in_memory(dst)):
        torch.from_numpy(dst).copy_(src)
    else:
        dst[...] = src.cpu().numpy()


def to_device(a, dtype, shape=None, name="array"):
    """Return a contiguous CUDA tensor of `dtype` holding `a` (numpy or torch)."""
    tdt = _NP2T[np.dtype(dtype).type]
    if isinstance(a, torch.Tensor):
        t = a
        if not t.is_cuda:
            require_cuda()
            t = t.to("cuda", non_blocking=False)
        if t.dtype != tdt:
            t = t.to(tdt)
        t = t.contiguous()
    else:
        require_cuda()
        t = upload(np.ascontiguousarray(a, dtype=dtype), tdt)
    if shape is not None and tuple(t.shape) != tuple(shape):
        raise ValueError(f"{name}: expected shape {tuple(shape)}, got {tuple(t.shape)}")
    return t


def check_vertices(v, name="verts"):
    if v.ndim != 2 or v.shape[1] != 3:
        raise ValueError(f"{name}: expected shape (N, 3), got {tuple(v.shape)}")


def check_tables(perm, pgi):
    p = np.asarray(perm.cpu() if isinstance(perm, torch.Tensor) else perm)
    g = np.asarray(pgi.cpu() if isinstance(pgi, torch.Tensor) else pgi)
    if p.shape != (256,) or g.shape != (256,):
        raise ValueError("perm and perm_grad_index_3D must have 256 entries")
    if p.min() < 0 or p.max() > 255 or g.min() < 0 or g.max() > 69 or np.any(g % 3):
        raise ValueError("perm / perm_grad_index_3D are not tables made by init()")
