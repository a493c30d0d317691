"""
Device plumbing: PyTorch is used only for device memory, streams and graph
capture. All arithmetic happens in the CUDA kernels of libptn_gb300.so.
"""

import warnings

import numpy as np
import torch

from . import _lib

CDT = torch.complex128


_DEVICES = {}


def device():
    """The current CUDA device (asked for several times per call: availability is checked
    once, the torch.device objects are kept)."""
    if not _DEVICES and not torch.cuda.is_available():
        raise RuntimeError("pytenet_gb300 needs a CUDA GPU (GB300, sm_103a); no CPU fallback exists")
    i = torch.cuda.current_device()
    d = _DEVICES.get(i)
    if d is None:
        d = _DEVICES[i] = torch.device("cuda", i)
    return d


def lib():
    return _lib.load()


def stream_ptr():
    return torch.cuda.current_stream().cuda_stream


def ptr(t):
    return t.data_ptr() if t is not None else None


def to_dev(x):
    """Host array (or device tensor) -> contiguous complex128 device tensor."""
    if isinstance(x, torch.Tensor):
        if x.dtype is CDT and x.is_cuda and x.get_device() == torch.cuda.current_device():
            return x if x.is_contiguous() else x.contiguous()
        t = x.to(device=device(), dtype=CDT)
        return t.contiguous()
    a = np.ascontiguousarray(np.asarray(x), dtype=np.complex128)
    return torch.from_numpy(a).to(device(), non_blocking=False)


def check_device():
    """Raise if a kernel on the device gave up on a bounded wait since the last check (results
    since then are NaN or incomplete). Waits for the current stream: for places that read a
    result anyway."""
    code = lib().ptn_device_error(stream_ptr())
    if code != 0:
        raise _lib.PtnError(_lib.PTN_TIMEOUT if code > 0 else _lib.PTN_CUDA_ERROR,
                            f"a bounded wait of a device kernel expired (code {code})"
                            if code > 0 else "the device's error word cannot be read")


def to_host_all(tensors):
    """Device tensors -> NumPy arrays; raises if a kernel before them did not finish."""
    out = [t.detach().cpu().numpy() for t in tensors]
    if any(t.is_cuda for t in tensors):
        check_device()
    return out


def to_host(t):
    return to_host_all([t])[0]


def scalar(t):
    """The first entry of a device tensor as a Python number, checked like to_host."""
    return to_host(t.reshape(-1)[:1])[0].item()


def empty(shape):
    return torch.empty(tuple(int(s) for s in shape), dtype=CDT, device=device())


def zeros(shape):
    return torch.zeros(tuple(int(s) for s in shape), dtype=CDT, device=device())


class Workspace:
    """Grow-only device scratch buffer (bytes). A run's buffer remembers a size that the device
    had no memory for (asking again is slow, and not possible while a graph is captured); with
    remember=False every call asks again."""

    def __init__(self, remember=True):
        self.buf = None
        self.remember = remember
        self.refused = None   # the smallest size that was refused

    def get(self, nbytes, least=None):
        """A buffer of nbytes, or where the device has no memory for that, of at least least()
        (None: nbytes); then use what fits, min(nbytes, buf.numel())."""
        nbytes = max(int(nbytes), 256)
        if self.buf is not None and self.buf.numel() >= nbytes:
            return self.buf
        if least is None or self.refused is None or nbytes < self.refused:
            try:
                self.buf = torch.empty(nbytes, dtype=torch.uint8, device=device())
                return self.buf
            except torch.cuda.OutOfMemoryError:
                if least is None:
                    raise
                if self.remember:
                    self.refused = nbytes
        low = max(int(least()), 256)
        if self.buf is None or self.buf.numel() < low:
            self.buf = None
            self.buf = torch.empty(low, dtype=torch.uint8, device=device())
        return self.buf

    def room(self, nbytes, least):
        """(buffer, bytes of it to use) of get(nbytes, least)."""
        nbytes = max(int(nbytes), 256)
        buf = self.get(nbytes, least)
        return buf, min(nbytes, buf.numel())

    def for_precision(self, query, prec):
        """Workspace of a contraction: (buffer, bytes, precision to call it with), `query` the
        size as a function of the precision. Where the device has no memory for it the FP64
        form takes the DMMA kernels, and the mixed form becomes the FP64 form on those."""
        need = query(prec)
        buf, n = self.room(need, lambda: query(_lib.PREC_FP64_DMMA))
        if n < need and prec == _lib.PREC_SPLIT_BF16:
            warnings.warn(f"no device memory for the {need / 2**30:.1f} GB workspace of the mixed "
                          "form: FP64 kernels", RuntimeWarning, stacklevel=3)
            prec = _lib.PREC_FP64
        return buf, n, prec

    def ptr(self, nbytes):
        return self.get(nbytes).data_ptr(), max(int(nbytes), 256)


def call(fn, *args):
    """Invoke a C entry point and raise on a non-OK status."""
    _lib.check(fn(*args))
