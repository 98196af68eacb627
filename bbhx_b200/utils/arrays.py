"""Array plumbing: torch CUDA tensors are the device container (the reference uses cupy)."""
import numpy as np


def torch():
    import torch as _t

    return _t


_cuda_seen = False
_devices = {}


def device():
    """The current CUDA device (as torch.device; one object per index)."""
    global _cuda_seen
    t = torch()
    if not _cuda_seen:
        if not t.cuda.is_available():
            raise RuntimeError("bbhx_b200 needs a CUDA device (there is no CPU fallback)")
        _cuda_seen = True
    i = t.cuda.current_device()
    if i not in _devices:
        _devices[i] = t.device("cuda", i)
    return _devices[i]


def to_dev(x, dtype=None):
    """numpy / scalar / torch -> contiguous CUDA tensor (float64 unless dtype given)."""
    t = torch()
    dtype = dtype or t.float64
    if isinstance(x, t.Tensor):
        if x.is_cuda and x.dtype == dtype and x.is_contiguous() and x.device == device():
            return x
        return x.to(device=device(), dtype=dtype).contiguous()
    return t.as_tensor(np.ascontiguousarray(x), dtype=dtype, device=device()).contiguous()


def param_rows(params):
    """The 12 source parameters as device arrays: host arrays of one length go over in one copy and
    come back as rows of that tensor (12 copies of a few bytes each were a fifth of a small
    call); anything else is converted one by one.  f_ref (6) does not enter the model and is passed
    through."""
    t = torch()
    if len(params) != 12:
        raise ValueError("12 source parameters are needed, got %d" % len(params))
    if not any(isinstance(v, t.Tensor) for v in params):
        rows = [np.atleast_1d(np.asarray(v)) for k, v in enumerate(params) if k != 6]
        if all(r.ndim == 1 and r.shape == rows[0].shape and r.dtype.kind in "fiub" for r in rows):
            dev = t.as_tensor(np.array(rows, dtype=np.float64), device=device())
            out = list(dev.unbind(0))
            return tuple(out[:6]) + (params[6],) + tuple(out[6:])
    return tuple(v if k == 6 else to_dev(atleast_1d(v)) for k, v in enumerate(params))


def to_np(x):
    t = torch()
    if isinstance(x, t.Tensor):
        return x.detach().cpu().numpy()
    return np.asarray(x)


def atleast_1d(x):
    t = torch()
    if isinstance(x, t.Tensor):
        return x.reshape(-1) if x.ndim == 0 else x
    return np.atleast_1d(x)
