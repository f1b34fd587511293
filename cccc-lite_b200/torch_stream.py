"""The stream that a call from Python goes to."""
from __future__ import annotations


def raw_stream(stream=None):
    """The raw cudaStream_t: the given one, or torch's current one for None.  That is asked for directly where torch has been initialised and has the two
    calls that its own stream object is made of: the object takes 3.2 us, a third of a call."""
    if stream is not None:
        return stream
    import torch

    if torch.cuda.is_initialized():
        try:
            return torch._C._cuda_getCurrentRawStream(torch._C._cuda_getDevice())
        except AttributeError:    # a version of torch without them
            pass
    return torch.cuda.current_stream().cuda_stream
