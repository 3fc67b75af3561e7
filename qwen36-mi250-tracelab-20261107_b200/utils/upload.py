"""Index tables from host memory to a device, complete on return."""

from __future__ import annotations

import torch

_streams: dict[int, torch.cuda.Stream] = {}  # one copy stream per device


def to_device(host: torch.Tensor, device: torch.device) -> torch.Tensor:
    """``host`` (pinned, where ``device`` is a GPU) on ``device``. The copy is complete when the call returns, so the result may
    be read on any stream; it goes through a stream of its own, so the call does not wait for what the current stream is busy
    with. Refused inside a graph capture: a replay would copy from host memory that has been given away since."""
    if device.type != "cuda":
        return host.to(device)
    with torch.cuda.device(device):
        if torch.cuda.is_current_stream_capturing():
            raise RuntimeError("host tables cannot be copied inside a graph capture: make them before it")
        current = torch.cuda.current_stream()
        copy = _streams.get(current.device_index)
        if copy is None:
            copy = _streams[current.device_index] = torch.cuda.Stream()
        torch.cuda.set_stream(copy)
        try:
            out = host.to(copy.device, non_blocking=True)
        finally:
            torch.cuda.set_stream(current)
        copy.synchronize()
        out.record_stream(current)  # the memory is the copy stream's: not reused before the current stream is done with it
    return out
