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
    current = torch.cuda.current_stream(device)
    with torch.cuda.stream(current):
        if torch.cuda.is_current_stream_capturing():
            raise RuntimeError("host tables cannot be copied inside a graph capture: make them before it")
    index = current.device_index
    copy = _streams.get(index)
    if copy is None:
        copy = _streams[index] = torch.cuda.Stream(device=current.device)
    with torch.cuda.stream(copy):
        out = host.to(current.device, non_blocking=True)
    copy.synchronize()
    out.record_stream(current)  # the memory is the copy stream's: not reused before the current stream is done with it
    return out
