"""CPU: batched plans, compressed bases and shards take any false value as "the
current stream", and a given stream as itself."""
from types import SimpleNamespace

import pytest
import torch

from frsz_b200 import BatchPlan, CompressedBasis, codec, shard


def _shard_stream(monkeypatch):
    def ptr(stream):
        seen = []
        fake = SimpleNamespace(frsz2_compress_blocks=lambda *a: seen.append(a[-1]) or 0,
                               frsz2_decompress_blocks=lambda *a: seen.append(a[-1]) or 0)
        monkeypatch.setattr(shard, "lib", lambda: fake)
        x, b = torch.zeros(64), torch.zeros(1024, dtype=torch.uint8)
        shard.compress_shard(x, 64, 16, 32, 0, 2, b, stream=stream)
        shard.decompress_shard(b, 64, torch.float32, 16, 32, 0, 2, x, stream=stream)
        assert seen[0] == seen[1]
        return seen[0]

    return ptr


@pytest.mark.parametrize("which", ["batch", "basis", "shard"])
def test_stream_argument(monkeypatch, which):
    monkeypatch.setattr(codec, "_raw_stream", lambda device: 4096 + device)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 3)
    ptr = {"batch": lambda s: BatchPlan._stream(None, s), "basis": lambda s: CompressedBasis._stream(None, s),
           "shard": _shard_stream(monkeypatch)}[which]
    for none in (None, 0, False):
        assert ptr(none) == 4099
    assert ptr(SimpleNamespace(cuda_stream=77)) == 77
