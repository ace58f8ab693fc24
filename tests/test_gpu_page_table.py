"""Page tables sent to the device without waiting: as many uploads as go round the host buffers twice, each read behind the next in stream order."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("slots,max_seq_len", [(6, 640), (130, 64 * 2100)])     # (the second table is over 1 MB: row by row)
def test_tables_follow_the_host(slots, max_seq_len):
    from inference_engine_rust_b200.cache import Cache, KVRequest
    cache = Cache({0: KVRequest(1, 16)}, max_tokens=64 * 300, max_seq_len=max_seq_len, max_sequences=slots, dtype=torch.bfloat16,
                  device="cuda:0")
    group, held, seen = cache.kv_groups[0], [cache.open_sequence() for _ in range(3)], []
    busy = torch.zeros(1 << 26, device="cuda:0")
    for step in range(10):
        for i, slot in enumerate(held):
            cache.reserve(slot, 64 * (step * (i + 1) % 7 + 1 + step // 2))
        if step == 5:
            cache.close_sequence(held.pop())
        busy.add_(1.0)                                            # the device is behind the host
        cache.upload(wait=False)
        seen.append((group.table.clone(), group.table_host.copy()))
    for device, host in seen:
        assert np.array_equal(device.cpu().numpy(), host)
