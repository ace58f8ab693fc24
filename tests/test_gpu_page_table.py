"""Page tables sent to the device without waiting: as many uploads as go round the host buffers twice, each read behind the next in stream order, the
first of either round queued behind work that outlasts the host's."""
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
        if step % 5 == 0:
            torch.cuda.synchronize()
            for _ in range(400):                                      # (some 30 ms: five steps here take the host a few)
                busy.add_(1.0)
            done = torch.cuda.Event()
            done.record()
        for i, slot in enumerate(held):
            cache.reserve(slot, 64 * (step + 1 if i == 0 else step * (i + 1) % 7 + 1 + step // 2))      # (the first grows every step)
        if step == 5:
            cache.close_sequence(held.pop())
        # the device is behind the host: four uploads do not wait for it, the fifth for the first one's buffer
        if step % 5 < 4:
            cache.upload(wait=False)
            assert not done.query()
        else:
            assert not done.query()
            cache.upload(wait=False)
            assert done.query()
        seen.append((group.table.clone(), group.table_host.copy()))
    for device, host in seen:
        assert np.array_equal(device.cpu().numpy(), host)
