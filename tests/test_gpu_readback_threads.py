"""GPU: reads of several fields by two threads through one store's readback
buffer: each thread's fields are overwritten before every read and compared
right after it, so bytes that a read did not copy, or took from the other
thread's, show."""
import threading

import numpy as np
import pytest

from sph import scenes

pytestmark = pytest.mark.gpu


def test_each_read_of_each_thread_is_the_devices_bytes():
    sc = scenes.wcsph_block(11, 7, 13, jitter=0.05)
    ps = sc.system()
    ps.update_fused(1)
    ps.sync_device_to_host()
    pairs = (("position", "velocity"), ("force", "density"))
    want = {f: ps.get_fields(f)[0].tobytes() for p in pairs for f in p}
    bad = []

    def read(names):
        views = [ps.get_fields(f)[0].view(np.uint8) for f in names]
        for k in range(200):
            for v in views:
                v[...] = 0xA5
            ps.sync_fields_device_to_host(*names)
            bad.extend((k, f) for f, v in zip(names, views) if v.tobytes() != want[f])

    ts = [threading.Thread(target=read, args=(p,)) for p in pairs]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not bad, bad[:10]
    ps.close()
