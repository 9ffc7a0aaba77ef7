"""GPU: reads of several fields are the device's bytes on either side of the
line between one copy each and the shared buffer, with names that repeat, an
unaligned field size and a name that is no field, from several threads."""
import threading

import numpy as np
import pytest

from sph import scenes

pytestmark = pytest.mark.gpu

READS = [("position",), ("position", "density"), ("density", "position", "density"), ("gridcell", "gridres", "mass"),
         ("position", "velocity", "force", "acceleration", "density"), ("position", "no such field", "density"),
         ("n", "position", "velocity", "force", "acceleration", "density", "gridcell", "mass", "gridres")]


# position and density fill the two-field line (64 KB) exactly at 4,096
@pytest.mark.parametrize("pnum", [37, 4095, 4096, 4097, 20000])
@pytest.mark.parametrize("names", READS)
def test_read_is_the_devices_bytes(pnum, names):
    sc = scenes.wcsph_block(3, 3, 4, pnum=pnum, jitter=0.05)
    ps = sc.system()
    ps.update_fused(2)
    ps.sync_device_to_host()
    want = {f: np.array(ps.get_fields(f)[0]) for f in names if f != "no such field"}
    for f in want:
        ps.get_fields(f)[0].view(np.uint8)[...] = 0xA5
    ps.sync_fields_device_to_host(*names)
    for f in want:
        assert ps.get_fields(f)[0].tobytes() == want[f].tobytes(), f
    ps.close()


def test_reads_from_threads():
    sc = scenes.wcsph_block(11, 7, 13, jitter=0.05)
    ps = sc.system()
    ps.update_fused(1)
    ps.sync_device_to_host()
    want = {f: np.array(ps.get_fields(f)[0]) for f in ("position", "velocity", "force", "density")}

    def read(names):
        for _ in range(50):
            ps.sync_fields_device_to_host(*names)

    ts = [threading.Thread(target=read, args=(p,)) for p in (("position", "velocity"), ("force", "density"))]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for f in want:
        assert ps.get_fields(f)[0].tobytes() == want[f].tobytes(), f
    ps.close()
