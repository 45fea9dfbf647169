"""The FP32 transforms' tables are in device memory before any stream may read
them: the copies that fill them go on one stream and are waited for before the
first kernel, whatever stream that runs on.  (A plain copy from pageable memory
may return before the device has the data, and a non-blocking stream is not
ordered after the default stream on which it runs.)  On a runtime that records the
calls; tests/test_gpu_fft_streams.py has the results."""
import ctypes as C
import re

import pytest

from tests import fake_runtime


@pytest.mark.parametrize("n", [64, 4096])
@pytest.mark.parametrize("stream", [None, 0x77])
def test_tables_are_waited_for_before_the_first_kernel(tmp_path, n, stream):
    fake = fake_runtime.load(str(tmp_path), ["gb_fft", "gb_imaging"])
    buf = (C.c_float * 16)()
    call = lambda: fake.lib.gb_image_to_grid_f32(buf, None, n, buf, C.c_void_p(stream))
    assert call() == 0
    ops = fake.ops()
    launches = [i for i, o in enumerate(ops) if o.startswith("launch")]
    copies = [i for i, o in enumerate(ops) if o.startswith("memcpy")]
    assert len(launches) == 2 and copies and copies[-1] < launches[0]
    streams = {re.search(r"stream=(\w+)", ops[i]) and re.search(r"stream=(\w+)", ops[i])[1] for i in copies}
    assert None not in streams, ops  # copies on no stream of their own
    assert len(streams) == 1
    assert f"sync stream={streams.pop()}" in ops[copies[-1] + 1:launches[0]], ops
    fake.clear()
    assert call() == 0
    assert all(o.startswith("launch") for o in fake.ops() if not o.startswith("attr"))
