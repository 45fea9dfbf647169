"""w-kernel generation sets the kernels' shared-memory limit, which all threads of
a process share, to the same value for every largest support and above what any
call launches with: a call for small supports cannot make another thread's launch
fail.  On a runtime that records the calls; the results of concurrent calls are in
tests/test_gpu_gcf_threads.py."""
import ctypes as C
import re

from tests import fake_runtime


def test_limit_is_the_same_for_every_support(tmp_path):
    fake = fake_runtime.load(str(tmp_path), ["gb_gcf"])
    out = (C.c_double * 2)()  # no kernel runs
    limits, smem = {}, 0
    for smax in (2, 16, 64, 250, 256):
        fake.clear()
        rc = fake.lib.gb_gcf_generate(1, (C.c_double * 1)(3.0), (C.c_int32 * 1)(smax),
                                      (C.c_int64 * 1)(0), smax, C.c_double(0.1), None, out, None, None)
        assert rc == 0
        for o in fake.ops():
            if m := re.match(r"attr (\S+) (\d+)", o):
                limits.setdefault(m[1], set()).add(int(m[2]))
            if m := re.match(r"launch \S+k_gcf_(?:first|second)\S* .*smem=(\d+)", o):
                smem = max(smem, int(m[1]))
    assert len(limits) == 2 and smem > 48 * 1024
    for v in limits.values():
        assert len(v) == 1 and v.pop() >= smem
