"""gb_gcf_generate from several host threads at once, each with its own largest
support, from less to more shared memory than a kernel may use by default: every
call gives what it gives alone."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_threads_with_different_largest_supports():
    import torch

    from rc_gb300 import gcf as G

    args = {s: (np.array([0.0, 90.0]), np.array([s, 3], np.int32), s, 0.08) for s in (250, 16, 128, 8)}
    alone = {s: G.generate(*a)[0] for s, a in args.items()}
    torch.cuda.synchronize()
    errors, gate = [], threading.Barrier(len(args))

    def one(s):
        try:
            gate.wait()
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(60):
                    got = G.generate(*args[s])[0]
                torch.cuda.current_stream().synchronize()
                assert torch.equal(got, alone[s])
        except Exception as e:  # shown below
            errors.append((s, e))

    threads = [threading.Thread(target=one, args=(s,)) for s in args]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
