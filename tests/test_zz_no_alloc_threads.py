"""sfwi_ot_noalloc from several threads, each on its own stream: the calls share
one fixed working array and take turns on it, so each gives what it gives
alone, bit for bit."""
import ctypes as C
import threading

import numpy as np
import pytest

from tests.test_zz_no_alloc import _call, _case

pytestmark = pytest.mark.gpu


def test_calls_of_several_threads_take_turns():
    torch = pytest.importorskip("torch")
    from sfwi_gb300 import _lib
    lib = _lib.load()
    jobs = []
    for k, (ntr, nt, kind) in enumerate(((8000, 300, 1), (3000, 900, 2), (40, 5000, 3), (700, 1200, 1))):
        dev = [torch.from_numpy(a).cuda() for a in _case(k, ntr, nt)]
        out = [torch.zeros((ntr, nt), dtype=torch.float32, device="cuda") for _ in range(2)]
        torch.cuda.synchronize()
        m = _call(lib, kind, dev, *out, nt, ntr, 1e-3)
        jobs.append((ntr, nt, kind, dev, m, [o.cpu().numpy() for o in out]))
    bad = []

    def work(ntr, nt, kind, dev, m, want):
        s = torch.cuda.Stream()
        out = [torch.zeros((ntr, nt), dtype=torch.float32, device="cuda") for _ in range(2)]
        torch.cuda.synchronize()
        for _ in range(40):
            got = _call(lib, kind, dev, *out, nt, ntr, 1e-3, C.c_void_p(s.cuda_stream))
            if got != m or not all(np.array_equal(o.cpu().numpy(), w) for o, w in zip(out, want)):
                bad.append((kind, got, m))

    threads = [threading.Thread(target=work, args=j) for j in jobs + jobs[:2]]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
